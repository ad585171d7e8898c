// Sums of partial results in a fixed order: the ranges of a cut reduction (filter gradients, convolutions with too few output tiles
// for the chip), the images of a bias gradient of a fully connected layer.  Deterministic, no atomics.
//
// HBM / L2 bound: parts * n reads, n writes.  Two forms:
//   wide     a thread owns four consecutive elements (one without 16-byte alignment) and adds the parts in ascending order, four
//            loads in flight; fills the chip from about 150 k elements on;
//   narrow   few elements of many parts (a CIFAR layer's 2400 filter elements from 280 ranges took 15.9 us in the wide form, all of it load
//            latency; 3.1 us here): a block owns 32 elements, its eight warps take every eighth part, the eight sums are added in
//            warp order.
#include "conv_internal.cuh"

namespace {

constexpr int kThreads = 256;

struct SumParams {
  float* out;
  float const* part;
  size_t n, stride;
  int parts;
  vlb::SumEpilogue e;
};

__device__ __forceinline__ float finish(SumParams const& p, float s, size_t i)
{
  float o = p.e.inMult * s;
  if (p.e.bias) o += p.e.bias[(i / p.e.P) % p.e.K];
  if (p.e.outMult != 0.f) o += p.e.outMult * p.out[i];
  if (p.e.relu) o = o > 0.f ? o : 0.f;
  if (p.e.mask) o = p.e.mask[i] > 0.f ? o : 0.f;
  return o;
}

template <bool kVec, bool kPlain>
__global__ void __launch_bounds__(kThreads) sum_parts_wide_kernel(SumParams p)
{
  vlb::pdl_wait();
  constexpr int V = kVec ? 4 : 1;
  size_t const step = (size_t)gridDim.x * kThreads;
  for (size_t q = (size_t)blockIdx.x * kThreads + threadIdx.x; q * V < p.n; q += step) {
    float const* src = p.part + q * V;
    float s[V];
    if (kVec) { float4 const t = *reinterpret_cast<float4 const*>(src); s[0] = t.x; s[1] = t.y; s[2] = t.z; s[3] = t.w; }
    else s[0] = src[0];
    int k = 1;
    for (; k + 4 <= p.parts; k += 4) {
      if (kVec) {
        float4 t[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) t[j] = *reinterpret_cast<float4 const*>(src + (size_t)(k + j) * p.stride);
#pragma unroll
        for (int j = 0; j < 4; ++j) { s[0] += t[j].x; s[1] += t[j].y; s[2] += t[j].z; s[3] += t[j].w; }
      } else {
        float t[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) t[j] = src[(size_t)(k + j) * p.stride];
#pragma unroll
        for (int j = 0; j < 4; ++j) s[0] += t[j];
      }
    }
    for (; k < p.parts; ++k) {
      if (kVec) { float4 const t = *reinterpret_cast<float4 const*>(src + (size_t)k * p.stride); s[0] += t.x; s[1] += t.y; s[2] += t.z; s[3] += t.w; }
      else s[0] += src[(size_t)k * p.stride];
    }
    if (!kPlain) {
#pragma unroll
      for (int j = 0; j < V; ++j) s[j] = finish(p, s[j], q * V + j);
    }
    if (kVec) *reinterpret_cast<float4*>(p.out + q * V) = make_float4(s[0], s[V > 1 ? 1 : 0], s[V > 2 ? 2 : 0], s[V > 3 ? 3 : 0]);
    else p.out[q] = s[0];
  }
}

__global__ void __launch_bounds__(kThreads) sum_parts_narrow_kernel(SumParams p)
{
  vlb::pdl_wait();
  __shared__ float red[kThreads / 32][32];
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  size_t const i = (size_t)blockIdx.x * 32 + lane;
  float s = 0.f;
  if (i < p.n) {
    float const* const src = p.part + i;
    int k = warp;
    for (; k + 24 < p.parts; k += 32) {
      float t[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) t[j] = src[(size_t)(k + 8 * j) * p.stride];
#pragma unroll
      for (int j = 0; j < 4; ++j) s += t[j];
    }
    for (; k < p.parts; k += 8) s += src[(size_t)k * p.stride];
  }
  red[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && i < p.n) {
    s = red[0][lane];
#pragma unroll
    for (int w = 1; w < kThreads / 32; ++w) s += red[w][lane];
    p.out[i] = finish(p, s, i);
  }
}

}  // namespace

namespace vlb {

int sum_parts(vlb_ctx* ctx, float* out, float const* part, size_t n, size_t stride, int parts, SumEpilogue const& e)
{
  if (n == 0) return VLB_Success;
  SumParams p = {out, part, n, stride, parts, e};
  bool const plain = !e.bias && e.outMult == 0.f && e.inMult == 1.f && !e.relu && !e.mask;
  if (parts >= 12 && n < (size_t)ctx->smCount * 1024) {
    vlb::launch(ctx->stream, sum_parts_narrow_kernel, (unsigned)((n + 31) / 32), kThreads, 0, p);
  } else {
    bool const vec = n % 4 == 0 && stride % 4 == 0 && ((((uintptr_t)out) | ((uintptr_t)part)) & 15) == 0;
    unsigned const grid = grid_for(vec ? n / 4 : n, kThreads, ctx->smCount * 8);
    if (vec) { if (plain) vlb::launch(ctx->stream, sum_parts_wide_kernel<true, true>, grid, kThreads, 0, p);
               else       vlb::launch(ctx->stream, sum_parts_wide_kernel<true, false>, grid, kThreads, 0, p); }
    else     { if (plain) vlb::launch(ctx->stream, sum_parts_wide_kernel<false, true>, grid, kThreads, 0, p);
               else       vlb::launch(ctx->stream, sum_parts_wide_kernel<false, false>, grid, kThreads, 0, p); }
  }
  VLB_LAUNCHED(ctx, 1);
  return check_launch(ctx, "sum_parts");
}

}  // namespace vlb
