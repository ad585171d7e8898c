// Fully connected forward pass for a handful of images (reference bits/nnfullyconnected.cu:45-70): Y(K x N) = F'(K x V) X(V x N) + b,
// N <= 8.  Bound by the one pass over the weights: V contiguous floats per filter, read once with 16-byte loads.  A tensor-core tile
// would be 1/128 to 1/16 full and its operand staging slower than the loads (VGG-16's fc6, one image: 116 us through the
// tensor-memory kernel's row mode, fc7 37 us).  A block owns kRows filters, so that a value of X serves kRows weights from a
// register; its 256 threads share the V positions, and warp shuffles and one pass through shared memory add up: exact products,
// sums of V/256 terms per thread.
#include "conv_internal.cuh"

namespace {

constexpr int kThreads = 256;

template <int kN, int kRows, bool kVec>
__global__ void __launch_bounds__(kThreads) fc_rows_kernel(float* __restrict__ y, float const* __restrict__ x, float const* __restrict__ f,
                                                           float const* __restrict__ bias, int V, int K, int N, int relu)
{
  vlb::pdl_wait();
  __shared__ float red[kThreads / 32][kRows * kN];
  int const k0 = (int)blockIdx.x * kRows;
  float acc[kRows][kN];
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int n = 0; n < kN; ++n) acc[r][n] = 0.f;
  if (kVec) {
    int const V4 = V >> 2;
    float4 const* const x4 = reinterpret_cast<float4 const*>(x);
    float4 const* row[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) row[r] = reinterpret_cast<float4 const*>(f) + (size_t)min(k0 + r, K - 1) * V4;      // (a row past the last is computed and dropped)
#pragma unroll 2
    for (int i = threadIdx.x; i < V4; i += kThreads) {
      float4 w[kRows];
#pragma unroll
      for (int r = 0; r < kRows; ++r) w[r] = __ldcs(row[r] + i);
#pragma unroll
      for (int n = 0; n < kN; ++n) {
        if (n < N) {
          float4 const v = __ldg(x4 + (size_t)n * V4 + i);
#pragma unroll
          for (int r = 0; r < kRows; ++r) {
            acc[r][n] = fmaf(w[r].x, v.x, acc[r][n]); acc[r][n] = fmaf(w[r].y, v.y, acc[r][n]);
            acc[r][n] = fmaf(w[r].z, v.z, acc[r][n]); acc[r][n] = fmaf(w[r].w, v.w, acc[r][n]);
          }
        }
      }
    }
  } else {
    for (int i = threadIdx.x; i < V; i += kThreads) {
      float w[kRows];
#pragma unroll
      for (int r = 0; r < kRows; ++r) w[r] = __ldcs(f + (size_t)min(k0 + r, K - 1) * V + i);
#pragma unroll
      for (int n = 0; n < kN; ++n) {
        if (n < N) {
          float const v = __ldg(x + (size_t)n * V + i);
#pragma unroll
          for (int r = 0; r < kRows; ++r) acc[r][n] = fmaf(w[r], v, acc[r][n]);
        }
      }
    }
  }
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int n = 0; n < kN; ++n) {
      float s = acc[r][n];
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) red[warp][r * kN + n] = s;
    }
  __syncthreads();
  int const t = threadIdx.x, r = t / kN, n = t - r * kN;
  if (t < kRows * kN && k0 + r < K && n < N) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) s += red[w][t];
    if (bias) s += bias[k0 + r];
    if (relu) s = s > 0.f ? s : 0.f;
    y[(size_t)n * K + k0 + r] = s;
  }
}

template <int kN, int kRows>
void run(vlb_ctx* ctx, float* Y, float const* X, float const* F, float const* b, int V, int K, int N)
{
  bool const vec = V % 4 == 0 && ((((uintptr_t)X) | ((uintptr_t)F)) & 15) == 0;
  unsigned const grid = (unsigned)vlb::ceil_div(K, kRows);
  if (vec) vlb::launch(ctx->stream, fc_rows_kernel<kN, kRows, true>, grid, kThreads, 0, Y, X, F, b, V, K, N, ctx->fuseRelu);
  else     vlb::launch(ctx->stream, fc_rows_kernel<kN, kRows, false>, grid, kThreads, 0, Y, X, F, b, V, K, N, ctx->fuseRelu);
}

}  // namespace

namespace vlb {

// At most 8 images and at least 256 positions per filter; two rows per block instead of four where there are too few filters for the chip.  Both sides of
// the lines, us here / on the tensor cores (K filters of V positions):
//   V = 25088, K = 4096   one image 64 / 125, two 64 / 125, three 92 / 125, four 95 / 125, five 144 / 125, eight 201 / 125
//   V = 9216, K = 4096    one 25 / 65, four 35 / 65, five 47 / 65, eight 77 / 65
//   V = 4096, K = 4096    one 13 / 48, eight 30 / 49;  K = 1000: one 4.8 / 16.6, eight 9.9 / 17.1
//   V = 256, K = 256      one 1.5 / 12.1, eight 2.0 / 12.2
//   V = 128, K = 64       one 1.4 / 7.9, eight 1.9 / 8.1 (left to the tensor cores)
// Five to eight images of the longest rows are slower than they could be, with exact products.
int fc_fprop_small(vlb_ctx* ctx, ConvGeom const& g, float* Y, float const* X, float const* F, float const* b)
{
  int const V = g.FH * g.FW * g.FC, N = g.N;
  if (N > 8 || V < 256) return VLB_Unsupported;
  bool const few = g.K < 8 * ctx->smCount;
  if (N == 1)      { if (few) run<1, 2>(ctx, Y, X, F, b, V, g.K, N); else run<1, 4>(ctx, Y, X, F, b, V, g.K, N); }
  else if (N == 2) { if (few) run<2, 2>(ctx, Y, X, F, b, V, g.K, N); else run<2, 4>(ctx, Y, X, F, b, V, g.K, N); }
  else if (N <= 4) { if (few) run<4, 2>(ctx, Y, X, F, b, V, g.K, N); else run<4, 4>(ctx, Y, X, F, b, V, g.K, N); }
  else             { if (few) run<8, 2>(ctx, Y, X, F, b, V, g.K, N); else run<8, 4>(ctx, Y, X, F, b, V, g.K, N); }
  ctx->reluDone = ctx->fuseRelu;
  VLB_LAUNCHED(ctx, 1);
  return check_launch(ctx, "fc_fprop_small");
}

}  // namespace vlb
