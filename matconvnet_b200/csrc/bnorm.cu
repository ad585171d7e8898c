// Batch normalisation (vl::nn::BatchNorm, reference bits/nnbnorm.hpp:22-59;
// CPU definition bits/nnbnorm.cu:46-164).
//
// HBM-bound.  The regular entry points run one fused launch (bnorm_fused_kernel below: reduce, derive the
// coefficients, apply, all by the cluster that owns the channel); forward with given moments and the
// allocation-free entry point use the separate passes:
//   1. reduce: per channel sum(x), sum(x^2) [, sum(dy*x), sum(dy)].  A channel is split
//      across a thread-block CLUSTER of kCluster CTAs (C alone would leave most of the
//      148 SMs idle: the reference launches exactly C blocks, bits/nnbnorm_gpu.cu:1113).
//      Each CTA sweeps its share with 128-bit loads, reduces with warp shuffles, and the
//      cluster's rank-0 CTA gathers the kCluster partials through distributed shared
//      memory in rank order and finishes the per-channel arithmetic in the reference's
//      order (bits/nnbnorm.cu:126-133).  No scratch memory, no atomics, deterministic.
//   2. apply: y or dx, element-wise with the per-channel coefficients.
// Algorithmic traffic of backward: 8*m*C bytes (pass 1) + 12*m*C bytes (pass 2), m = H*W*N.
#include "common.cuh"
#include <cooperative_groups.h>
#include <math.h>
#include <type_traits>

namespace cg = cooperative_groups;

namespace {

constexpr int kCluster = 8;
constexpr int kThreads = 256;

// stats layout handed from pass 1 to pass 2 (device memory, 4*C floats):
// [0,C) mean, [C,2C) sigma, [2C,3C) dgamma, [3C,4C) dbeta

// Position of a thread in its channel's items (float4s or floats: item i is element i % per of image i / per), moved by a fixed stride without
// dividing.
struct Walk {
  size_t off;                        // of the item, in floats
  size_t stride, wrap;               // of one move, and what is added when that leaves the plane
  int q, dq, per;
  __device__ Walk(int first, int step, int per_, int width, int c, int C, int WH) : per(per_)
  {
    int const n = first / per;
    q = first - n * per;
    off = ((size_t)n * C + c) * (size_t)WH + (size_t)width * q;
    int const dn = step / per;
    dq = step - dn * per;
    stride = (size_t)dn * C * WH + (size_t)width * dq;
    wrap = (size_t)C * WH - (size_t)width * per;
  }
  __device__ __forceinline__ void move()
  {
    q += dq; off += stride;
    if (q >= per) { q -= per; off += wrap; }
  }
};

// kMode 0: sums of x, x^2.  1: and of dy*x, dy.  2: the latter two alone.  Four values among themselves first.
__device__ __forceinline__ float sum4(float4 a) { return (a.x + a.y) + (a.z + a.w); }
__device__ __forceinline__ float dot4(float4 a, float4 b) { return fmaf(a.x, b.x, a.y * b.y) + fmaf(a.z, b.z, a.w * b.w); }
template <int kMode> __device__ __forceinline__ void add4(float (&acc)[4], float4 x, float4 dy)
{
  if (kMode != 2) { acc[0] += sum4(x); acc[1] += dot4(x, x); }
  if (kMode != 0) { acc[2] += dot4(dy, x); acc[3] += sum4(dy); }
}

// The sums over a thread's `mine` items from w on (kVec: float4s).  In steps -- four values, eight items, all -- for with one block per channel a
// thread has eight times the terms it has with eight, and one running sum over all of them loses the digits that eight blocks keep
// (28 x 28 x 512 x 64, the mean of inputs around zero: 2.7e-7 off in one sum, 1.4e-7 with eight blocks, 1.3e-7 in steps; the groups of
// loads that this makes: 60 -> 53 us forward, 82 as before backward).
template <int kMode, bool kVec>
__device__ __forceinline__ void sum_items(float (&acc)[4], Walk w, int mine, float const* x, float const* dy)
{
  auto eight = [&](auto whole, int left) {
    float run[4] = {0.f, 0.f, 0.f, 0.f};
    int k = 0;
    auto next = [&](auto item, float const* p) {
      using Item = decltype(item);
      return decltype(whole)::value || k < left ? *reinterpret_cast<Item const*>(p + w.off) : Item{};
    };
    if (kVec) {
#pragma unroll
      for (k = 0; k < 8; ++k) {
        float4 const d = kMode != 0 ? next(float4{}, dy) : float4{};
        add4<kMode>(run, next(float4{}, x), d);
        w.move();
      }
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float v[4], d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          k = 4 * h + j;
          d[j] = kMode != 0 ? next(0.f, dy) : 0.f; v[j] = next(0.f, x);
          w.move();
        }
        add4<kMode>(run, make_float4(v[0], v[1], v[2], v[3]), make_float4(d[0], d[1], d[2], d[3]));
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] += run[j];
  };
  int left = mine;
  for (; left >= 8; left -= 8) eight(std::true_type{}, 8);
  if (left > 0) eight(std::false_type{}, left);
}

// Moments and derivatives of the parameters (backward pass of the entry point that may not allocate).
template <bool kVec>
__global__ void __cluster_dims__(1, kCluster, 1) __launch_bounds__(kThreads)
bnorm_reduce_kernel(float* __restrict__ momentsOut,   // 2*C
                    float* __restrict__ dgOut, float* __restrict__ dbOut,
                    float const* __restrict__ x, float const* __restrict__ dy,
                    int WH, int C, int N, float eps)
{
  vlb::pdl_wait();
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ float part[4];
  __shared__ float warpRed[kThreads / 32][4];
  int c = blockIdx.x;
  int rank = (int)cluster.block_rank();   // the cluster spans grid y
  float acc[4] = {0.f, 0.f, 0.f, 0.f};

  // Work items: (image n, chunk of the plane).  Item i of this channel goes to CTA (i / kThreads) % kCluster.
  int const per = kVec ? WH >> 2 : WH, step = kCluster * kThreads, first = rank * kThreads + (int)threadIdx.x;
  long long const items = (long long)N * per;
  int const mine = first < items ? (int)((items - first + step - 1) / step) : 0;
  sum_items<1, kVec>(acc, Walk(first, step, per, kVec ? 4 : 1, c, C, WH), mine, x, dy);

#pragma unroll
  for (int j = 0; j < 4; ++j)
    for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { for (int j = 0; j < 4; ++j) warpRed[warp][j] = acc[j]; }
  __syncthreads();
  if (threadIdx.x < 4) {
    float s = 0.f;
    for (int w = 0; w < kThreads / 32; ++w) s += warpRed[w][threadIdx.x];
    part[threadIdx.x] = s;
  }
  cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    float tot[4] = {0.f, 0.f, 0.f, 0.f};
    for (int r = 0; r < kCluster; ++r) {
      float const* remote = cluster.map_shared_rank(part, r);
      for (int j = 0; j < 4; ++j) tot[j] += remote[j];
    }
    float mass = (float)((long long)WH * N);
    // reference bits/nnbnorm.cu:65-70
    float mean = __fdiv_rn(tot[0], mass);
    float s2 = __fadd_rn(__fdiv_rn(tot[1], mass), -__fmul_rn(mean, mean));
    s2 = fmaxf(s2, 0.f);
    float sigma = __fsqrt_rn(__fadd_rn(s2, eps));
    momentsOut[c] = mean; momentsOut[c + C] = sigma;
    // reference bits/nnbnorm.cu:94-98
    dbOut[c] = tot[3];
    dgOut[c] = __fdiv_rn(__fadd_rn(tot[2], -__fmul_rn(mean, tot[3])), sigma);
  }
  cluster.sync();   // keep every CTA's shared memory alive until rank 0 has read it
}

// kMode 0: k = {mean, G1, b, -}; else {mean, db/m, G1, G2}
template <int kMode> __device__ __forceinline__ float apply_item(float x, float dy, float4 k, int relu)
{
  if (kMode != 0) return __fadd_rn(__fmul_rn(k.z, __fadd_rn(dy, -k.y)), -__fmul_rn(k.w, __fadd_rn(x, -k.x)));
  float const o = __fadd_rn(__fmul_rn(k.y, __fadd_rn(x, -k.x)), k.z);
  return relu && !(o > 0.f) ? 0.f : o;
}
template <int kMode> __device__ __forceinline__ float4 apply_item(float4 x, float4 dy, float4 k, int relu)
{
  return make_float4(apply_item<kMode>(x.x, dy.x, k, relu), apply_item<kMode>(x.y, dy.y, k, relu), apply_item<kMode>(x.z, dy.z, k, relu),
                     apply_item<kMode>(x.w, dy.w, k, relu));
}

// One launch for the whole operator: the cluster that reduced a channel also applies it.
// After the reduction rank 0 derives the channel's coefficients into its shared memory, the other
// CTAs read them through distributed shared memory, and every CTA sweeps the same items again --
// they are still in L2 (a channel's x and dy, 8*m bytes, times the clusters in flight), so DRAM sees
// x and dy once and the result once: 12*m*C bytes backward, 8*m*C forward.  What binds beside the traffic is the two
// meetings of a cluster, and the issue of instructions: a block must have enough to do between the meetings, and no item divides.
// Clusters of eight with a 64-bit division per item: 28 x 28 x 512 x 64 took 70 us forward and 89 us backward, x 32 images 43 and 66, 28 x 28 x 128 x 64
// 21 and 26; now 53 and 82, 26 and 43, 14 and 20 (at copy speed 32 and 48, 16 and 24, 8 and 12).  Holding the items in registers or shared memory between
// the two sweeps was slower: it costs the blocks that hide one another's meetings.
constexpr int kFusedThreads = 256;
// Six blocks per SM are asked for where planes are read float by float in the backward pass (48 registers otherwise, five blocks: 55 x 55 x 96 x 16 24.5 us, with
// six and a few spills 19.3; forward and float4 reads lose 10 to 40% by it).
// kMode 0: forward, moments computed.  1: backward, moments computed.  2: backward, moments given.
template <int kMode, bool kVec, int kCl>
__global__ void __cluster_dims__(1, kCl, 1) __launch_bounds__(kFusedThreads, !kVec && kMode != 0 ? 6 : 0)
bnorm_fused_kernel(float* __restrict__ out,            // y or dx
                   float* __restrict__ momentsOut,     // 2*C or nullptr
                   float* __restrict__ dgOut, float* __restrict__ dbOut,
                   float const* __restrict__ momentsIn,  // mode 2
                   float const* __restrict__ x, float const* __restrict__ dy,
                   float const* __restrict__ g, float const* __restrict__ b,
                   int WH, int C, int N, float eps, int relu)      // relu (forward): the stored value is max(y, 0)
{
  vlb::pdl_wait();
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ float part[4];
  __shared__ float coef[4];
  __shared__ float warpRed[kFusedThreads / 32][4];
  int const c = blockIdx.x;
  int const rank = (int)cluster.block_rank();   // the cluster spans grid y
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  using Item = std::conditional_t<kVec, float4, float>;
  int const per = kVec ? WH >> 2 : WH;                                  // items of a plane
  int const step = kCl * kFusedThreads, first = rank * kFusedThreads + (int)threadIdx.x;
  long long const items = (long long)N * per;
  auto xAt = [&](size_t off) { return *reinterpret_cast<Item const*>(x + off); };
  auto dyAt = [&](size_t off) { return *reinterpret_cast<Item const*>(dy + off); };

  int const mine = first < items ? (int)((items - first + step - 1) / step) : 0;
  Walk const w0(first, step, per, kVec ? 4 : 1, c, C, WH);
  sum_items<kMode, kVec>(acc, w0, mine, x, dy);

#pragma unroll
  for (int j = 0; j < 4; ++j)
    for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
  int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { for (int j = 0; j < 4; ++j) warpRed[warp][j] = acc[j]; }
  __syncthreads();
  if (threadIdx.x < 4) {
    float s = 0.f;
    for (int w = 0; w < kFusedThreads / 32; ++w) s += warpRed[w][threadIdx.x];
    part[threadIdx.x] = s;
  }
  cluster.sync();
  // rank 0 gathers the partial sums of all ranks through distributed shared memory -- 32 threads fetch one value each, so that
  // the remote reads are one round trip instead of 32 -- and thread 0 adds them in rank order
  __shared__ float gath[kCl][4];
  if (rank == 0 && threadIdx.x < kCl * 4) {
    int const r = threadIdx.x >> 2, j = threadIdx.x & 3;
    gath[r][j] = cluster.map_shared_rank(part, r)[j];
  }
  if (rank == 0) __syncwarp();
  if (rank == 0 && threadIdx.x == 0) {
    float tot[4] = {0.f, 0.f, 0.f, 0.f};
    for (int r = 0; r < kCl; ++r)
      for (int j = 0; j < 4; ++j) tot[j] += gath[r][j];
    float const mass = (float)((long long)WH * N);
    float mean, sigma;
    if (kMode == 2) { mean = momentsIn[c]; sigma = momentsIn[c + C]; }
    else {
      // reference bits/nnbnorm.cu:65-70
      mean = __fdiv_rn(tot[0], mass);
      float s2 = __fadd_rn(__fdiv_rn(tot[1], mass), -__fmul_rn(mean, mean));
      s2 = fmaxf(s2, 0.f);
      sigma = __fsqrt_rn(__fadd_rn(s2, eps));
      if (momentsOut) { momentsOut[c] = mean; momentsOut[c + C] = sigma; }
    }
    float const G1 = __fdiv_rn(g[c], sigma);
    if (kMode != 0) {
      // reference bits/nnbnorm.cu:94-98, 148-153
      float const dbv = tot[3];
      float const dgv = __fdiv_rn(__fadd_rn(tot[2], -__fmul_rn(mean, tot[3])), sigma);
      dbOut[c] = dbv;
      dgOut[c] = dgv;
      coef[0] = mean; coef[1] = __fdiv_rn(dbv, mass); coef[2] = G1;
      coef[3] = __fdiv_rn(__fmul_rn(G1, dgv), __fmul_rn(mass, sigma));
    } else {
      // reference bits/nnbnorm.cu:192-196
      coef[0] = mean; coef[1] = G1; coef[2] = b[c]; coef[3] = 0.f;
    }
  }
  cluster.sync();
  float k0, k1, k2, k3;
  {
    float const* rc = cluster.map_shared_rank(coef, 0);
    k0 = rc[0]; k1 = rc[1]; k2 = rc[2]; k3 = rc[3];
  }
  // (rank 0's shared memory has to outlive these reads: the cluster meets once more at the very end, where nobody waits long)

  float4 const k = make_float4(k0, k1, k2, k3);
  Walk w = w0;
#pragma unroll 8
  for (int i = 0; i < mine; ++i) {
    Item const d = kMode != 0 ? dyAt(w.off) : Item{};
    *reinterpret_cast<Item*>(out + w.off) = apply_item<kMode>(xAt(w.off), d, k, relu);
    w.move();
  }
  cluster.sync();   // every CTA has read rank 0's coefficients long ago; rank 0 may exit
}

// Blocks per channel: as few as give every SM three (of the eight that fit), for every block then has the most to do between the meetings.
template <int kMode>
void launch_fused(vlb_ctx* ctx, bool vec, float* out, float* momOut, float* dg, float* db, float const* momIn,
                 float const* x, float const* dy, float const* g, float const* b, int WH, int C, int N, float eps, int relu = 0)
{
  int cl = 1;
  while (cl < 8 && (long long)C * cl < 3LL * ctx->smCount) cl *= 2;
  auto go = [&](auto v, auto n) {
    vlb::launch(ctx->stream, bnorm_fused_kernel<kMode, decltype(v)::value, decltype(n)::value>, dim3(C, decltype(n)::value), kFusedThreads, 0, out, momOut, dg, db,
                momIn, x, dy, g, b, WH, C, N, eps, relu);
  };
  auto pick = [&](auto v) {
    if (cl == 1) return go(v, std::integral_constant<int, 1>{});
    if (cl == 2) return go(v, std::integral_constant<int, 2>{});
    if (cl == 4) return go(v, std::integral_constant<int, 4>{});
    return go(v, std::integral_constant<int, 8>{});
  };
  if (vec) pick(std::true_type{}); else pick(std::false_type{});
  VLB_LAUNCHED(ctx, 1);
}

// Per-channel coefficients, computed once so that pass 2 is pure multiply/add.
// forward: cf = {mean, g/sigma, b, -}   (reference bits/nnbnorm.cu:192-196)
// backward: cf = {mean, db/m, G1 = g/sigma, G2 = G1*dg/(m*sigma)}   (bits/nnbnorm.cu:148-153)
__global__ void bnorm_coef_kernel(float4* __restrict__ cf, float const* __restrict__ moments,
                                  float const* __restrict__ g, float const* __restrict__ b,
                                  float const* __restrict__ dg, float const* __restrict__ db, int C, float mass)
{
  vlb::pdl_wait();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  float mean = moments[c], sigma = moments[c + C];
  float G1 = __fdiv_rn(g[c], sigma);
  if (dg) {
    float muz = __fdiv_rn(db[c], mass);
    float G2 = __fdiv_rn(__fmul_rn(G1, dg[c]), __fmul_rn(mass, sigma));
    cf[c] = make_float4(mean, muz, G1, G2);
  } else {
    cf[c] = make_float4(mean, G1, b[c], 0.f);
  }
}

// y = g/sigma * (x - mean) + b (reference bits/nnbnorm.cu:192-203)
template <bool kVec>
__global__ void bnorm_fwd_apply_kernel(float* __restrict__ y, float const* __restrict__ x,
                                       float4 const* __restrict__ cf, int WH, int C, size_t total)
{
  vlb::pdl_wait();
  size_t stride = (size_t)gridDim.x * blockDim.x;
  if (kVec) {
    size_t total4 = total >> 2;
    int WH4 = WH >> 2;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total4; i += stride) {
      int c = (int)((i / WH4) % C);
      float4 k = __ldg(cf + c);
      float4 v = reinterpret_cast<float4 const*>(x)[i];
      v.x = __fadd_rn(__fmul_rn(k.y, __fadd_rn(v.x, -k.x)), k.z);
      v.y = __fadd_rn(__fmul_rn(k.y, __fadd_rn(v.y, -k.x)), k.z);
      v.z = __fadd_rn(__fmul_rn(k.y, __fadd_rn(v.z, -k.x)), k.z);
      v.w = __fadd_rn(__fmul_rn(k.y, __fadd_rn(v.w, -k.x)), k.z);
      reinterpret_cast<float4*>(y)[i] = v;
    }
  } else {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
      int c = (int)((i / WH) % C);
      float4 k = __ldg(cf + c);
      y[i] = __fadd_rn(__fmul_rn(k.y, __fadd_rn(x[i], -k.x)), k.z);
    }
  }
}

// dx = G1*(dy - db/m) - G2*(x - mean) (reference bits/nnbnorm.cu:136-164)
template <bool kVec>
__global__ void bnorm_bwd_apply_kernel(float* __restrict__ dx, float const* __restrict__ x,
                                       float const* __restrict__ dy, float4 const* __restrict__ cf,
                                       int WH, int C, size_t total)
{
  vlb::pdl_wait();
  size_t stride = (size_t)gridDim.x * blockDim.x;
  if (kVec) {
    size_t total4 = total >> 2;
    int WH4 = WH >> 2;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total4; i += stride) {
      int c = (int)((i / WH4) % C);
      float4 k = __ldg(cf + c);
      float4 xv = reinterpret_cast<float4 const*>(x)[i];
      float4 dv = reinterpret_cast<float4 const*>(dy)[i];
      float4 o;
      o.x = __fadd_rn(__fmul_rn(k.z, __fadd_rn(dv.x, -k.y)), -__fmul_rn(k.w, __fadd_rn(xv.x, -k.x)));
      o.y = __fadd_rn(__fmul_rn(k.z, __fadd_rn(dv.y, -k.y)), -__fmul_rn(k.w, __fadd_rn(xv.y, -k.x)));
      o.z = __fadd_rn(__fmul_rn(k.z, __fadd_rn(dv.z, -k.y)), -__fmul_rn(k.w, __fadd_rn(xv.z, -k.x)));
      o.w = __fadd_rn(__fmul_rn(k.z, __fadd_rn(dv.w, -k.y)), -__fmul_rn(k.w, __fadd_rn(xv.w, -k.x)));
      reinterpret_cast<float4*>(dx)[i] = o;
    }
  } else {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
      int c = (int)((i / WH) % C);
      float4 k = __ldg(cf + c);
      dx[i] = __fadd_rn(__fmul_rn(k.z, __fadd_rn(dy[i], -k.y)), -__fmul_rn(k.w, __fadd_rn(x[i], -k.x)));
    }
  }
}

bool vec_ok(int WH, void const* a, void const* b, void const* c)
{
  uintptr_t bits = (uintptr_t)a | (uintptr_t)b | (uintptr_t)c;
  return (WH % 4 == 0) && (bits & 15) == 0;
}

int validate(vlb_ctx* ctx, int H, int W, int C, int N)
{
  VLB_REQUIRE(ctx, H > 0 && W > 0 && C > 0 && N > 0, "bnorm: empty input");
  VLB_REQUIRE(ctx, (long long)H * W * N < (1LL << 31), "bnorm: H*W*N too large");
  return VLB_Success;
}

// Scratch layout (context workspace): [0, 2C) moments when the caller passes none,
// then 4C floats of per-channel coefficients (16-byte aligned).
static float* scratch(vlb_ctx* ctx, int C, float4** cf)
{
  size_t momBytes = ((sizeof(float) * 2 * (size_t)C + 255) / 256) * 256;
  char* ws = (char*)vlb::workspace(ctx, momBytes + sizeof(float4) * (size_t)C);
  if (!ws) return nullptr;
  *cf = (float4*)(ws + momBytes);
  return (float*)ws;
}

static int forward_common(vlb_ctx* ctx, float* Y, float* momOut, float const* momIn, float const* X, float const* g,
                          float const* b, int H, int W, int C, int N, double eps, char const* where, int relu = 0)
{
  int rc = validate(ctx, H, W, C, N);
  if (rc) return rc;
  VLB_REQUIRE(ctx, Y && X && g && b, "bnorm_forward: null tensor");
  float4* cf = nullptr;
  float* ownMom = scratch(ctx, C, &cf);
  if (!ownMom) return vlb::pass_error(ctx, ctx->lastError, where);
  int WH = H * W;
  float const* mom = momIn;
  if (!momIn) {
    // moments computed and applied by the same clusters (the reference computes them into the context
    // workspace when the caller does not ask for them, bits/nnbnorm.cu:233-240)
    launch_fused<0>(ctx, vec_ok(WH, Y, X, X), Y, momOut, nullptr, nullptr, nullptr, X, nullptr, g, b, WH, C, N, (float)eps, relu);
    return vlb::check_launch(ctx, where);
  }
  vlb::launch(ctx->stream, bnorm_coef_kernel, vlb::ceil_div(C, 256), 256, 0, cf, mom, g, b, nullptr, nullptr, C, 0.f);
  size_t total = (size_t)WH * C * N;
  bool vec = vec_ok(WH, Y, X, X);
  unsigned grid = vlb::grid_for(vec ? total / 4 : total, kThreads, ctx->smCount * 16);
  if (vec) vlb::launch(ctx->stream, bnorm_fwd_apply_kernel<true>, grid, kThreads, 0, Y, X, cf, WH, C, total);
  else     vlb::launch(ctx->stream, bnorm_fwd_apply_kernel<false>, grid, kThreads, 0, Y, X, cf, WH, C, total);
  VLB_LAUNCHED(ctx, 2);
  return vlb::check_launch(ctx, where);
}

static int backward_common(vlb_ctx* ctx, float* dX, float* dG, float* dB, float* momOut, float const* momIn,
                           float const* X, float const* g, float const* dY, int H, int W, int C, int N,
                           double eps, char const* where)
{
  int rc = validate(ctx, H, W, C, N);
  if (rc) return rc;
  VLB_REQUIRE(ctx, dX && dG && dB && X && g && dY, "bnorm_backward: null tensor");
  int WH = H * W;
  bool vec = vec_ok(WH, X, dY, dX);
  if (!momIn) launch_fused<1>(ctx, vec, dX, momOut, dG, dB, nullptr, X, dY, g, nullptr, WH, C, N, (float)eps);
  else        launch_fused<2>(ctx, vec, dX, nullptr, dG, dB, momIn, X, dY, g, nullptr, WH, C, N, (float)eps);
  return vlb::check_launch(ctx, where);
}

}  // namespace

extern "C" {

int vlb_bnorm_forward_moment(vlb_ctx* ctx, float* Y, float const* moments, float const* X, float const* g,
                             float const* b, int H, int W, int C, int N, double eps)
{
  if (!ctx) return VLB_IllegalArgument;
  VLB_REQUIRE(ctx, moments, "bnorm_forward_moment: null moments");
  return forward_common(ctx, Y, nullptr, moments, X, g, b, H, W, C, N, eps, "vlb_bnorm_forward_moment");
}

int vlb_bnorm_forward(vlb_ctx* ctx, float* Y, float* moments, float const* X, float const* g, float const* b,
                      int H, int W, int C, int N, double eps)
{
  if (!ctx) return VLB_IllegalArgument;
  return forward_common(ctx, Y, moments, nullptr, X, g, b, H, W, C, N, eps, "vlb_bnorm_forward");
}

int vlb_bnorm_relu_forward(vlb_ctx* ctx, float* Y, float* moments, float const* X, float const* g, float const* b,
                           int H, int W, int C, int N, double eps)
{
  if (!ctx) return VLB_IllegalArgument;
  return forward_common(ctx, Y, moments, nullptr, X, g, b, H, W, C, N, eps, "vlb_bnorm_relu_forward", 1);
}

int vlb_bnorm_backward(vlb_ctx* ctx, float* dX, float* dG, float* dB, float* moments, float const* X,
                       float const* g, float const* b, float const* dY, int H, int W, int C, int N, double eps)
{
  if (!ctx) return VLB_IllegalArgument;
  (void)b;
  return backward_common(ctx, dX, dG, dB, moments, nullptr, X, g, dY, H, W, C, N, eps, "vlb_bnorm_backward");
}

int vlb_bnorm_backward_moment(vlb_ctx* ctx, float* dX, float* dG, float* dB, float const* moments, float const* X,
                              float const* g, float const* b, float const* dY, int H, int W, int C, int N, double eps)
{
  if (!ctx) return VLB_IllegalArgument;
  (void)b;
  VLB_REQUIRE(ctx, moments, "bnorm_backward_moment: null moments");
  return backward_common(ctx, dX, dG, dB, nullptr, moments, X, g, dY, H, W, C, N, eps, "vlb_bnorm_backward_moment");
}

}  // extern "C"

// ====================================================================================
// Batch-norm backward for callers that must not allocate
// ====================================================================================
// Some hosts hand the whole device to an allocator of their own (MATLAB's gpuArray pool, a
// serving process with a fixed arena) or run inside a latency budget that a cudaMalloc --
// which synchronises the whole device -- would break.  Such callers cannot create a vlb_ctx
// (it allocates) nor let the scratch buffer grow.  For them the two per-channel scratch arrays
// of the backward pass live in a fixed array inside the library image: moments (2*C floats,
// used when the caller passes none) and the coefficients {mean, db/m, G1, G2} (4*C floats).
constexpr int kNoAllocMaxChannels = 4096;
static __device__ __align__(256) float g_bnormNoAllocScratch[6 * kNoAllocMaxChannels];   // 96 KB per GPU that loads the library

namespace {

// Device address of the array above, one per device.  The array's name is only a stand-in in
// host code; the address a kernel can use comes from cudaGetSymbolAddress, asked once per
// device with that device current.
constexpr int kMaxDevices = 64;
float* g_noAllocPtr[kMaxDevices] = {};

void report(char* errbuf, size_t errlen, char const* msg)
{
  if (errbuf && errlen) snprintf(errbuf, errlen, "%s", msg);
}

}  // namespace

extern "C" int vlb_bnorm_backward_noalloc(void* cudaStream, float* dX, float* dG, float* dB, float* moments,
                                          float const* X, float const* g, float const* dY, int H, int W, int C,
                                          int N, double eps, char* errbuf, size_t errlen)
{
  if (!dX || !dG || !dB || !X || !g || !dY) { report(errbuf, errlen, "bnorm_backward_noalloc: null tensor"); return VLB_IllegalArgument; }
  if (H <= 0 || W <= 0 || C <= 0 || N <= 0 || (long long)H * W * N >= (1LL << 31)) {
    report(errbuf, errlen, "bnorm_backward_noalloc: empty or oversized input");
    return VLB_IllegalArgument;
  }
  if (C > kNoAllocMaxChannels) {
    report(errbuf, errlen, "bnorm_backward_noalloc: more than 4096 channels do not fit the built-in scratch array; "
                           "use vlb_bnorm_backward with a context");
    return VLB_IllegalArgument;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) { report(errbuf, errlen, "bnorm_backward_noalloc: no usable current device"); return VLB_Cuda; }
  if (!g_noAllocPtr[dev]) {
    // first call on this device: the kernels are built for sm_100a only, so refuse anything else before a launch
    // could fail and leave its error pending for the host process; then resolve the array's device address (no
    // allocation takes place).  Two host threads making their first call on one device at the same time would both
    // do this and store the same address: harmless, but the entry point is meant for one calling thread per device.
    int major = 0;
    e = cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
    if (e != cudaSuccess) { cudaGetLastError(); report(errbuf, errlen, cudaGetErrorString(e)); return VLB_Cuda; }
    if (major != 10) { report(errbuf, errlen, "bnorm_backward_noalloc: the kernels are built for sm_100a only"); return VLB_Unsupported; }
    float* p = nullptr;
    e = cudaGetSymbolAddress((void**)&p, g_bnormNoAllocScratch);
    if (e != cudaSuccess || !p) {
      cudaGetLastError();
      report(errbuf, errlen, cudaGetErrorString(e));
      return VLB_Cuda;
    }
    g_noAllocPtr[dev] = p;
  }
  cudaStream_t stream = (cudaStream_t)cudaStream;
  float* ownMom = g_noAllocPtr[dev];
  float4* cf = reinterpret_cast<float4*>(g_noAllocPtr[dev] + 2 * kNoAllocMaxChannels);
  float* mom = moments ? moments : ownMom;
  // Nothing in the scratch has to start from zero: pass 1 writes every moment and pass 1b every
  // coefficient of channels [0, C) before pass 2 reads them; entries beyond C keep an earlier call's
  // values and are never read.
  int WH = H * W;
  bool vec = vec_ok(WH, X, dY, dX);
  dim3 grid(C, kCluster);
  if (vec) vlb::launch(stream, bnorm_reduce_kernel<true>, grid, kThreads, 0, mom, dG, dB, X, dY, WH, C, N, (float)eps);
  else     vlb::launch(stream, bnorm_reduce_kernel<false>, grid, kThreads, 0, mom, dG, dB, X, dY, WH, C, N, (float)eps);
  float mass = (float)((long long)WH * N);
  vlb::launch(stream, bnorm_coef_kernel, vlb::ceil_div(C, 256), 256, 0, cf, mom, g, nullptr, dG, dB, C, mass);
  size_t total = (size_t)WH * C * N;
  unsigned blocks = vlb::grid_for(vec ? total / 4 : total, kThreads, 148 * 16);
  if (vec) vlb::launch(stream, bnorm_bwd_apply_kernel<true>, blocks, kThreads, 0, dX, X, dY, cf, WH, C, total);
  else     vlb::launch(stream, bnorm_bwd_apply_kernel<false>, blocks, kThreads, 0, dX, X, dY, cf, WH, C, total);
  e = cudaPeekAtLastError();
  if (e != cudaSuccess) {
    report(errbuf, errlen, cudaGetErrorString(e));
    cudaGetLastError();      // reported once: cleared so that later calls are not blamed for it
    return VLB_Cuda;
  }
  return VLB_Success;
}
