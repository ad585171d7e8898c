// Blocks of the reference's other ImageNet models (AlexNet, VGG-F/M/S: examples/imagenet/cnn_imagenet_init.m:148-154,
// 392-396): cross-channel local response normalisation (vl::nn::LRN, reference bits/nnnormalize.hpp:20-44, CPU definition
// bits/nnnormalize.cu:143-400), softmax (matlab/vl_nnsoftmax.m) and dropout (matlab/vl_nndropout.m).
//
// LRN: y_t = x_t * L_t^-beta with L_t = kappa + alpha * sum of x_q^2 over the channels q in [t - m1, t + m2] that exist,
// m1 = (normDepth - 1) / 2, m2 = normDepth - m1 - 1.  One thread per (pixel, image) walks the channels, a stride of one
// plane apart, so a warp reads and writes whole lines; the window sum slides as in the CPU loop (add the square that
// enters, subtract the one that leaves).  Backward follows the CPU's three sweeps (bits/nnnormalize.cu:296-383): the term
// dz_t * L_t^-beta and the running integral over the channels of x_t * 2*alpha*beta * dz_t * L_t^(-beta-1) -- kept in the
// context's scratch, written and read back by the same thread -- then the difference of the integral over the window.
// The reference's CPU code evaluates the power with a cubic approximation of log2 and exp2 (VL_NNNORMALIZE_FAST,
// bits/nnnormalize.cu:49-125); here it is powf, which the reference's own GPU kernels use (bits/nnnormalize_gpu.cu:27-66).
#include "common.cuh"
#include <math.h>

namespace {

constexpr int kThreads = 256;

struct LrnParams {
  int P, C, N, m1, m2;
  float kappa, alpha, beta;
  int relu;            // backward: X is the output of a ReLU, dX is zero where it is not positive
};

__global__ void lrn_forward_kernel(float* __restrict__ y, float const* __restrict__ x, LrnParams p)
{
  vlb::pdl_wait();
  size_t const total = (size_t)p.P * p.N, step = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
    size_t const n = i / p.P, pix = i - n * p.P;
    float const* xp = x + pix + (size_t)p.P * p.C * n;
    float* yp = y + pix + (size_t)p.P * p.C * n;
    float acc = 0.f;
    for (int t = -p.m2; t < p.C; ++t) {
      int const tm = t - p.m1 - 1, tp = t + p.m2;
      float const am = tm >= 0 ? xp[(size_t)p.P * tm] : 0.f, ap = tp < p.C ? xp[(size_t)p.P * tp] : 0.f;
      acc += ap * ap - am * am;
      if (t >= 0) yp[(size_t)p.P * t] = xp[(size_t)p.P * t] * powf(p.kappa + p.alpha * acc, -p.beta);
    }
  }
}

__global__ void lrn_backward_kernel(float* __restrict__ dx, float* __restrict__ integral, float const* __restrict__ x,
                                    float const* __restrict__ dz, LrnParams p)
{
  vlb::pdl_wait();
  size_t const total = (size_t)p.P * p.N, step = (size_t)gridDim.x * blockDim.x;
  float const ab2 = 2.f * p.alpha * p.beta;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
    size_t const n = i / p.P, pix = i - n * p.P, off = pix + (size_t)p.P * p.C * n;
    float const* xp = x + off;
    float const* zp = dz + off;
    float* dp = dx + off;
    float* ip = integral + off;
    float acc = 0.f, run = 0.f;
    for (int t = -p.m2; t < p.C; ++t) {
      int const tm = t - p.m1 - 1, tp = t + p.m2;
      float const am = tm >= 0 ? xp[(size_t)p.P * tm] : 0.f, ap = tp < p.C ? xp[(size_t)p.P * tp] : 0.f;
      acc += ap * ap - am * am;
      if (t >= 0) {
        float const L = p.kappa + p.alpha * acc;
        float const temp1 = zp[(size_t)p.P * t] * powf(L, -p.beta);
        float const temp2 = xp[(size_t)p.P * t] * ab2 * temp1 / L;
        dp[(size_t)p.P * t] = temp1;
        run += temp2;
        ip[(size_t)p.P * t] = run;
      }
    }
    // the sum of temp2 over the channels q whose window holds t: q in [t - m2, t + m1]
    for (int t = 0; t < p.C; ++t) {
      int const q1 = t - p.m2 - 1, q2 = min(t + p.m1, p.C - 1);
      float s = ip[(size_t)p.P * q2];
      if (q1 >= 0) s -= ip[(size_t)p.P * q1];
      float const xt = xp[(size_t)p.P * t], d = dp[(size_t)p.P * t] - s * xt;
      dp[(size_t)p.P * t] = p.relu && !(xt > 0.f) ? 0.f : d;
    }
  }
}

// L^-beta and 1 / L.  kThreeQuarters: beta = 0.75 (every LRN layer of the reference's model builders), from the hardware's approximations r of
// L^-1/2 and s of r^1/2 and their residuals, which fused multiply-adds give exactly: with e = 1 - L r^2 and f = r - s^2 (both of the order of 2^-22)
// L^-3/4 = r s (1 + 3/4 e) + f s / 2 and 1 / L = r^2 (1 + e) to the order of e^2.  What is left of the power is the rounding of its last addition, nearer
// than powf (y against 64 bits: 4.1e-8 with powf, 5.9e-8 with one Newton step for r and s as it comes, 3.5e-8 here) at a third of its time.
struct Powers { float negBeta, inv; };

template <bool kThreeQuarters>
__device__ __forceinline__ Powers powers_of(float L, float beta)
{
  Powers w;
  if (!kThreeQuarters) { w.negBeta = powf(L, -beta); w.inv = __fdiv_rn(1.f, L); return w; }
  float const r = rsqrtf(L);
  float s;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(s) : "f"(r));
  float const u = __fmul_rn(L, r), e = fmaf(-fmaf(L, r, -u), r, fmaf(-u, r, 1.f)), f = fmaf(-s, s, r);
  float const p = __fmul_rn(r, s), q = __fmul_rn(r, r);
  float const dp = fmaf(__fmul_rn(0.5f, f), s, fmaf(__fmul_rn(0.75f, e), p, fmaf(r, s, -p)));
  bool const fine = dp == dp;          // (L = 0 or infinite: nothing to refine)
  w.negBeta = __fadd_rn(p, fine ? dp : 0.f);
  w.inv = fmaf(q, fine ? e : 0.f, q);
  return w;
}

// Windows of kD channels, kD small: everything a channel needs is in registers while the thread walks its channels, so x, dz and
// the result cross memory once and no integral is kept (the form with the integral in scratch moved 2.7 times the bytes: the
// backward passes of AlexNet's two layers at batch 128, 55x55x96 and 27x27x256, 733 MB, went from 912 to 227 us, the forward passes,
// 489 MB, from 368 to 174 us).  A thread takes `per` consecutive channels of one
// (pixel, image), kD - 1 more at either end for the windows that reach in: channels are split where there are too few pixels for the chip.
// (A window is summed afresh, so an infinite or not-a-number value spoils the windows that hold it and not, as in a sliding sum, all channels behind.)
// At step s the ring x[] holds the channels s - kD + 1 .. s: the window of channel t = s - m2.
template <int kD, bool kThreeQuarters>
__global__ void __launch_bounds__(128) lrn_forward_window_kernel(float* __restrict__ y, float const* __restrict__ x, LrnParams p, int per, int segments)
{
  vlb::pdl_wait();
  constexpr int m1 = (kD - 1) / 2, m2 = kD - m1 - 1;
  size_t const i = (size_t)blockIdx.x * blockDim.x + threadIdx.x, total = (size_t)p.P * p.N;
  if (i >= total * segments) return;
  size_t const seg = i / total, j = i - seg * total, n = j / p.P, off = j - n * p.P + (size_t)p.P * p.C * n;
  int const c0 = (int)seg * per, c1 = min(c0 + per, p.C);
  float const* const xp = x + off;
  float* const yp = y + off;
  float r[kD];
#pragma unroll
  for (int k = 0; k < kD; ++k) { int const c = c0 - m1 - 1 + k; r[k] = c >= 0 && c < p.C ? xp[(size_t)p.P * c] : 0.f; }
#pragma unroll 4
  for (int t = c0; t < c1; ++t) {
#pragma unroll
    for (int k = 0; k + 1 < kD; ++k) r[k] = r[k + 1];
    r[kD - 1] = t + m2 < p.C ? __ldg(xp + (size_t)p.P * (t + m2)) : 0.f;
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < kD; ++k) acc = fmaf(r[k], r[k], acc);
    yp[(size_t)p.P * t] = r[m1] * powers_of<kThreeQuarters>(p.kappa + p.alpha * acc, p.beta).negBeta;
  }
}

// Backward: with b_t = x_t * 2*alpha*beta * a_t / L_t and a_t = dz_t * L_t^-beta, dx_o = a_o - x_o * (sum of b_q over q in [o - m2, o + m1]).
// At step s: b of channel t = s - m2 enters its ring, and channel o = t - m1 -- the oldest of x[] -- is complete.
template <int kD, bool kThreeQuarters>
__global__ void __launch_bounds__(128) lrn_backward_window_kernel(float* __restrict__ dx, float const* __restrict__ x, float const* __restrict__ dz,
                                                                  LrnParams p, int per, int segments)
{
  vlb::pdl_wait();
  constexpr int m1 = (kD - 1) / 2, m2 = kD - m1 - 1;
  size_t const i = (size_t)blockIdx.x * blockDim.x + threadIdx.x, total = (size_t)p.P * p.N;
  if (i >= total * segments) return;
  size_t const seg = i / total, j = i - seg * total, n = j / p.P, off = j - n * p.P + (size_t)p.P * p.C * n;
  int const c0 = (int)seg * per, c1 = min(c0 + per, p.C);
  float const* const xp = x + off;
  float const* const zp = dz + off;
  float* const dp = dx + off;
  float const ab2 = 2.f * p.alpha * p.beta;
  float r[kD], b[kD], a[m1 + 1];
  // the first b needed is that of channel c0 - m2, whose window starts m1 channels before it
  int const t0 = c0 - m2;
#pragma unroll
  for (int k = 0; k < kD; ++k) { int const c = t0 - m1 - 1 + k; r[k] = c >= 0 && c < p.C ? xp[(size_t)p.P * c] : 0.f; b[k] = 0.f; }
#pragma unroll
  for (int k = 0; k <= m1; ++k) a[k] = 0.f;
  auto xAt = [&](int c) { return c < p.C && c >= 0 ? __ldg(xp + (size_t)p.P * c) : 0.f; };
  auto zAt = [&](int c) { return c < p.C && c >= 0 ? __ldg(zp + (size_t)p.P * c) : 0.f; };
  // four channels at a time, their loads on the way together (left to the compiler, the power's correction terms cost 30 to 50%: 55x55x96x128 133 us
  // against 184, 27x27x256x128 93 against 123; with the shorter power of 5.9e-8 the compiler's order took 141 and 81)
  for (int t4 = t0; t4 < c1 + m1; t4 += 4) {
    float xn[4], zn[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) { xn[u] = xAt(t4 + u + m2); zn[u] = zAt(t4 + u); }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      int const t = t4 + u, o = t - m1;
#pragma unroll
      for (int k = 0; k + 1 < kD; ++k) { r[k] = r[k + 1]; b[k] = b[k + 1]; }
#pragma unroll
      for (int k = 0; k < m1; ++k) a[k] = a[k + 1];
      r[kD - 1] = xn[u];
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < kD; ++k) acc = fmaf(r[k], r[k], acc);
      float const L = p.kappa + p.alpha * acc;
      Powers const w = powers_of<kThreeQuarters>(L, p.beta);
      a[m1] = zn[u] * w.negBeta;
      b[kD - 1] = t >= 0 && t < p.C ? r[m1] * ab2 * a[m1] * w.inv : 0.f;
      float sum = 0.f;
#pragma unroll
      for (int k = 0; k < kD; ++k) sum += b[k];
      if (o >= c0 && o < c1) dp[(size_t)p.P * o] = p.relu && !(r[0] > 0.f) ? 0.f : a[0] - sum * r[0];
    }
  }
}

// Launches the window kernels where they apply (depths 3, 5, 7, 9); false: the caller takes the general kernel.
template <bool kBackward>
bool launch_lrn_window(vlb_ctx* ctx, float* out, float const* x, float const* dz, LrnParams const& p, int depth)
{
  size_t const total = (size_t)p.P * p.N;
  // channels per thread: all of them, or a share of at least 16 (the windows that reach in cost depth - 1 channels per share)
  int per = p.C;
  while (per > 16 && total * (size_t)((p.C + per - 1) / per) < (size_t)ctx->smCount * 1024) per = (per + 1) / 2;
  int const segments = (p.C + per - 1) / per;
  size_t const blocks = (total * segments + 127) / 128;
  if (blocks >= (1u << 31)) return false;
  bool const tq = p.beta == 0.75f;
#define VLB_LRN(d) \
  case d: \
    if (kBackward) { if (tq) vlb::launch(ctx->stream, lrn_backward_window_kernel<d, true>, (unsigned)blocks, 128, 0, out, x, dz, p, per, segments); \
                     else    vlb::launch(ctx->stream, lrn_backward_window_kernel<d, false>, (unsigned)blocks, 128, 0, out, x, dz, p, per, segments); } \
    else           { if (tq) vlb::launch(ctx->stream, lrn_forward_window_kernel<d, true>, (unsigned)blocks, 128, 0, out, x, p, per, segments); \
                     else    vlb::launch(ctx->stream, lrn_forward_window_kernel<d, false>, (unsigned)blocks, 128, 0, out, x, p, per, segments); } \
    break;
  switch (depth) {
    VLB_LRN(3) VLB_LRN(5) VLB_LRN(7) VLB_LRN(9)
    default: return false;
  }
#undef VLB_LRN
  VLB_LAUNCHED(ctx, 1);
  return true;
}

// ---- softmax over the channels: one block per (pixel, image)
__device__ float block_reduce(float v, bool isMax, float* red)
{
  for (int o = 16; o > 0; o >>= 1) {
    float u = __shfl_xor_sync(0xffffffffu, v, o);
    v = isMax ? fmaxf(v, u) : v + u;
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  int const nw = blockDim.x >> 5;
  v = (int)threadIdx.x < nw ? red[threadIdx.x] : (isMax ? -INFINITY : 0.f);
  if (threadIdx.x < 32) {
    for (int o = 16; o > 0; o >>= 1) {
      float u = __shfl_xor_sync(0xffffffffu, v, o);
      v = isMax ? fmaxf(v, u) : v + u;
    }
    if (threadIdx.x == 0) red[0] = v;
  }
  __syncthreads();
  v = red[0];
  __syncthreads();
  return v;
}

// forward: y = exp(x - max) / sum; backward (dz != nullptr): out = y .* (dz - sum(dz .* y))   (matlab/vl_nnsoftmax.m:24-29)
__global__ void softmax_kernel(float* __restrict__ out, float const* __restrict__ x, float const* __restrict__ dz, int P, int C)
{
  vlb::pdl_wait();
  __shared__ float red[32];
  size_t const off = blockIdx.x + (size_t)P * C * blockIdx.y;
  float const* xp = x + off;
  float m = -INFINITY;
  for (int c = threadIdx.x; c < C; c += blockDim.x) m = fmaxf(m, xp[(size_t)P * c]);
  m = block_reduce(m, true, red);
  float s = 0.f;
  for (int c = threadIdx.x; c < C; c += blockDim.x) s += expf(xp[(size_t)P * c] - m);
  s = block_reduce(s, false, red);
  float dot = 0.f;
  if (dz) {
    for (int c = threadIdx.x; c < C; c += blockDim.x) dot += dz[off + (size_t)P * c] * (expf(xp[(size_t)P * c] - m) / s);
    dot = block_reduce(dot, false, red);
  }
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float const yv = expf(xp[(size_t)P * c] - m) / s;
    out[off + (size_t)P * c] = dz ? yv * (dz[off + (size_t)P * c] - dot) : yv;
  }
}

// ---- dropout: mask = scale * (u >= rate), u uniform in [0, 1) from a counter-based generator: element i of a call with
// seed s always gets the same number, whatever the grid
__device__ __forceinline__ uint32_t mix(uint32_t a, uint32_t b, uint32_t c)
{
  // three rounds of a multiply-xorshift finaliser over (index, seed)
  uint32_t h = a * 0x9E3779B1u ^ b * 0x85EBCA77u ^ c * 0xC2B2AE3Du;
  h ^= h >> 15; h *= 0x2C1B3C6Du; h ^= h >> 12; h *= 0x297A2D39u; h ^= h >> 15;
  h += a; h ^= h >> 16; h *= 0x7FEB352Du; h ^= h >> 15; h *= 0x846CA68Bu; h ^= h >> 16;
  return h;
}

__global__ void dropout_mask_kernel(float* __restrict__ mask, size_t n, float rate, float scale, uint32_t seedLo, uint32_t seedHi)
{
  vlb::pdl_wait();
  size_t const step = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
    uint32_t const h = mix((uint32_t)i, (uint32_t)(i >> 32) ^ seedLo, seedHi);
    float const u = (float)(h >> 8) * (1.f / 16777216.f);       // 24 bits: every value is representable
    mask[i] = u >= rate ? scale : 0.f;
  }
}

__global__ void mul_kernel(float* y, float const* a, float const* b, size_t n)
{
  vlb::pdl_wait();
  size_t const step = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) y[i] = a[i] * b[i];
}

int lrn_params(vlb_ctx* ctx, LrnParams* p, int H, int W, int C, int N, int normDepth, double kappa, double alpha, double beta)
{
  VLB_REQUIRE(ctx, H > 0 && W > 0 && C > 0 && N > 0, "normalize: empty tensor");
  VLB_REQUIRE(ctx, normDepth >= 1, "normalize: the normalisation depth is smaller than 1");       // matlab/src/vl_nnnormalize.cu:128-130
  p->P = H * W; p->C = C; p->N = N;
  p->m1 = (normDepth - 1) / 2; p->m2 = normDepth - p->m1 - 1;
  p->relu = 0;
  p->kappa = (float)kappa; p->alpha = (float)alpha; p->beta = (float)beta;
  return VLB_Success;
}

}  // namespace

extern "C" {

int vlb_lrn_forward(vlb_ctx* ctx, float* Y, float const* X, int H, int W, int C, int N, int normDepth, double kappa,
                    double alpha, double beta)
{
  if (!ctx) return VLB_IllegalArgument;
  LrnParams p;
  int rc = lrn_params(ctx, &p, H, W, C, N, normDepth, kappa, alpha, beta);
  if (rc) return rc;
  VLB_REQUIRE(ctx, Y && X, "lrn_forward: null tensor");
  if (launch_lrn_window<false>(ctx, Y, X, nullptr, p, normDepth)) return vlb::check_launch(ctx, "vlb_lrn_forward");
  vlb::launch(ctx->stream, lrn_forward_kernel, vlb::grid_for((size_t)p.P * N, kThreads, ctx->smCount * 8), kThreads, 0, Y, X, p);
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, "vlb_lrn_forward");
}

static int lrn_backward_common(vlb_ctx* ctx, float* dX, float const* X, float const* dY, int H, int W, int C, int N, int normDepth,
                               double kappa, double alpha, double beta, int relu, char const* where)
{
  if (!ctx) return VLB_IllegalArgument;
  LrnParams p;
  int rc = lrn_params(ctx, &p, H, W, C, N, normDepth, kappa, alpha, beta);
  if (rc) return rc;
  p.relu = relu;
  VLB_REQUIRE(ctx, dX && X && dY, "lrn_backward: null tensor");
  if (launch_lrn_window<true>(ctx, dX, X, dY, p, normDepth)) return vlb::check_launch(ctx, where);
  float* integral = (float*)vlb::workspace(ctx, sizeof(float) * (size_t)p.P * C * N);
  if (!integral) return vlb::pass_error(ctx, ctx->lastError, where);
  vlb::launch(ctx->stream, lrn_backward_kernel, vlb::grid_for((size_t)p.P * N, kThreads, ctx->smCount * 8), kThreads, 0, dX, integral, X, dY, p);
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, where);
}

int vlb_lrn_backward(vlb_ctx* ctx, float* dX, float const* X, float const* dY, int H, int W, int C, int N, int normDepth,
                     double kappa, double alpha, double beta)
{ return lrn_backward_common(ctx, dX, X, dY, H, W, C, N, normDepth, kappa, alpha, beta, 0, "vlb_lrn_backward"); }

int vlb_relu_lrn_backward(vlb_ctx* ctx, float* dX, float const* X, float const* dY, int H, int W, int C, int N, int normDepth,
                          double kappa, double alpha, double beta)
{ return lrn_backward_common(ctx, dX, X, dY, H, W, C, N, normDepth, kappa, alpha, beta, 1, "vlb_relu_lrn_backward"); }

int vlb_softmax_forward(vlb_ctx* ctx, float* Y, float const* X, int H, int W, int C, int N)
{
  if (!ctx) return VLB_IllegalArgument;
  VLB_REQUIRE(ctx, Y && X, "softmax_forward: null tensor");
  VLB_REQUIRE(ctx, H > 0 && W > 0 && C > 0 && N > 0 && N <= 65535, "softmax_forward: bad shape");
  int const threads = C >= 256 ? 256 : (C >= 64 ? 64 : 32);
  vlb::launch(ctx->stream, softmax_kernel, dim3(H * W, N), threads, 0, Y, X, nullptr, H * W, C);
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, "vlb_softmax_forward");
}

int vlb_softmax_backward(vlb_ctx* ctx, float* dX, float const* X, float const* dY, int H, int W, int C, int N)
{
  if (!ctx) return VLB_IllegalArgument;
  VLB_REQUIRE(ctx, dX && X && dY, "softmax_backward: null tensor");
  VLB_REQUIRE(ctx, H > 0 && W > 0 && C > 0 && N > 0 && N <= 65535, "softmax_backward: bad shape");
  int const threads = C >= 256 ? 256 : (C >= 64 ? 64 : 32);
  vlb::launch(ctx->stream, softmax_kernel, dim3(H * W, N), threads, 0, dX, X, dY, H * W, C);
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, "vlb_softmax_backward");
}

int vlb_dropout_mask(vlb_ctx* ctx, float* mask, size_t n, double rate, unsigned long long seed)
{
  if (!ctx) return VLB_IllegalArgument;
  VLB_REQUIRE(ctx, mask, "dropout_mask: null tensor");
  VLB_REQUIRE(ctx, rate >= 0.0 && rate < 1.0, "dropout_mask: RATE must be in [0, 1)");
  if (n == 0) return VLB_Success;
  float const scale = (float)(1.0 / (1.0 - rate));         // scale = 1 / (1 - rate), converted to single (matlab/vl_nndropout.m:44-56)
  vlb::launch(ctx->stream, dropout_mask_kernel, vlb::grid_for(n, kThreads, ctx->smCount * 8), kThreads, 0, 
      mask, n, (float)rate, scale, (uint32_t)seed, (uint32_t)(seed >> 32));
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, "vlb_dropout_mask");
}

int vlb_mul(vlb_ctx* ctx, float* Y, float const* A, float const* B, size_t n)
{
  if (!ctx) return VLB_IllegalArgument;
  VLB_REQUIRE(ctx, Y && A && B, "mul: null tensor");
  if (n == 0) return VLB_Success;
  vlb::launch(ctx->stream, mul_kernel, vlb::grid_for(n, kThreads, ctx->smCount * 8), kThreads, 0, Y, A, B, n);
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, "vlb_mul");
}

}  // extern "C"
