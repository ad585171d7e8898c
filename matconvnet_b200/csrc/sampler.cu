// Bilinear sampler (vl::nn::BilinearSampler, reference bits/nnbilinearsampler.hpp:21-36;
// CPU definition bits/nnbilinearsampler.cu:32-149).
//
// Forward and backward-to-grid stage the planes of a few channels in shared memory and walk the output
// pixels (q = ho + Ho*wo, grid n); where that does not pay, one thread per output pixel reads its taps
// from global memory.  The tap weights are formed once per pixel and the channels of the grid derivative
// added in ascending order, as in the CPU loop; each grid entry is written once.
//
// Backward-to-data is a gather, not the reference GPU code's four atomicAdds per output element
// (bits/impl/nnbilinearsampler_gpu.cu:38-118).  Which output pixels touch an input pixel depends
// on the grid alone, not on the channel, so one CTA per image first inverts the grid in shared
// memory: it counts the taps that land on every input pixel, prefix-sums the counts, fills one
// list (output pixel, tap) per input pixel and sorts each list by output pixel.  Then every
// input pixel adds up its list in ascending output-pixel order -- the order in which the CPU loop
// reaches that element (bits/nnbilinearsampler.cu:72-131) -- for eight channels per walk of the
// list, and writes dX once: no atomics, no zero fill, the CPU's result bit for bit, identical from
// run to run.  A grid that sends more than kMaxList taps to one input pixel, and planes too large for
// the lists, take the atomic scatter instead.
//
// Boundary rule of the CPU reference, kept as it is: the taps are guarded by
// `-1 <= sy && sy < inHeight` with inHeight a size_t (bits/nnbilinearsampler.cu:92), so
// sy == -1 is compared as a huge unsigned number and fails: samples whose floor is -1
// in either coordinate contribute nothing.
#include "common.cuh"
#include <math.h>
#include <type_traits>

namespace {

constexpr int kThreads = 128;

struct Taps {
  int sx, sy;
  float wx, wy;
  bool inside;
};

__device__ __forceinline__ Taps make_taps(float gy, float gx, int H, int W)
{
  Taps t;
  float py = __fmul_rn(__fmul_rn(0.5f, __fadd_rn(gy, 1.f)), (float)(H - 1));
  float px = __fmul_rn(__fmul_rn(0.5f, __fadd_rn(gx, 1.f)), (float)(W - 1));
  float fx = floorf(px), fy = floorf(py);
  // keep the int conversion defined for wild grid values
  fx = fminf(fmaxf(fx, -2.f), (float)W + 1.f);
  fy = fminf(fmaxf(fy, -2.f), (float)H + 1.f);
  t.sx = (int)fx; t.sy = (int)fy;
  t.inside = (t.sy >= 0 && t.sy < H && t.sx >= 0 && t.sx < W);
  t.wx = __fadd_rn(px, -(float)t.sx);
  t.wy = __fadd_rn(py, -(float)t.sy);
  return t;
}

// mode 0: forward.  mode 1: backward (dx and/or dgrid).
template <int kMode>
__global__ void sampler_kernel(float* __restrict__ y, float* __restrict__ dx, float* __restrict__ dgrid,
                               float const* __restrict__ x, float const* __restrict__ grid,
                               float const* __restrict__ dy, int H, int W, int C, int N, int Q, int Ng)
{
  vlb::pdl_wait();
  int group = Ng / N;
  size_t total = (size_t)Q * Ng;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    int q = (int)(i % Q);
    int n = (int)(i / Q);
    float2 gv = reinterpret_cast<float2 const*>(grid)[i];
    Taps t = make_taps(gv.x, gv.y, H, W);
    // tap (i = row offset, j = column offset); weights as in bits/nnbilinearsampler.cu:108-110
    float wwx[2] = {__fadd_rn(1.f, -t.wx), t.wx};
    float wwy[2] = {__fadd_rn(1.f, -t.wy), t.wy};
    bool ok[2][2];
    int idx[2][2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int ii = 0; ii < 2; ++ii) {
        int ssy = t.sy + ii, ssx = t.sx + j;
        ok[j][ii] = t.inside && ssy >= 0 && ssy < H && ssx >= 0 && ssx < W;
        idx[j][ii] = ssy + ssx * H;
      }
    size_t imgOff = (size_t)H * W * C * (size_t)(n / group);
    float const* xz = x + imgOff;
    float* dxz = (kMode == 1 && dx) ? dx + imgOff : nullptr;
    size_t outOff = (size_t)q + (size_t)Q * C * (size_t)n;
    float accGy = 0.f, accGx = 0.f;
    if (kMode == 0) {
      // Four channels at a time, all sixteen loads on the way before the first is used: one channel at a time the thread waited for memory
      // once per channel (64 x 64 x 32 x 256: 140 us -> 79 us; 41 us at copy speed).  A tap outside the plane reads the plane's first
      // element and its product is dropped; adding the +0 in its place changes no sum, none of which is ever -0.
      float wt[4];
      int at[4];
      bool on[4];
#pragma unroll
      for (int t4 = 0; t4 < 4; ++t4) {
        on[t4] = ok[t4 >> 1][t4 & 1];
        wt[t4] = __fmul_rn(wwx[t4 >> 1], wwy[t4 & 1]);
        at[t4] = on[t4] ? idx[t4 >> 1][t4 & 1] : 0;
      }
      int const HW = H * W;
      float* o = y + outOff;
      for (int c = 0; c < C; c += 4) {
        float v[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float const* const xk = xz + (size_t)min(k, C - 1 - c) * HW;
#pragma unroll
          for (int t4 = 0; t4 < 4; ++t4) v[k][t4] = __ldg(xk + at[t4]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float acc = 0.f;
#pragma unroll
          for (int t4 = 0; t4 < 4; ++t4) acc = __fadd_rn(acc, on[t4] ? __fmul_rn(wt[t4], v[k][t4]) : 0.f);
          if (c + k < C) o[(size_t)k * Q] = acc;
        }
        xz += 4 * (size_t)HW; o += 4 * (size_t)Q;
      }
      continue;
    }
    for (int c = 0; c < C; ++c) {
      float d = dy[outOff];
      float dgx = 0.f, dgy = 0.f;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int ii = 0; ii < 2; ++ii)
          if (ok[j][ii]) {
            if (dxz) atomicAdd(dxz + idx[j][ii], __fmul_rn(__fmul_rn(wwx[j], wwy[ii]), d));
            if (dgrid) {
              float xv = xz[idx[j][ii]];
              float sj = j ? 1.f : -1.f, si = ii ? 1.f : -1.f;
              dgx = __fadd_rn(dgx, __fmul_rn(__fmul_rn(__fmul_rn(sj, wwy[ii]), d), xv));
              dgy = __fadd_rn(dgy, __fmul_rn(__fmul_rn(__fmul_rn(si, wwx[j]), d), xv));
            }
          }
      if (dgrid) {
        accGy = __fadd_rn(accGy, __fmul_rn(__fmul_rn(0.5f, (float)(H - 1)), dgy));
        accGx = __fadd_rn(accGx, __fmul_rn(__fmul_rn(0.5f, (float)(W - 1)), dgx));
      }
      xz += (size_t)H * W;
      if (dxz) dxz += (size_t)H * W;
      outOff += Q;
    }
    if (kMode == 1 && dgrid) reinterpret_cast<float2*>(dgrid)[i] = make_float2(accGy, accGx);
  }
}

// ---- forward and grid derivative with the planes of four channels in shared memory, one float4 per pixel ----
// The direct kernel above is bound by the tags of L1: the 32 output pixels of a warp lie on a slanted line of the input, so that every
// load touches up to seven lines.  From shared memory a tap of four channels is one 16-byte read that the banks serve in four passes.
// B200, 64 x 64 x 32 x 256: forward 79 -> 61 us; 41 us at copy speed, the issue of
// instructions 71 % busy.
constexpr int kPlaneThreads = 512;
constexpr int kGridThreads = 512;
constexpr int kPlaneQ = 2;             // output pixels per thread of the grid derivative
constexpr int kGridCh = 2;             // channels per stage of the grid derivative

struct PixTaps { int at, ok; float wx, wy; };      // first tap's offset; bit ii + 2*j: tap (row offset ii, column offset j) exists

__device__ __forceinline__ PixTaps pix_taps(float2 gv, int H, int W)
{
  Taps const t = make_taps(gv.x, gv.y, H, W);
  PixTaps r;
  r.wx = t.wx; r.wy = t.wy;
  r.at = t.inside ? t.sy + t.sx * H : 0;
  r.ok = t.inside ? (1 | (t.sy + 1 < H ? 2 : 0) | (t.sx + 1 < W ? 4 : 0) | ((t.sy + 1 < H && t.sx + 1 < W) ? 8 : 0)) : 0;
  return r;
}

__device__ __forceinline__ void cp_async4(uint32_t dst, void const* src)
{ asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async16(uint32_t dst, void const* src)
{ asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory"); }

// n floats global -> shared by the whole block, asynchronously (16-byte pieces when both sides allow; copies of four bytes
// keep the load/store unit busy four times as long)
__device__ __forceinline__ void stage_plane(float* dst, float const* src, int n)
{
  uint32_t const d = (uint32_t)__cvta_generic_to_shared(dst);
  if ((n & 3) == 0 && ((((uintptr_t)src) | d) & 15) == 0) {
    for (int i = threadIdx.x; i < n / 4; i += blockDim.x) cp_async16(d + 16u * i, src + 4 * i);
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) cp_async4(d + 4u * i, src + i);
  }
}

__device__ __forceinline__ void add_tap(float4& a, float w, float4 v)
{
  a.x = __fadd_rn(a.x, __fmul_rn(w, v.x)); a.y = __fadd_rn(a.y, __fmul_rn(w, v.y));
  a.z = __fadd_rn(a.z, __fmul_rn(w, v.z)); a.w = __fadd_rn(a.w, __fmul_rn(w, v.w));
}

// One block: one image, four channels, all output pixels of its grids.
__global__ void __launch_bounds__(kPlaneThreads)
sampler_fwd_planes_kernel(float* __restrict__ y, float const* __restrict__ x, float const* __restrict__ grid, int H, int W, int C, int Q, int group,
                          int quads)
{
  vlb::pdl_wait();
  extern __shared__ float4 xs[];
  int const img = blockIdx.x / quads, c0 = (blockIdx.x - img * quads) * 4, nc = min(4, C - c0), HW = H * W;
  vlb::stage_planes(xs, x + (size_t)HW * ((size_t)C * img + c0), HW, nc);
  __syncthreads();
  for (int gi = 0; gi < group; ++gi) {
    int const n = img * group + gi;
    float2 const* const gr = reinterpret_cast<float2 const*>(grid) + (size_t)Q * n;
    float* const o = y + (size_t)Q * ((size_t)C * n + c0);
    int q = threadIdx.x;
    float2 next = q < Q ? __ldg(gr + q) : make_float2(0.f, 0.f);
    for (; q < Q; q += kPlaneThreads) {
      PixTaps const t = pix_taps(next, H, W);
      if (q + kPlaneThreads < Q) next = __ldg(gr + q + kPlaneThreads);
      float const wx0 = __fadd_rn(1.f, -t.wx), wy0 = __fadd_rn(1.f, -t.wy);
      float4 const* const p0 = xs + t.at;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t.ok & 1) add_tap(a, __fmul_rn(wx0, wy0), p0[0]);
      if (t.ok & 2) add_tap(a, __fmul_rn(wx0, t.wy), p0[1]);
      if (t.ok & 4) add_tap(a, __fmul_rn(t.wx, wy0), p0[H]);
      if (t.ok & 8) add_tap(a, __fmul_rn(t.wx, t.wy), p0[H + 1]);
      o[q] = a.x;
      if (nc == 4) {
        o[q + Q] = a.y; o[q + 2 * Q] = a.z; o[q + 3 * Q] = a.w;
      } else {
        if (nc > 1) o[q + Q] = a.y;
        if (nc > 2) o[q + 2 * Q] = a.z;
      }
    }
  }
}

// One channel's terms of an output pixel, the taps in the CPU loop's order (column offset j outer, row offset i inner;
// bits/nnbilinearsampler.cu:98-128).  (2j-1)*wwy*dy*x is evaluated left to right there; a negation is exact, so the two magnitudes
// wwy0*dy and wwy1*dy serve all four taps.
__device__ __forceinline__ void grid_terms(float& accGy, float& accGx, int ok, float wx0, float wx1, float wy0, float wy1, float d,
                                           float x00, float x10, float x01, float x11, float sclY, float sclX)
{
  float const ty0 = __fmul_rn(wy0, d), ty1 = __fmul_rn(wy1, d), tx0 = __fmul_rn(wx0, d), tx1 = __fmul_rn(wx1, d);
  float dgx = __fsub_rn(0.f, __fmul_rn(ty0, x00)), dgy = __fsub_rn(0.f, __fmul_rn(tx0, x00));
  if (ok & 2) { dgx = __fsub_rn(dgx, __fmul_rn(ty1, x10)); dgy = __fadd_rn(dgy, __fmul_rn(tx0, x10)); }
  if (ok & 4) { dgx = __fadd_rn(dgx, __fmul_rn(ty0, x01)); dgy = __fsub_rn(dgy, __fmul_rn(tx1, x01)); }
  if (ok & 8) { dgx = __fadd_rn(dgx, __fmul_rn(ty1, x11)); dgy = __fadd_rn(dgy, __fmul_rn(tx1, x11)); }
  accGy = __fadd_rn(accGy, __fmul_rn(sclY, dgy));
  accGx = __fadd_rn(accGx, __fmul_rn(sclX, dgx));
}

// Grid derivative.  One block: one grid and QP <= kGridThreads * kPlaneQ of its output pixels, all channels in ascending order, kGridCh per
// stage.  Bound by the issue of instructions, hence three blocks per SM
// (64 x 64 x 32 x 256, two channels of two pixels per thread: 129 us; four channels or four pixels, with fewer warps: 137 to 160).  The x planes of the next stage travel by asynchronous copies, its dY
// through registers: an output pixel's values are asked for as soon as those of this stage are used.
__global__ void __launch_bounds__(kGridThreads, 3)
sampler_grid_planes_kernel(float* __restrict__ dgrid, float const* __restrict__ x, float const* __restrict__ grid, float const* __restrict__ dy,
                           int H, int W, int C, int Q, int group, int parts, int QP)
{
  vlb::pdl_wait();
  extern __shared__ float4 xsm[];
  int const n = blockIdx.x / parts, q0 = (blockIdx.x - n * parts) * QP, qEnd = min(Q, q0 + QP), HW = H * W;
  float* const xs = reinterpret_cast<float*>(xsm);          // [2][kGridCh][HW]
  float const* const xi = x + (size_t)HW * C * (n / group);
  float2 const* const gr = reinterpret_cast<float2 const*>(grid) + (size_t)Q * n;
  float const* const dyn = dy + (size_t)Q * C * n;
  float const sclY = __fmul_rn(0.5f, (float)(H - 1)), sclX = __fmul_rn(0.5f, (float)(W - 1));
  stage_plane(xs, xi, HW * min(kGridCh, C));
  float accGy[kPlaneQ], accGx[kPlaneQ], wx[kPlaneQ], wy[kPlaneQ], d[kPlaneQ][kGridCh];
  int at[kPlaneQ];                                          // first tap | which taps exist << 28
#pragma unroll
  for (int k = 0; k < kPlaneQ; ++k) {
    int const q = q0 + threadIdx.x + k * kGridThreads;
    accGy[k] = accGx[k] = 0.f;
#pragma unroll
    for (int j = 0; j < kGridCh; ++j) d[k][j] = 0.f;
    at[k] = 0; wx[k] = wy[k] = 0.f;
    if (q < qEnd) {
      PixTaps const t = pix_taps(__ldg(gr + q), H, W);
      at[k] = t.at | (t.ok << 28); wx[k] = t.wx; wy[k] = t.wy;
#pragma unroll
      for (int j = 0; j < kGridCh; ++j)
        if (j < C) d[k][j] = __ldg(dyn + (size_t)Q * j + q);
    }
  }
  int buf = 0;
  for (int c0 = 0; c0 < C; c0 += kGridCh, buf ^= 1) {
    int const nc = min(kGridCh, C - c0), left = C - c0 - kGridCh;
    float const* const xc = xs + (size_t)(buf * kGridCh) * HW;
    cp_async_wait_all();
    __syncthreads();                    // this stage's planes have landed; the other buffer is no longer read
    if (left > 0) stage_plane(xs + (size_t)((buf ^ 1) * kGridCh) * HW, xi + (size_t)HW * (c0 + kGridCh), HW * min(kGridCh, left));
    float const* const dn = dyn + (size_t)Q * (c0 + kGridCh) + q0 + threadIdx.x;
#pragma unroll
    for (int k = 0; k < kPlaneQ; ++k) {
      int const ok = (int)((unsigned)at[k] >> 28);
      if (ok) {
        float const wx0 = __fadd_rn(1.f, -wx[k]), wy0 = __fadd_rn(1.f, -wy[k]);
        float const* p0 = xc + (at[k] & 0x0fffffff);
        float v[kGridCh][4];
#pragma unroll
        for (int j = 0; j < kGridCh; ++j) {
          v[j][0] = v[j][1] = v[j][2] = v[j][3] = 0.f;
          if (j < nc) {
            v[j][0] = p0[0];
            if (ok & 2) v[j][1] = p0[1];
            if (ok & 4) v[j][2] = p0[H];
            if (ok & 8) v[j][3] = p0[H + 1];
          }
          p0 += HW;
        }
#pragma unroll
        for (int j = 0; j < kGridCh; ++j)
          if (j < nc) grid_terms(accGy[k], accGx[k], ok, wx0, wx[k], wy0, wy[k], d[k][j], v[j][0], v[j][1], v[j][2], v[j][3], sclY, sclX);
#pragma unroll
        for (int j = 0; j < kGridCh; ++j)
          if (j < left) d[k][j] = __ldg(dn + Q * j + k * kGridThreads);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kPlaneQ; ++k) {
    int const q = q0 + threadIdx.x + k * kGridThreads;
    if (q < qEnd) reinterpret_cast<float2*>(dgrid)[(size_t)Q * n + q] = make_float2(accGy[k], accGx[k]);
  }
}

// ---- backward-to-data as a gather (see the header comment) ----
constexpr int kGatherThreads = 1024;
constexpr int kMaxList = 48;          // taps of one grid on one input pixel beyond which the scatter path is used
constexpr int kMaxQPerThread = 4;     // output pixels per thread
constexpr int kCB = 8;                // channels per stage: one walk of a pixel's list serves eight channels

// Shared memory (bytes): dys float4[2][Q] (dY of eight channels, four side by side) | wq float2[Q] (the two fractions of every output pixel) |
// ent uint16[4Q] (list entries: output pixel << 2 | tap) | cur int[HW + 1] (where every input pixel's list begins)
__host__ __device__ inline size_t gather_smem(int HW, int Q)
{ return (2 * sizeof(float4) + sizeof(float2) + 4 * sizeof(uint16_t)) * (size_t)Q + sizeof(int) * ((size_t)HW + 1) + 64; }

// Bound by shared memory: an entry of a list costs one 2-byte, one 8-byte and two 16-byte reads for eight channels, the last two bank passes
// per channel.  dY travels through registers (it has to be laid side by side), asked for one stage ahead.
// B200, 64 x 64 x 32 x 256, both derivatives: 268 us with four channels per walk and the grid derivative in the same
// block, 255 us now; half of that is the data gradient, for which 256 images on 148 SMs are two rounds, the second not full.
__global__ void __launch_bounds__(kGatherThreads, 1)
sampler_bwd_gather_kernel(float* __restrict__ dx, float const* __restrict__ grid, float const* __restrict__ dy, int H, int W, int C, int N, int Q, int Ng,
                          int chunks, int CH)
{
  vlb::pdl_wait();
  extern __shared__ __align__(16) uint8_t sm[];
  __shared__ int warpSums[32];
  int const HW = H * W, tid = threadIdx.x;
  float4* dys = reinterpret_cast<float4*>(sm);                              // [2][Q]
  float2* wq = reinterpret_cast<float2*>(dys + 2 * (size_t)Q);              // [Q]   (wx, wy) of every output pixel
  uint16_t* ent = reinterpret_cast<uint16_t*>(wq + Q);                      // [4Q]  output pixel << 2 | tap (tap = 2*column offset + row offset)
  int* cur = reinterpret_cast<int*>(ent + 4 * (size_t)Q);                   // [HW + 1]
  int const group = Ng / N;
  int const img = blockIdx.x / chunks, c0 = (blockIdx.x % chunks) * CH, nch = min(CH, C - c0);
  int const nStages = (nch + kCB - 1) / kCB;
  size_t const imgOff = (size_t)HW * C * (size_t)img;

  for (int gi = 0; gi < group; ++gi) {
    int const n = img * group + gi;
    float2 const* gr = reinterpret_cast<float2 const*>(grid) + (size_t)Q * n;
    float const* const dyn = dy + (size_t)Q * C * (size_t)n;
    // ---- invert the grid: count, scan, fill, sort
    for (int i = tid; i <= HW; i += kGatherThreads) cur[i] = 0;
    __syncthreads();
    int at[kMaxQPerThread];               // first tap of this thread's output pixels | which taps exist << 28
    uint32_t rank[kMaxQPerThread];        // its four taps' places in their lists, a byte each
#pragma unroll
    for (int k = 0; k < kMaxQPerThread; ++k) {
      int const q = tid + k * kGatherThreads;
      at[k] = 0; rank[k] = 0;
      if (q < Q) {
        PixTaps const t = pix_taps(__ldg(gr + q), H, W);
        wq[q] = make_float2(t.wx, t.wy);
        at[k] = t.at | (t.ok << 28);
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (t.ok & (1 << b)) rank[k] |= ((uint32_t)atomicAdd(&cur[t.at + (b & 1) + (b >> 1) * H], 1) & 255u) << (8 * b);
      }
    }
    __syncthreads();
    bool tooLong = false;
    for (int i = tid; i < HW; i += kGatherThreads) tooLong |= cur[i] > kMaxList;
    bool const scatter = __syncthreads_or(tooLong) != 0;
    if (!scatter) {
      vlb::block_exclusive_scan<kGatherThreads>(cur, HW + 1, warpSums);
#pragma unroll
      for (int k = 0; k < kMaxQPerThread; ++k) {
        int const q = tid + k * kGatherThreads, ok = (int)((unsigned)at[k] >> 28), first = at[k] & 0x0fffffff;
#pragma unroll
        for (int b = 0; b < 4; ++b)
          if (ok & (1 << b)) ent[cur[first + (b & 1) + (b >> 1) * H] + (int)((rank[k] >> (8 * b)) & 255u)] = (uint16_t)((q << 2) | b);
      }
      // the dY of the stage that comes next, on its way while this one is computed
      float v[kMaxQPerThread][kCB] = {};
      auto ask = [&](int cs) {
        int const left = c0 + nch - cs;
#pragma unroll
        for (int k = 0; k < kMaxQPerThread; ++k) {
          int const q = tid + k * kGatherThreads;
          if (q < Q) {
            float const* const d = dyn + (size_t)Q * cs + q;
#pragma unroll
            for (int j = 0; j < kCB; ++j)
              if (j < left) v[k][j] = __ldg(d + (size_t)Q * j);
          }
        }
      };
      ask(c0);
      __syncthreads();
      // every input pixel sorts its list by output pixel (an output pixel reaches an input pixel with one tap at most)
      for (int pix = tid; pix < HW; pix += kGatherThreads) {
        int const beg = cur[pix], end = cur[pix + 1];
        for (int a = beg + 1; a < end; ++a) {
          uint16_t const kq = ent[a];
          int b = a - 1;
          while (b >= beg && ent[b] > kq) { ent[b + 1] = ent[b]; --b; }
          ent[b + 1] = kq;
        }
      }
      for (int st = 0; st < nStages; ++st) {
        int const cs = c0 + st * kCB, nst = min(kCB, c0 + nch - cs);
        if (st > 0) __syncthreads();        // the previous stage is no longer read
#pragma unroll
        for (int k = 0; k < kMaxQPerThread; ++k) {
          int const q = tid + k * kGatherThreads;
          if (q < Q) {
            dys[q] = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
            if (nst > 4) dys[Q + q] = make_float4(v[k][4], v[k][5], v[k][6], v[k][7]);
          }
        }
        __syncthreads();                    // (and the lists are sorted)
        if (st + 1 < nStages) ask(cs + kCB);
        // every input pixel adds up its list in output-pixel order.  The weight of an entry is wwx[j] * wwy[i] as the CPU loop
        // forms it (bits/nnbilinearsampler.cu:108-110), from the output pixel's two fractions.
        float* const dxc = dx + imgOff + (size_t)HW * cs;
        auto walk = [&](auto full) {
          int const m = decltype(full)::value ? kCB : nst;       // (a constant in all stages but the last)
          for (int pix = tid; pix < HW; pix += kGatherThreads) {
            int const beg = cur[pix], end = cur[pix + 1];
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
            float* const o = dxc + pix;
            if (gi > 0) {
              a.x = o[0];
              if (m > 1) a.y = o[HW];
              if (m > 2) a.z = o[2 * HW];
              if (m > 3) a.w = o[3 * HW];
              if (m > 4) b.x = o[4 * HW];
              if (m > 5) b.y = o[5 * HW];
              if (m > 6) b.z = o[6 * HW];
              if (m > 7) b.w = o[7 * HW];
            }
#pragma unroll 2
            for (int e = beg; e < end; ++e) {
              unsigned const en = ent[e];
              unsigned const q = en >> 2;
              float2 const f = wq[q];
              float4 const da = dys[q], db = m > 4 ? dys[Q + q] : da;
              float const wx = (en & 2u) ? f.x : __fadd_rn(1.f, -f.x), wy = (en & 1u) ? f.y : __fadd_rn(1.f, -f.y);
              float const w = __fmul_rn(wx, wy);
              add_tap(a, w, da);
              if (m > 4) add_tap(b, w, db);
            }
            o[0] = a.x;
            if (m > 1) o[HW] = a.y;
            if (m > 2) o[2 * HW] = a.z;
            if (m > 3) o[3 * HW] = a.w;
            if (m > 4) o[4 * HW] = b.x;
            if (m > 5) o[5 * HW] = b.y;
            if (m > 6) o[6 * HW] = b.z;
            if (m > 7) o[7 * HW] = b.w;
          }
        };
        if (nst == kCB) walk(std::integral_constant<bool, true>{});
        else            walk(std::integral_constant<bool, false>{});
      }
    } else {
      // a grid that piles its taps on a few input pixels: zero (first grid of the image) and scatter with atomics, from
      // global memory
      if (gi == 0) {
        for (size_t i = tid; i < (size_t)HW * nch; i += kGatherThreads) dx[imgOff + (size_t)HW * c0 + i] = 0.f;
      }
      __syncthreads();
      for (int q = tid; q < Q; q += kGatherThreads) {
        PixTaps const t = pix_taps(__ldg(gr + q), H, W);
        float const wwx[2] = {__fadd_rn(1.f, -t.wx), t.wx};
        float const wwy[2] = {__fadd_rn(1.f, -t.wy), t.wy};
        for (int c = c0; c < c0 + nch; ++c) {
          float const d = dyn[q + (size_t)Q * c];
          float* const dxz = dx + imgOff + (size_t)HW * c + t.at;
#pragma unroll
          for (int b = 0; b < 4; ++b)
            if (t.ok & (1 << b)) atomicAdd(dxz + (b & 1) + (b >> 1) * H, __fmul_rn(__fmul_rn(wwx[b >> 1], wwy[b & 1]), d));
        }
      }
    }
    __syncthreads();       // this grid's additions to dX are visible to the block, and the lists free, before the next grid
  }
}

// The planes of four channels in shared memory (pixels: of the plane or planes that a block holds at a time), where an image fills a good part of
// the chip with blocks, a stage of x is not mostly unread (Q at least half of a plane), and the planes fit.  These kernels count output pixels, and
// four planes of them, in 32 bits: grids of 2^29 pixels and more, and more blocks than a launch has, take the thread-per-pixel kernel.
bool planes_apply(vlb_ctx* ctx, long long pixels, bool readsMost, int C, int Q, long long blocks)
{
  return C >= 3 && (long long)sizeof(float4) * pixels <= 220 * 1024 && readsMost && Q < (1 << 29) && blocks >= ctx->smCount && blocks < (1LL << 31);
}

// the three kernels above take as much shared memory as an SM has; false with a CUDA error pending
bool allow_smem(vlb_ctx* ctx)
{
  static bool done[64] = {};
  if (ctx->device < 64 && done[ctx->device]) return true;
  bool const ok = vlb::allow_max_dynamic_smem(sampler_fwd_planes_kernel) == cudaSuccess && vlb::allow_max_dynamic_smem(sampler_grid_planes_kernel) == cudaSuccess &&
                  vlb::allow_max_dynamic_smem(sampler_bwd_gather_kernel) == cudaSuccess;
  if (ok && ctx->device < 64) done[ctx->device] = true;
  return ok;
}

int validate(vlb_ctx* ctx, int H, int W, int C, int N, int Ho, int Wo, int Ng)
{
  VLB_REQUIRE(ctx, H > 0 && W > 0 && C > 0 && N > 0 && Ho > 0 && Wo > 0 && Ng > 0, "bilinearsampler: empty tensor");
  // GRID must hold a whole number of grids per image (matlab/src/vl_nnbilinearsampler.cu:141-146)
  VLB_REQUIRE(ctx, Ng % N == 0, "bilinearsampler: the number of grids is not a multiple of the number of images");
  VLB_REQUIRE(ctx, (long long)H * W < (1LL << 31) && (long long)Ho * Wo < (1LL << 31), "bilinearsampler: plane too large");
  return VLB_Success;
}

}  // namespace

extern "C" {

int vlb_sampler_forward(vlb_ctx* ctx, float* Y, float const* X, float const* grid, int H, int W, int C, int N,
                        int Ho, int Wo, int Ng)
{
  if (!ctx) return VLB_IllegalArgument;
  int rc = validate(ctx, H, W, C, N, Ho, Wo, Ng);
  if (rc) return rc;
  VLB_REQUIRE(ctx, Y && X && grid, "sampler_forward: null tensor");
  VLB_REQUIRE(ctx, (((uintptr_t)grid) & 7) == 0, "sampler_forward: grid must be 8-byte aligned");
  int const Q = Ho * Wo, quads = vlb::ceil_div(C, 4);
  if (planes_apply(ctx, (long long)H * W, 2LL * Q >= (long long)H * W, C, Q, (long long)N * quads)) {
    if (!allow_smem(ctx)) return vlb::check_launch(ctx, "vlb_sampler_forward");
    vlb::launch(ctx->stream, sampler_fwd_planes_kernel, (unsigned)(N * quads), kPlaneThreads, sizeof(float4) * (size_t)H * W, Y, X, grid, H, W, C, Q, Ng / N, quads);
    VLB_LAUNCHED(ctx, 1);
    return vlb::check_launch(ctx, "vlb_sampler_forward");
  }
  size_t total = (size_t)Ho * Wo * Ng;
  vlb::launch(ctx->stream, sampler_kernel<0>, vlb::grid_for(total, kThreads, ctx->smCount * 32), kThreads, 0, 
      Y, nullptr, nullptr, X, grid, nullptr, H, W, C, N, Ho * Wo, Ng);
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, "vlb_sampler_forward");
}

int vlb_sampler_backward(vlb_ctx* ctx, float* dX, float* dGrid, float const* X, float const* grid, float const* dY,
                         int H, int W, int C, int N, int Ho, int Wo, int Ng)
{
  if (!ctx) return VLB_IllegalArgument;
  int rc = validate(ctx, H, W, C, N, Ho, Wo, Ng);
  if (rc) return rc;
  VLB_REQUIRE(ctx, grid && dY, "sampler_backward: null tensor");
  VLB_REQUIRE(ctx, !dGrid || X, "sampler_backward: the grid derivative needs the input");
  VLB_REQUIRE(ctx, ((((uintptr_t)grid) | ((uintptr_t)dGrid)) & 7) == 0, "sampler_backward: grid must be 8-byte aligned");
  if (!dX && !dGrid) return VLB_Success;
  int const Qo = Ho * Wo, HWi = H * W;
  if (dX && Qo <= kMaxQPerThread * kGatherThreads && HWi < (1 << 28) && gather_smem(HWi, Qo) <= 226 * 1024) {
    // gather: one CTA per image; with fewer images than SMs the channels are shared out among several CTAs per image
    int chunks = 1;
    if (N < ctx->smCount) chunks = vlb::ceil_div(ctx->smCount, N);
    int CH = vlb::ceil_div(C, chunks);
    chunks = vlb::ceil_div(C, CH);
    if (!allow_smem(ctx)) return vlb::check_launch(ctx, "vlb_sampler_backward");
    size_t const smem = gather_smem(HWi, Qo);
    unsigned const blocks = (unsigned)(N * chunks);
    vlb::launch(ctx->stream, sampler_bwd_gather_kernel, blocks, kGatherThreads, smem, dX, grid, dY, H, W, C, N, Qo, Ng, chunks, CH);
    VLB_LAUNCHED(ctx, 1);
    dX = nullptr;
    if (!dGrid) return vlb::check_launch(ctx, "vlb_sampler_backward");
  }
  if (!dX) {
    // the grid derivative alone: blocks of at most kGridThreads * kPlaneQ output pixels (each reads the whole image, from L2 all but once)
    int const parts = vlb::ceil_div(Qo, kGridThreads * kPlaneQ);
    if (planes_apply(ctx, 2LL * HWi * kGridCh / 4, 2LL * Qo >= HWi, C, Qo, (long long)Ng * parts)) {
      int const QP = vlb::ceil_div(Qo, parts);
      if (!allow_smem(ctx)) return vlb::check_launch(ctx, "vlb_sampler_backward");
      vlb::launch(ctx->stream, sampler_grid_planes_kernel, (unsigned)(Ng * parts), kGridThreads, 2 * kGridCh * sizeof(float) * (size_t)HWi, dGrid, X, grid, dY, H, W, C, Qo,
          Ng / N, parts, QP);
      VLB_LAUNCHED(ctx, 1);
      return vlb::check_launch(ctx, "vlb_sampler_backward");
    }
  }
  if (dX) {
    cudaError_t e = cudaMemsetAsync(dX, 0, sizeof(float) * (size_t)H * W * C * N, ctx->stream);
    if (e != cudaSuccess) return vlb::set_error(ctx, VLB_Cuda, cudaGetErrorString(e));
  }
  size_t total = (size_t)Ho * Wo * Ng;
  vlb::launch(ctx->stream, sampler_kernel<1>, vlb::grid_for(total, kThreads, ctx->smCount * 32), kThreads, 0, 
      nullptr, dX, dGrid, X, grid, dY, H, W, C, N, Ho * Wo, Ng);
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, "vlb_sampler_backward");
}

}  // extern "C"
