// Max / average pooling, forward and backward (vl::nn::Pooling,
// reference bits/nnpooling.hpp:21-49; CPU definition bits/nnpooling.cu:102-214).
//
// HBM-bound.  Two families:
//  * non-overlapping 2x2 / stride 2 / no pad on even H and W (every pooling layer of
//    VGG-16): each thread owns whole windows, so the backward pass REPLAYS the argmax
//    scan and overwrites dx with 64/128-bit stores -- no atomics, no zero fill, no
//    scratch; algorithmic traffic 4*(2*in + out) bytes is also the real traffic.
//  * everything else: tiles in shared memory (pool_fwd_tiled, pool_bwd_tiled); backward is a gather, every
//    INPUT element visiting the windows that cover it in the
//    reference's order (wo outer, ho inner), so sums are formed in the same order as
//    on the CPU and the result is bit-identical and run-to-run deterministic.  Columns too long
//    for a tile take the thread-per-element kernels.
#include "common.cuh"
#include <math.h>
#include <algorithm>

namespace {

constexpr int kThreads = 256;

using vlb::FastDiv;

struct PoolParams {
  int H, W, Ho, Wo;
  int poolH, poolW, strideY, strideX, padTop, padLeft;
  size_t planes;   // C * N
};

// ------------------------------------------------------------------ generic forward
template <bool kMax>
__global__ void pool_fwd_generic(float* __restrict__ y, float const* __restrict__ x, PoolParams p)
{
  vlb::pdl_wait();
  size_t total = p.planes * (size_t)p.Ho * p.Wo;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    int ho = (int)(i % p.Ho);
    size_t t = i / p.Ho;
    int wo = (int)(t % p.Wo);
    size_t z = t / p.Wo;
    int x1 = wo * p.strideX - p.padLeft, y1 = ho * p.strideY - p.padTop;
    int x2 = min(x1 + p.poolW, p.W), y2 = min(y1 + p.poolH, p.H);
    x1 = max(x1, 0); y1 = max(y1, 0);
    float const* xz = x + z * (size_t)p.H * p.W;
    if (kMax) {
      float best = -INFINITY;
      for (int u = x1; u < x2; ++u)
        for (int v = y1; v < y2; ++v) { float a = xz[(size_t)u * p.H + v]; best = (best < a) ? a : best; }
      y[i] = best;
    } else {
      float s = 0.f;
      for (int u = x1; u < x2; ++u)
        for (int v = y1; v < y2; ++v) s = __fadd_rn(s, xz[(size_t)u * p.H + v]);
      float scale = __fdiv_rn(1.f, (float)((y2 - y1) * (x2 - x1)));
      y[i] = __fmul_rn(s, scale);
    }
  }
}

// ------------------------------------------------------------------ generic backward (gather)
// Thread per input element (v = row, u = column, plane z).  Windows covering it:
// ho in [ceil((v + padTop - poolH + 1)/strideY), floor((v + padTop)/strideY)], likewise wo.
__device__ __forceinline__ int floor_div(int a, int b) { int q = a / b; return (a % b != 0 && ((a < 0) != (b < 0))) ? q - 1 : q; }
__device__ __forceinline__ int ceil_div_i(int a, int b) { return -floor_div(-a, b); }

// relu: x is the output of a ReLU and dx the derivative with respect to that ReLU's input: zero where x is not positive.
template <bool kMax>
__global__ void pool_bwd_generic(float* __restrict__ dx, float const* __restrict__ x,
                                 float const* __restrict__ dy, PoolParams p, bool relu)
{
  vlb::pdl_wait();
  size_t total = p.planes * (size_t)p.H * p.W;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    int v = (int)(i % p.H);
    size_t t = i / p.H;
    int u = (int)(t % p.W);
    size_t z = t / p.W;
    int ho0 = max(ceil_div_i(v + p.padTop - p.poolH + 1, p.strideY), 0);
    int ho1 = min(floor_div(v + p.padTop, p.strideY), p.Ho - 1);
    int wo0 = max(ceil_div_i(u + p.padLeft - p.poolW + 1, p.strideX), 0);
    int wo1 = min(floor_div(u + p.padLeft, p.strideX), p.Wo - 1);
    float const* xz = x + z * (size_t)p.H * p.W;
    float const* dyz = dy + z * (size_t)p.Ho * p.Wo;
    float acc = 0.f;
    for (int wo = wo0; wo <= wo1; ++wo)
      for (int ho = ho0; ho <= ho1; ++ho) {
        int x1 = wo * p.strideX - p.padLeft, y1 = ho * p.strideY - p.padTop;
        int x2 = min(x1 + p.poolW, p.W), y2 = min(y1 + p.poolH, p.H);
        x1 = max(x1, 0); y1 = max(y1, 0);
        float d = dyz[(size_t)wo * p.Ho + ho];
        if (kMax) {
          // Replay the reference scan: column-outer, row-inner, first strictly greater wins.
          float best = -INFINITY;
          int bu = -1, bv = -1;
          for (int uu = x1; uu < x2; ++uu)
            for (int vv = y1; vv < y2; ++vv) {
              float a = xz[(size_t)uu * p.H + vv];
              if (a > best) { best = a; bu = uu; bv = vv; }
            }
          if (bu == u && bv == v) acc = __fadd_rn(acc, d);
        } else {
          float scale = __fdiv_rn(1.f, (float)((y2 - y1) * (x2 - x1)));
          acc = __fadd_rn(acc, __fmul_rn(d, scale));
        }
      }
    if (relu) acc = xz[(size_t)u * p.H + v] > 0.f ? acc : 0.f;
    dx[i] = acc;
  }
}

// ------------------------------------------------------------------ overlapping windows: tiles in shared memory
// A block takes whole planes, or a strip of columns of one plane, that fit its shared memory: the input is read once, coalesced; a
// window's arg-max is found once, by one thread, instead of once per input element that the window covers (a 3x3 / stride-2 backward pass
// scanned every window nine times: 1273 us on 55x55x96x128 where its 334 MB take 51 us; this kernel: 292 us); then every
// input element adds the derivatives of the windows that chose it, in the reference's order (wo outer, ho inner).
struct TileParams {
  PoolParams p;
  int planesPerTile, cols, tilesPerPlane;     // one plane and `cols` columns per tile (backward: of the input, forward: of the output), or several whole planes
  int xCols, winCols;                         // columns of the input / of windows that a tile holds at most
  FastDiv H, Ho, sy, sx, xPlane, winPlane, blkPlane, blkRows;    // ..Plane: elements of a tile per plane (planesPerTile > 1)
};

// A tile's place: first plane, planes, its range of windows [w0, w1) and of input columns [c0, c1).
struct Tile { size_t z0; int planes, u0, u1, w0, w1, c0, c1; };

__device__ __forceinline__ Tile tile_of(TileParams const& t, bool backward)
{
  Tile r;
  PoolParams const& p = t.p;
  if (t.planesPerTile > 1) {
    r.z0 = (size_t)blockIdx.x * t.planesPerTile;
    r.planes = (int)min((size_t)t.planesPerTile, p.planes - r.z0);
    r.u0 = 0; r.u1 = p.W; r.w0 = 0; r.w1 = p.Wo; r.c0 = 0; r.c1 = p.W;
    return r;
  }
  r.z0 = blockIdx.x / t.tilesPerPlane;
  r.planes = 1;
  int const s = (int)(blockIdx.x - r.z0 * t.tilesPerPlane) * t.cols;
  if (backward) {
    r.u0 = s; r.u1 = min(s + t.cols, p.W);
    r.w0 = max(ceil_div_i(r.u0 + p.padLeft - p.poolW + 1, p.strideX), 0);
    r.w1 = min((r.u1 - 1 + p.padLeft) / p.strideX + 1, p.Wo);
  } else {
    r.w0 = s; r.w1 = min(s + t.cols, p.Wo);
    r.u0 = r.u1 = 0;
  }
  r.c0 = max(r.w0 * p.strideX - p.padLeft, 0);
  r.c1 = max(r.c0, min((r.w1 - 1) * p.strideX - p.padLeft + p.poolW, p.W));
  if (backward && r.w1 > r.w0) { r.c0 = min(r.c0, r.u0); r.c1 = max(r.c1, r.u1); }      // (the ReLU mask reads the tile's own elements too)
  if (r.w1 <= r.w0) { r.w1 = r.w0; r.c0 = r.u0; r.c1 = r.u1; }
  return r;
}

// The columns [c0, c1) of `planes` planes of x into shared memory.  Whole planes are one contiguous run.
__device__ __forceinline__ void load_tile(float* xs, float const* __restrict__ x, TileParams const& t, Tile const& r)
{
  size_t const plane = (size_t)t.p.H * t.p.W;
  int const n = t.planesPerTile > 1 ? r.planes * (int)plane : (r.c1 - r.c0) * t.p.H;
  float const* const src = x + r.z0 * plane + (size_t)r.c0 * t.p.H;
  for (int i = threadIdx.x; i < n; i += 4 * kThreads) {
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = i + k * kThreads < n ? __ldg(src + i + k * kThreads) : 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) if (i + k * kThreads < n) xs[i + k * kThreads] = v[k];
  }
}

struct Window { int x1, x2, y1, y2; };

__device__ __forceinline__ Window window_of(PoolParams const& p, int ho, int wo)
{
  Window w;
  w.x1 = wo * p.strideX - p.padLeft; w.y1 = ho * p.strideY - p.padTop;
  w.x2 = min(w.x1 + p.poolW, p.W); w.y2 = min(w.y1 + p.poolH, p.H);
  w.x1 = max(w.x1, 0); w.y1 = max(w.y1, 0);
  return w;
}

template <bool kMax>
__global__ void __launch_bounds__(kThreads) pool_fwd_tiled(float* __restrict__ y, float const* __restrict__ x, const __grid_constant__ TileParams t)
{
  vlb::pdl_wait();
  extern __shared__ float xs[];
  PoolParams const& p = t.p;
  Tile const r = tile_of(t, false);
  load_tile(xs, x, t, r);
  __syncthreads();
  int const wp = (r.w1 - r.w0) * p.Ho, n = r.planes * wp;
  float* const yp = y + (r.z0 * p.Wo + r.w0) * (size_t)p.Ho;              // (several planes: w0 = 0, so the outputs are contiguous too)
  for (int i = threadIdx.x; i < n; i += kThreads) {
    int const pl = t.planesPerTile > 1 ? t.winPlane(i) : 0, q = i - pl * wp, wl = t.Ho(q), ho = q - wl * p.Ho;
    Window const w = window_of(p, ho, r.w0 + wl);
    float const* const xp = xs + (t.planesPerTile > 1 ? pl * p.H * p.W : 0);
    if (kMax) {
      float best = -INFINITY;
      for (int u = w.x1; u < w.x2; ++u)
        for (int v = w.y1; v < w.y2; ++v) { float const a = xp[(u - r.c0) * p.H + v]; best = (best < a) ? a : best; }
      yp[i] = best;
    } else {
      float s = 0.f;
      for (int u = w.x1; u < w.x2; ++u)
        for (int v = w.y1; v < w.y2; ++v) s = __fadd_rn(s, xp[(u - r.c0) * p.H + v]);
      yp[i] = __fmul_rn(s, __fdiv_rn(1.f, (float)((w.y2 - w.y1) * (w.x2 - w.x1))));
    }
  }
}

// relu: as for pool_bwd_generic.
template <bool kMax>
__global__ void __launch_bounds__(kThreads) pool_bwd_tiled(float* __restrict__ dx, float const* __restrict__ x, float const* __restrict__ dy,
                                                           const __grid_constant__ TileParams t, bool relu)
{
  vlb::pdl_wait();
  extern __shared__ float smem[];
  PoolParams const& p = t.p;
  Tile const r = tile_of(t, true);
  bool const needX = kMax || relu;
  float* const xs = smem;                                               // [planes][columns][H]
  float* const ds = smem + (needX ? t.planesPerTile * t.xCols * p.H : 0);      // derivative of each window (average: times its scale)
  int* const arg = reinterpret_cast<int*>(ds + t.planesPerTile * t.winCols * p.Ho);      // arg-max of each window, as an index into the plane's part of xs
  if (needX) load_tile(xs, x, t, r);
  if (kMax) __syncthreads();
  int const wp = (r.w1 - r.w0) * p.Ho, nWin = r.planes * wp;
  float const* const dyp = dy + (r.z0 * p.Wo + r.w0) * (size_t)p.Ho;
  for (int i = threadIdx.x; i < nWin; i += kThreads) {
    float const d = __ldg(dyp + i);
    int const pl = t.planesPerTile > 1 ? t.winPlane(i) : 0, q = i - pl * wp, wl = t.Ho(q), ho = q - wl * p.Ho;
    Window const w = window_of(p, ho, r.w0 + wl);
    if (kMax) {
      float const* const xp = xs + (t.planesPerTile > 1 ? pl * p.H * p.W : 0);
      // the reference's scan: column-outer, row-inner, first strictly greater wins
      float best = -INFINITY;
      int at = -1;
      for (int u = w.x1; u < w.x2; ++u)
        for (int v = w.y1; v < w.y2; ++v) {
          int const k = (u - r.c0) * p.H + v;
          float const a = xp[k];
          if (a > best) { best = a; at = k; }
        }
      ds[i] = d;
      arg[i] = at;
    } else {
      ds[i] = __fmul_rn(d, __fdiv_rn(1.f, (float)((w.y2 - w.y1) * (w.x2 - w.x1))));
    }
  }
  __syncthreads();
  int const xp = (r.u1 - r.u0) * p.H, n = r.planes * xp;
  float* const out = dx + (r.z0 * p.W + r.u0) * (size_t)p.H;
  for (int i = threadIdx.x; i < n; i += kThreads) {
    int const pl = t.planesPerTile > 1 ? t.xPlane(i) : 0, q = i - pl * xp, ul = t.H(q), v = q - ul * p.H, u = r.u0 + ul;
    int const self = (u - r.c0) * p.H + v;
    int const hb = v + p.padTop - p.poolH + 1, wb = u + p.padLeft - p.poolW + 1;
    int const ho0 = hb > 0 ? t.sy(hb + p.strideY - 1) : 0, ho1 = min(t.sy(v + p.padTop), p.Ho - 1);
    int const wo0 = wb > 0 ? t.sx(wb + p.strideX - 1) : 0, wo1 = min(t.sx(u + p.padLeft), p.Wo - 1);
    float acc = 0.f;
    for (int wo = wo0; wo <= wo1; ++wo)
      for (int ho = ho0; ho <= ho1; ++ho) {
        int const k = pl * wp + (wo - r.w0) * p.Ho + ho;
        if (!kMax || arg[k] == self) acc = __fadd_rn(acc, ds[k]);
      }
    if (relu) acc = xs[(t.planesPerTile > 1 ? pl * p.H * p.W : 0) + self] > 0.f ? acc : 0.f;
    out[i] = acc;
  }
}

// 3x3 windows two apart (AlexNet, CIFAR, ResNet): pool_bwd_tiled's general loops cost about 130 instructions per element there.  A
// thread finds a window's arg-max with the nine reads unrolled; then it takes the 2 x 2 elements around (2k - padTop, 2l - padLeft),
// which only the windows (k-1..k, l-1..l) reach -- four arg-maxima and four derivatives for four elements -- from tables with a border of
// "no window", and the result leaves through shared memory in whole lines.  55x55x96x128: 1273 us (generic), 292 (tiled), 132 (this).
template <bool kMax>
__global__ void __launch_bounds__(kThreads) pool33_bwd_tiled(float* __restrict__ dx, float const* __restrict__ x, float const* __restrict__ dy,
                                                             const __grid_constant__ TileParams t, bool relu)
{
  vlb::pdl_wait();
  extern __shared__ float smem[];
  PoolParams const& p = t.p;
  Tile const r = tile_of(t, true);
  int const H = p.H, Ho = p.Ho, Hw = Ho + 2;                             // window tables: rows -1 .. Ho, columns w0-1 .. w1
  int const xPer = t.planesPerTile > 1 ? H * p.W : 0, wCols = r.w1 - r.w0, tab = (wCols + 2) * Hw;
  float* const xs = smem;
  float* const ds = smem + t.planesPerTile * t.xCols * H;
  int* const arg = reinterpret_cast<int*>(ds + t.planesPerTile * (t.winCols + 2) * Hw);
  if (kMax || relu) load_tile(xs, x, t, r);
  for (int i = threadIdx.x; i < r.planes * tab; i += kThreads) { ds[i] = 0.f; if (kMax) arg[i] = -1; }
  __syncthreads();
  int const wp = wCols * Ho, nWin = r.planes * wp;
  float const* const dyp = dy + (r.z0 * p.Wo + r.w0) * (size_t)Ho;
  for (int i = threadIdx.x; i < nWin; i += kThreads) {
    float const d = __ldg(dyp + i);
    int const pl = t.planesPerTile > 1 ? t.winPlane(i) : 0, q = i - pl * wp, wl = t.Ho(q), ho = q - wl * Ho;
    int const x1 = 2 * (r.w0 + wl) - p.padLeft, y1 = 2 * ho - p.padTop, k = pl * tab + (wl + 1) * Hw + ho + 1;
    if (kMax) {
      float const* const xp = xs + pl * xPer;
      float best = -INFINITY;
      int at = -1;
      int const base = (x1 - r.c0) * H + y1;
      if (x1 >= 0 && y1 >= 0 && x1 + 3 <= p.W && y1 + 3 <= H) {
#pragma unroll
        for (int u = 0; u < 3; ++u)
#pragma unroll
          for (int v = 0; v < 3; ++v) {
            float const a = xp[base + u * H + v];
            if (a > best) { best = a; at = base + u * H + v; }
          }
      } else {
        for (int u = max(-x1, 0); u < min(3, p.W - x1); ++u)
          for (int v = max(-y1, 0); v < min(3, H - y1); ++v) {
            float const a = xp[base + u * H + v];
            if (a > best) { best = a; at = base + u * H + v; }
          }
      }
      ds[k] = d;
      arg[k] = at;
    } else {
      int const n = (min(x1 + 3, p.W) - max(x1, 0)) * (min(y1 + 3, H) - max(y1, 0));
      ds[k] = __fmul_rn(d, __fdiv_rn(1.f, (float)n));
    }
  }
  __syncthreads();
  // blocks of 2 x 2 elements: rows 2k - padTop + {0, 1}, columns 2l - padLeft + {0, 1}, from the first block that touches the tile
  int const k0 = p.padTop >> 1, kN = ((H - 1 + p.padTop) >> 1) - k0 + 1;
  int const l0 = (r.u0 + p.padLeft) >> 1, lN = ((r.u1 - 1 + p.padLeft) >> 1) - l0 + 1, blk = kN * lN;
  for (int i = threadIdx.x; i < r.planes * blk; i += kThreads) {
    int const pl = t.planesPerTile > 1 ? t.blkPlane(i) : 0, q = i - pl * blk, ll = t.blkRows(q), k = k0 + q - ll * kN, l = l0 + ll;
    int const v0 = 2 * k - p.padTop, u0 = 2 * l - p.padLeft;
    // table entries of the windows (k-1, k) x (l-1, l); windows below or right of the last one are border
    int const ka = min(k - 1, Ho) + 1, kb = min(k, Ho) + 1, la = min(max(l - 1 - r.w0, -1), wCols) + 1, lb = min(max(l - r.w0, -1), wCols) + 1;
    int const w00 = pl * tab + la * Hw + ka, w01 = pl * tab + la * Hw + kb, w10 = pl * tab + lb * Hw + ka, w11 = pl * tab + lb * Hw + kb;
    float const d00 = ds[w00], d01 = ds[w01], d10 = ds[w10], d11 = ds[w11];
    int a00 = 0, a01 = 0, a10 = 0, a11 = 0;
    if (kMax) { a00 = arg[w00]; a01 = arg[w01]; a10 = arg[w10]; a11 = arg[w11]; }
    float* const xp = xs + pl * xPer;
    int const s = (u0 - r.c0) * H + v0;
    // (the order of the reference: wo outer, ho inner; an absent window of an average adds its zero, which changes no sum)
    auto put = [&](int u, int v, int self, float acc) {
      if ((unsigned)v < (unsigned)H && u >= r.u0 && u < r.u1) xp[self] = relu && !(xp[self] > 0.f) ? 0.f : acc;
    };
    float acc = 0.f;
    if (!kMax || a00 == s) acc = __fadd_rn(acc, d00);
    if (!kMax || a01 == s) acc = __fadd_rn(acc, d01);
    if (!kMax || a10 == s) acc = __fadd_rn(acc, d10);
    if (!kMax || a11 == s) acc = __fadd_rn(acc, d11);
    put(u0, v0, s, acc);
    acc = 0.f;
    if (!kMax || a01 == s + 1) acc = __fadd_rn(acc, d01);
    if (!kMax || a11 == s + 1) acc = __fadd_rn(acc, d11);
    put(u0, v0 + 1, s + 1, acc);
    acc = 0.f;
    if (!kMax || a10 == s + H) acc = __fadd_rn(acc, d10);
    if (!kMax || a11 == s + H) acc = __fadd_rn(acc, d11);
    put(u0 + 1, v0, s + H, acc);
    acc = 0.f;
    if (!kMax || a11 == s + H + 1) acc = __fadd_rn(acc, d11);
    put(u0 + 1, v0 + 1, s + H + 1, acc);
  }
  __syncthreads();
  int const n = r.planes * (r.u1 - r.u0) * H, off = (r.u0 - r.c0) * H;
  float* const out = dx + (r.z0 * p.W + r.u0) * (size_t)H;
  for (int i = threadIdx.x; i < n; i += kThreads) out[i] = xs[off + i];
}

// Tile sizes for a shared-memory budget that leaves six blocks of 256 threads per SM; false when not even the narrowest strip fits it
// (columns of thousands of rows: the generic kernels).
constexpr size_t kTileBytes = 36 * 1024;

bool is_33s2(PoolParams const& p) { return p.poolH == 3 && p.poolW == 3 && p.strideY == 2 && p.strideX == 2; }

bool plan_tiles(PoolParams const& p, bool backward, bool needX, bool max, TileParams* t, size_t* smem, unsigned* grid)
{
  bool const t33 = backward && is_33s2(p);         // (its result passes through the x tile, its window tables have a border)
  if (t33) needX = true;
  size_t const winBytes = backward ? (max ? 8 : 4) : 0;
  // (planned as if x were always loaded, which also bounds the elements per tile)
  auto bytes = [&](int xCols, int winCols) { return (size_t)xCols * p.H * 4 + (t33 ? (size_t)(winCols + 2) * (p.Ho + 2) : (size_t)winCols * p.Ho) * winBytes; };
  t->p = p;
  // the multiply-for-division of the stride: positions reach H + padTop and W + padLeft
  auto divides = [](long long extent, long long pad, long long pool, long long stride) { return (extent + pad + pool + stride) * stride < (1LL << 31); };
  if (!divides(p.H, p.padTop, p.poolH, p.strideY) || !divides(p.W, p.padLeft, p.poolW, p.strideX)) return false;
  size_t const whole = bytes(p.W, p.Wo);
  t->cols = backward ? p.W : p.Wo; t->tilesPerPlane = 1; t->xCols = p.W; t->winCols = p.Wo;
  t->planesPerTile = 1;
  if (whole <= kTileBytes) {
    // several small planes per block: at least 1024 elements of work, as long as there are blocks enough for the chip
    size_t const elems = (size_t)(backward ? p.H * p.W : p.Ho * p.Wo);
    size_t n = std::min<size_t>(kTileBytes / std::max<size_t>(whole, 1), std::max<size_t>(1, 2048 / elems));
    while (n > 1 && (p.planes + n - 1) / n < 148 * 4) n = (n + 1) / 2;
    if (n * std::max((size_t)p.H * p.W, (size_t)p.Ho * p.Wo) < 65536) t->planesPerTile = (int)std::max<size_t>(1, n);
  } else {
    auto fits = [&](int cols, int* xc, int* wc) {
      if (backward) { *wc = std::min(p.Wo, (cols + p.poolW - 2) / p.strideX + 2); *xc = std::min(p.W, cols + 2 * (p.poolW - 1)); }
      else          { *wc = cols; *xc = std::min(p.W, (cols - 1) * p.strideX + p.poolW); }
      return bytes(*xc, *wc) <= kTileBytes;
    };
    int cols = t->cols, xc = 0, wc = 0;
    while (cols > 1 && !fits(cols, &xc, &wc)) cols = (cols + 1) / 2;
    if (!fits(cols, &xc, &wc)) return false;
    t->cols = cols; t->xCols = xc; t->winCols = wc;
    t->tilesPerPlane = ((backward ? p.W : p.Wo) + cols - 1) / cols;
  }
  size_t const blocks = t->planesPerTile > 1 ? (p.planes + t->planesPerTile - 1) / t->planesPerTile : p.planes * t->tilesPerPlane;
  if (blocks >= (1u << 31) || (long long)t->winCols * p.Ho * p.Ho >= (1LL << 32)) return false;
  *grid = (unsigned)blocks;
  *smem = (bytes(t->xCols, t->winCols) - (needX ? 0 : (size_t)t->xCols * p.H * 4)) * t->planesPerTile;
  // the 2 x 2 blocks of pool33_bwd_tiled (the plane's decomposition is only used with whole planes)
  int const kN = ((p.H - 1 + p.padTop) >> 1) - (p.padTop >> 1) + 1, lN = ((p.W - 1 + p.padLeft) >> 1) - (p.padLeft >> 1) + 1;
  t->blkRows = FastDiv(kN); t->blkPlane = FastDiv(kN * lN);
  t->H = FastDiv(p.H); t->Ho = FastDiv(p.Ho); t->sy = FastDiv(p.strideY); t->sx = FastDiv(p.strideX);
  t->xPlane = FastDiv(p.H * p.W); t->winPlane = FastDiv(p.Ho * p.Wo);
  return true;
}

// ------------------------------------------------------------------ 2x2 / stride 2 fast path
// kV outputs (consecutive ho) per thread; loads 2*kV floats from each of the two columns.
template <int kV> struct VecT;
template <> struct VecT<1> { typedef float2 in_t; typedef float out_t; };
template <> struct VecT<2> { typedef float4 in_t; typedef float2 out_t; };

__device__ __forceinline__ void unpack(float2 v, float* o) { o[0] = v.x; o[1] = v.y; }
__device__ __forceinline__ void unpack(float4 v, float* o) { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
__device__ __forceinline__ void pack(float2& v, float const* o) { v.x = o[0]; v.y = o[1]; }
__device__ __forceinline__ void pack(float4& v, float const* o) { v.x = o[0]; v.y = o[1]; v.z = o[2]; v.w = o[3]; }
__device__ __forceinline__ void unpack(float v, float* o) { o[0] = v; }
__device__ __forceinline__ void pack(float& v, float const* o) { v = o[0]; }

template <int kV, bool kMax>
__global__ void pool2x2_fwd(float* __restrict__ y, float const* __restrict__ x, int H, int W, size_t planes)
{
  vlb::pdl_wait();
  typedef typename VecT<kV>::in_t in_t;
  typedef typename VecT<kV>::out_t out_t;
  int Ho = H >> 1, Wo = W >> 1, Hv = Ho / kV;
  size_t total = planes * (size_t)Wo * Hv;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    int hv = (int)(i % Hv);
    size_t col = i / Hv;                       // = wo + Wo * z
    size_t z = col / Wo;
    int wo = (int)(col - z * Wo);
    float const* base = x + (z * W + 2 * (size_t)wo) * H + 2 * kV * (size_t)hv;
    float a[2 * kV], b[2 * kV], o[kV];
    unpack(*reinterpret_cast<in_t const*>(base), a);
    unpack(*reinterpret_cast<in_t const*>(base + H), b);
#pragma unroll
    for (int j = 0; j < kV; ++j) {
      if (kMax) {
        float best = -INFINITY;
        best = (best < a[2 * j]) ? a[2 * j] : best;
        best = (best < a[2 * j + 1]) ? a[2 * j + 1] : best;
        best = (best < b[2 * j]) ? b[2 * j] : best;
        best = (best < b[2 * j + 1]) ? b[2 * j + 1] : best;
        o[j] = best;
      } else {
        float s = __fadd_rn(__fadd_rn(__fadd_rn(a[2 * j], a[2 * j + 1]), b[2 * j]), b[2 * j + 1]);
        o[j] = __fmul_rn(s, 0.25f);
      }
    }
    out_t ov;
    pack(ov, o);
    *reinterpret_cast<out_t*>(y + col * Ho + kV * (size_t)hv) = ov;
  }
}

template <int kV, bool kMax, bool kRelu>
__global__ void pool2x2_bwd(float* __restrict__ dx, float const* __restrict__ x, float const* __restrict__ dy,
                            int H, int W, size_t planes)
{
  vlb::pdl_wait();
  typedef typename VecT<kV>::in_t in_t;
  typedef typename VecT<kV>::out_t out_t;
  int Ho = H >> 1, Wo = W >> 1, Hv = Ho / kV;
  size_t total = planes * (size_t)Wo * Hv;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    int hv = (int)(i % Hv);
    size_t col = i / Hv;
    size_t z = col / Wo;
    int wo = (int)(col - z * Wo);
    size_t off = (z * W + 2 * (size_t)wo) * H + 2 * kV * (size_t)hv;
    float d[kV], ra[2 * kV], rb[2 * kV];
    unpack(*reinterpret_cast<out_t const*>(dy + col * Ho + kV * (size_t)hv), d);
    float a[2 * kV], b[2 * kV];
    if (kMax || kRelu) {
      unpack(*reinterpret_cast<in_t const*>(x + off), a);
      unpack(*reinterpret_cast<in_t const*>(x + off + H), b);
    }
    if (kMax) {
#pragma unroll
      for (int j = 0; j < kV; ++j) {
        // scan order of the reference: column 0 rows 0,1 then column 1 rows 0,1; strict '>'
        float best = -INFINITY;
        int w = -1;
        if (a[2 * j] > best) { best = a[2 * j]; w = 0; }
        if (a[2 * j + 1] > best) { best = a[2 * j + 1]; w = 1; }
        if (b[2 * j] > best) { best = b[2 * j]; w = 2; }
        if (b[2 * j + 1] > best) { best = b[2 * j + 1]; w = 3; }
        float g = __fadd_rn(0.f, d[j]);   // the reference adds dy to a zero-filled dx: -0 becomes +0
        ra[2 * j] = (w == 0) ? g : 0.f;
        ra[2 * j + 1] = (w == 1) ? g : 0.f;
        rb[2 * j] = (w == 2) ? g : 0.f;
        rb[2 * j + 1] = (w == 3) ? g : 0.f;
      }
    } else {
#pragma unroll
      for (int j = 0; j < kV; ++j) {
        float g = __fadd_rn(0.f, __fmul_rn(d[j], 0.25f));
        ra[2 * j] = g; ra[2 * j + 1] = g; rb[2 * j] = g; rb[2 * j + 1] = g;
      }
    }
    if (kRelu) {
#pragma unroll
      for (int j = 0; j < 2 * kV; ++j) { ra[j] = a[j] > 0.f ? ra[j] : 0.f; rb[j] = b[j] > 0.f ? rb[j] : 0.f; }
    }
    in_t va, vb;
    pack(va, ra);
    pack(vb, rb);
    *reinterpret_cast<in_t*>(dx + off) = va;
    *reinterpret_cast<in_t*>(dx + off + H) = vb;
  }
}

bool fast2x2(vlb_pool_desc const* d, void const* a, void const* b, void const* c)
{
  bool shape = d->poolH == 2 && d->poolW == 2 && d->strideY == 2 && d->strideX == 2 && d->padTop == 0 &&
               d->padBottom == 0 && d->padLeft == 0 && d->padRight == 0 && (d->H % 2 == 0) && (d->W % 2 == 0);
  uintptr_t bits = (uintptr_t)a | (uintptr_t)b | (uintptr_t)c;
  return shape && (bits & 15) == 0;
}

int validate(vlb_ctx* ctx, vlb_pool_desc const* d, int* Ho, int* Wo)
{
  VLB_REQUIRE(ctx, d, "pooling: null descriptor");
  VLB_REQUIRE(ctx, d->H > 0 && d->W > 0 && d->C > 0 && d->N > 0, "pooling: empty input");
  VLB_REQUIRE(ctx, d->poolH >= 1 && d->poolW >= 1, "pooling: POOL has a dimension smaller than 1");
  VLB_REQUIRE(ctx, d->strideY >= 1 && d->strideX >= 1, "pooling: STRIDE smaller than 1");
  VLB_REQUIRE(ctx, d->padTop >= 0 && d->padBottom >= 0 && d->padLeft >= 0 && d->padRight >= 0, "pooling: negative PAD");
  VLB_REQUIRE(ctx, d->H + d->padTop + d->padBottom >= d->poolH && d->W + d->padLeft + d->padRight >= d->poolW,
              "pooling: pooling window larger than the padded input");
  // The gateway rejects a padding as large as the window (matlab/src/vl_nnpool.cu:232-237).
  VLB_REQUIRE(ctx, d->padTop < d->poolH && d->padBottom < d->poolH && d->padLeft < d->poolW && d->padRight < d->poolW,
              "pooling: padding larger or equal than the pooling window");
  VLB_REQUIRE(ctx, d->method == VLB_POOL_MAX || d->method == VLB_POOL_AVG, "pooling: unknown method");
  vlb_pool_output_shape(d, Ho, Wo);
  return VLB_Success;
}

}  // namespace

namespace {

template <int kV, bool kMax>
void launch2x2_bwd(vlb_ctx* ctx, unsigned grid, float* dX, float const* X, float const* dY, int H, int W, size_t planes, bool relu)
{
  if (relu) vlb::launch(ctx->stream, pool2x2_bwd<kV, kMax, true>, grid, kThreads, 0, dX, X, dY, H, W, planes);
  else      vlb::launch(ctx->stream, pool2x2_bwd<kV, kMax, false>, grid, kThreads, 0, dX, X, dY, H, W, planes);
}

int pool_backward(vlb_ctx* ctx, float* dX, float const* X, float const* dY, vlb_pool_desc const* d, bool relu, char const* where)
{
  if (!ctx) return VLB_IllegalArgument;
  int Ho, Wo;
  int rc = validate(ctx, d, &Ho, &Wo);
  if (rc) return vlb::pass_error(ctx, rc, where);
  VLB_REQUIRE(ctx, dX && X && dY, "pool_backward: null tensor");
  size_t planes = (size_t)d->C * d->N;
  bool isMax = d->method == VLB_POOL_MAX;
  if (fast2x2(d, dX, X, dY)) {
    bool v2 = (d->H % 4 == 0);
    size_t total = planes * (size_t)Wo * (v2 ? Ho / 2 : Ho);
    unsigned grid = vlb::grid_for(total, kThreads, ctx->smCount * 16);
    if (v2) { if (isMax) launch2x2_bwd<2, true>(ctx, grid, dX, X, dY, d->H, d->W, planes, relu);
              else       launch2x2_bwd<2, false>(ctx, grid, dX, X, dY, d->H, d->W, planes, relu); }
    else    { if (isMax) launch2x2_bwd<1, true>(ctx, grid, dX, X, dY, d->H, d->W, planes, relu);
              else       launch2x2_bwd<1, false>(ctx, grid, dX, X, dY, d->H, d->W, planes, relu); }
  } else {
    PoolParams p = {d->H, d->W, Ho, Wo, d->poolH, d->poolW, d->strideY, d->strideX, d->padTop, d->padLeft, planes};
    TileParams t;
    size_t smem = 0;
    unsigned grid = 0;
    if (plan_tiles(p, true, isMax || relu, isMax, &t, &smem, &grid)) {
      bool const t33 = is_33s2(p);
      if (t33 && isMax) vlb::launch(ctx->stream, pool33_bwd_tiled<true>, grid, kThreads, smem, dX, X, dY, t, relu);
      else if (t33)     vlb::launch(ctx->stream, pool33_bwd_tiled<false>, grid, kThreads, smem, dX, X, dY, t, relu);
      else if (isMax)   vlb::launch(ctx->stream, pool_bwd_tiled<true>, grid, kThreads, smem, dX, X, dY, t, relu);
      else              vlb::launch(ctx->stream, pool_bwd_tiled<false>, grid, kThreads, smem, dX, X, dY, t, relu);
      VLB_LAUNCHED(ctx, 1);
      return vlb::check_launch(ctx, where);
    }
    grid = vlb::grid_for(planes * (size_t)d->H * d->W, kThreads, ctx->smCount * 16);
    if (isMax) vlb::launch(ctx->stream, pool_bwd_generic<true>, grid, kThreads, 0, dX, X, dY, p, relu);
    else       vlb::launch(ctx->stream, pool_bwd_generic<false>, grid, kThreads, 0, dX, X, dY, p, relu);
  }
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, where);
}

}  // namespace

extern "C" {

int vlb_pool_output_shape(vlb_pool_desc const* d, int* Ho, int* Wo)
{
  if (!d) return VLB_IllegalArgument;
  if (Ho) *Ho = (d->H + d->padTop + d->padBottom - d->poolH) / d->strideY + 1;
  if (Wo) *Wo = (d->W + d->padLeft + d->padRight - d->poolW) / d->strideX + 1;
  return VLB_Success;
}

int vlb_pool_forward(vlb_ctx* ctx, float* Y, float const* X, vlb_pool_desc const* d)
{
  if (!ctx) return VLB_IllegalArgument;
  int Ho, Wo;
  int rc = validate(ctx, d, &Ho, &Wo);
  if (rc) return vlb::pass_error(ctx, rc, "vlb_pool_forward");
  VLB_REQUIRE(ctx, Y && X, "pool_forward: null tensor");
  size_t planes = (size_t)d->C * d->N;
  bool isMax = d->method == VLB_POOL_MAX;
  if (fast2x2(d, Y, X, X)) {
    bool v2 = (d->H % 4 == 0);
    size_t total = planes * (size_t)Wo * (v2 ? Ho / 2 : Ho);
    unsigned grid = vlb::grid_for(total, kThreads, ctx->smCount * 16);
    if (v2) { if (isMax) vlb::launch(ctx->stream, pool2x2_fwd<2, true>, grid, kThreads, 0, Y, X, d->H, d->W, planes);
              else       vlb::launch(ctx->stream, pool2x2_fwd<2, false>, grid, kThreads, 0, Y, X, d->H, d->W, planes); }
    else    { if (isMax) vlb::launch(ctx->stream, pool2x2_fwd<1, true>, grid, kThreads, 0, Y, X, d->H, d->W, planes);
              else       vlb::launch(ctx->stream, pool2x2_fwd<1, false>, grid, kThreads, 0, Y, X, d->H, d->W, planes); }
  } else {
    PoolParams p = {d->H, d->W, Ho, Wo, d->poolH, d->poolW, d->strideY, d->strideX, d->padTop, d->padLeft, planes};
    TileParams t;
    size_t smem = 0;
    unsigned grid = 0;
    if (plan_tiles(p, false, true, isMax, &t, &smem, &grid)) {
      if (isMax) vlb::launch(ctx->stream, pool_fwd_tiled<true>, grid, kThreads, smem, Y, X, t);
      else       vlb::launch(ctx->stream, pool_fwd_tiled<false>, grid, kThreads, smem, Y, X, t);
      VLB_LAUNCHED(ctx, 1);
      return vlb::check_launch(ctx, "vlb_pool_forward");
    }
    grid = vlb::grid_for(planes * (size_t)Ho * Wo, kThreads, ctx->smCount * 16);
    if (isMax) vlb::launch(ctx->stream, pool_fwd_generic<true>, grid, kThreads, 0, Y, X, p);
    else       vlb::launch(ctx->stream, pool_fwd_generic<false>, grid, kThreads, 0, Y, X, p);
  }
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, "vlb_pool_forward");
}

int vlb_pool_backward(vlb_ctx* ctx, float* dX, float const* X, float const* dY, vlb_pool_desc const* d)
{
  return pool_backward(ctx, dX, X, dY, d, false, "vlb_pool_backward");
}

int vlb_relu_pool_backward(vlb_ctx* ctx, float* dX, float const* X, float const* dY, vlb_pool_desc const* d)
{
  return pool_backward(ctx, dX, X, dY, d, true, "vlb_relu_pool_backward");
}

}  // extern "C"
