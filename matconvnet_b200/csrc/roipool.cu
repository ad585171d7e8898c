// ROI pooling (vl::nn::ROIPooling, reference bits/nnroipooling.hpp:23-45; CPU definition
// bits/nnroipooling.cu:102-189 forward, :217-305 backward).
//
// The bin geometry follows the CPU reference's arithmetic exactly -- affine map in
// double rounded to float, round-half-away, bin size as a double quotient rounded to
// float, float products with floor/ceil (bits/nnroipooling.cu:129-165) -- using the
// _rn intrinsics so that no multiply-add is contracted; the reference's own GPU code
// does the same maths in float throughout and can differ in the last place.
// Forward: one thread per output bin and four channels, whose planes lie side by side in shared memory; maps too large for that
// are read from global memory, one thread per output bin and channel.  The scan order for the arg-max is
// the CPU's (w outer, h inner, first strictly greater).
//
// Backward (max) does not scatter with atomics as the reference GPU code does
// (bits/impl/nnroipooling_gpu.cu:114-246).  One CTA takes one image and a few channels.  All its
// threads first find, from the input plane in shared memory, the arg-max pixel of every bin of every
// ROI of the image; then one warp per channel walks the bins in the order of the CPU loop (ROI, bin
// column, bin row; bits/nnroipooling.cu:239-300), 32 at a time, and adds their derivatives to a copy
// of the channel's dX plane in shared memory, the additions of one step to one pixel in lane order.  The work is proportional to the
// number of bins, the sums are the CPU's bit for bit and identical from run to run, dX is written
// exactly once (no zero fill), and nothing but x, dY and dX crosses HBM.  Backward (avg), where every
// pixel of a bin receives a share, is a gather: every pixel of a channel slab walks the ROIs that
// cover it, in the same order.  Maps too large for shared memory take a zero fill and an atomic
// scatter.
#include "common.cuh"
#include <math.h>
#include <algorithm>

namespace {

constexpr int kThreads = 256;

struct RoiParams {
  int H, W, C, N, numROIs, S0, S1;
  double tf[6];
};

struct RoiGeom { int image, start_h, start_w; float bin_h, bin_w; };

__device__ __forceinline__ RoiGeom roi_geom(float const* r, RoiParams const& p)
{
  RoiGeom g;
  double u1_ = (double)r[1], v1_ = (double)r[2], u2_ = (double)r[3], v2_ = (double)r[4];
  // (tf0*u + tf2*v) + tf4, each step rounded to double: no fused multiply-add
  float u1 = (float)__dadd_rn(__dadd_rn(__dmul_rn(p.tf[0], u1_), __dmul_rn(p.tf[2], v1_)), p.tf[4]);
  float v1 = (float)__dadd_rn(__dadd_rn(__dmul_rn(p.tf[1], u1_), __dmul_rn(p.tf[3], v1_)), p.tf[5]);
  float u2 = (float)__dadd_rn(__dadd_rn(__dmul_rn(p.tf[0], u2_), __dmul_rn(p.tf[2], v2_)), p.tf[4]);
  float v2 = (float)__dadd_rn(__dadd_rn(__dmul_rn(p.tf[1], u2_), __dmul_rn(p.tf[3], v2_)), p.tf[5]);
  int image = (int)r[0];
  // ::round on the float promoted to double (bits/nnroipooling.cu:137-140)
  g.start_h = (int)round((double)v1) - 1;
  g.start_w = (int)round((double)u1) - 1;
  int end_h = (int)round((double)v2) - 1, end_w = (int)round((double)u2) - 1;
  int rh = max(end_h - g.start_h + 1, 1), rw = max(end_w - g.start_w + 1, 1);
  g.image = min(max(image - 1, 0), p.N - 1);
  g.bin_h = (float)((double)rh / (double)p.S0);
  g.bin_w = (float)((double)rw / (double)p.S1);
  return g;
}

__device__ __forceinline__ void roi_bin(int q, float bin, int start, int extent, int& lo, int& hi)
{
  int a = (int)floorf(__fmul_rn((float)q, bin));
  int b = (int)ceilf(__fmul_rn((float)(q + 1), bin));
  lo = min(max(a + start, 0), extent);
  hi = min(max(b + start, 0), extent);
}

__global__ void roipool_bounds_kernel(int* __restrict__ bounds, int* __restrict__ images,
                                      float const* __restrict__ rois, RoiParams p)
{
  vlb::pdl_wait();
  int total = p.S0 * p.S1 * p.numROIs;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    int ph = i % p.S0, pw = (i / p.S0) % p.S1, r = i / (p.S0 * p.S1);
    RoiGeom g = roi_geom(rois + 5 * (size_t)r, p);
    int hs, he, ws, we;
    roi_bin(ph, g.bin_h, g.start_h, p.H, hs, he);
    roi_bin(pw, g.bin_w, g.start_w, p.W, ws, we);
    bounds[4 * (size_t)i + 0] = hs; bounds[4 * (size_t)i + 1] = he;
    bounds[4 * (size_t)i + 2] = ws; bounds[4 * (size_t)i + 3] = we;
    if (images && ph == 0 && pw == 0) images[r] = g.image;
  }
}

// kBackward = false: y[bin] = max / mean.  kBackward = true: dx += routed dy.
template <bool kMax, bool kBackward>
__global__ void roipool_kernel(float* __restrict__ out, float const* __restrict__ x,
                               float const* __restrict__ rois, float const* __restrict__ dy, RoiParams p)
{
  vlb::pdl_wait();
  size_t total = (size_t)p.S0 * p.S1 * p.C * p.numROIs;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    int ph = (int)(i % p.S0);
    size_t t = i / p.S0;
    int pw = (int)(t % p.S1); t /= p.S1;
    int c = (int)(t % p.C);
    int r = (int)(t / p.C);
    RoiGeom g = roi_geom(rois + 5 * (size_t)r, p);
    int hs, he, ws, we;
    roi_bin(ph, g.bin_h, g.start_h, p.H, hs, he);
    roi_bin(pw, g.bin_w, g.start_w, p.W, ws, we);
    size_t off = (size_t)p.H * p.W * ((size_t)c + (size_t)p.C * g.image);
    float const* xz = x + off;
    bool empty = (he <= hs) || (we <= ws);
    if (!kBackward) {
      float o = 0.f;
      if (!empty) {
        if (kMax) {
          float best = -INFINITY;
          for (int w = ws; w < we; ++w)
            for (int h = hs; h < he; ++h) { float a = xz[(size_t)w * p.H + h]; best = (best < a) ? a : best; }
          o = best;
        } else {
          float s = 0.f;
          for (int w = ws; w < we; ++w)
            for (int h = hs; h < he; ++h) s = __fadd_rn(s, xz[(size_t)w * p.H + h]);
          o = __fmul_rn(s, __fdiv_rn(1.f, (float)((he - hs) * (we - ws))));
        }
      }
      out[i] = o;
    } else {
      if (empty) continue;
      float d = dy[i];
      float* dxz = out + off;
      if (kMax) {
        float best = -INFINITY;
        long where = -1;
        for (int w = ws; w < we; ++w)
          for (int h = hs; h < he; ++h) {
            float a = xz[(size_t)w * p.H + h];
            if (a > best) { best = a; where = (long)w * p.H + h; }
          }
        if (where >= 0) atomicAdd(dxz + where, d);
      } else {
        float g2 = __fmul_rn(d, __fdiv_rn(1.f, (float)((he - hs) * (we - ws))));
        for (int w = ws; w < we; ++w)
          for (int h = hs; h < he; ++h) atomicAdd(dxz + (size_t)w * p.H + h, g2);
      }
    }
  }
}

// ---- forward with the planes of four channels in shared memory ----
// The direct kernel above computes the bin geometry, in double precision, for every channel, and its scans wait for L1 at every pixel.  Here a
// block takes one image, four channels and up to RB ROIs: the geometry once per ROI into tables, the four planes side by side, and
// a bin is scanned for four channels at once.  B200, 38 x 50 x 512 x 2, 256 ROIs, 7 x 7 bins: 117 -> 35 us.
constexpr int kFwdThreads = 256;

__host__ __device__ inline size_t fwd_smem(int RB, long long HW, int S0, int S1)
{ return sizeof(float4) * (size_t)HW + sizeof(uint32_t) * (size_t)RB * (S0 + S1) + sizeof(int) * (size_t)RB; }

// start | end << 16 of every bin row and bin column of nb ROIs (the double-precision part of the arithmetic, once per ROI)
__device__ __forceinline__ void bin_tables(uint32_t* binRow, uint32_t* binCol, int const* roiIdx, int nb, float const* rois, RoiParams const& p)
{
  for (int i = threadIdx.x; i < nb * (p.S0 + p.S1); i += blockDim.x) {
    bool const isRow = i < nb * p.S0;
    int const k = isRow ? i : i - nb * p.S0;
    int const S = isRow ? p.S0 : p.S1;
    int const j = k / S, b = k - j * S;
    RoiGeom g = roi_geom(rois + 5 * (size_t)roiIdx[j], p);
    int s, e;
    roi_bin(b, isRow ? g.bin_h : g.bin_w, isRow ? g.start_h : g.start_w, isRow ? p.H : p.W, s, e);
    (isRow ? binRow : binCol)[k] = (uint32_t)s | ((uint32_t)e << 16);
  }
}

template <bool kMax>
__global__ void __launch_bounds__(kFwdThreads)
roipool_fwd_planes_kernel(float* __restrict__ y, float const* __restrict__ x, float const* __restrict__ rois, RoiParams p, int RB, int parts, int quads)
{
  vlb::pdl_wait();
  extern __shared__ __align__(16) uint8_t sm[];
  __shared__ int sCount;
  int const HW = p.H * p.W, bins = p.S0 * p.S1, tid = threadIdx.x;
  int const plane = blockIdx.x / parts, part = blockIdx.x - plane * parts;
  int const img = plane / quads, c0 = (plane - img * quads) * 4, nc = min(4, p.C - c0);
  float4* const xs = reinterpret_cast<float4*>(sm);
  uint32_t* const binRow = reinterpret_cast<uint32_t*>(xs + HW);
  uint32_t* const binCol = binRow + (size_t)RB * p.S0;
  int* const roiIdx = reinterpret_cast<int*>(binCol + (size_t)RB * p.S1);
  if (tid == 0) sCount = 0;
  __syncthreads();
  // the ROIs of this part that lie on this image, in any order
  for (int r = part * RB + tid; r < min(p.numROIs, (part + 1) * RB); r += kFwdThreads)
    if (min(max((int)rois[5 * (size_t)r] - 1, 0), p.N - 1) == img) roiIdx[atomicAdd(&sCount, 1)] = r;
  __syncthreads();
  int const nb = sCount;
  if (nb == 0) return;
  vlb::stage_planes(xs, x + (size_t)HW * ((size_t)c0 + (size_t)p.C * img), HW, nc);
  bin_tables(binRow, binCol, roiIdx, nb, rois, p);
  __syncthreads();
  float const invBins = 1.f / (float)bins, invS0 = 1.f / (float)p.S0;
  for (int b = tid; b < nb * bins; b += kFwdThreads) {
    int const j = (int)(((float)b + 0.5f) * invBins), t = b - j * bins;      // (exact: see the rule in vlb_roipool_forward)
    int const pw = (int)(((float)t + 0.5f) * invS0), ph = t - pw * p.S0;
    uint32_t const rs = binRow[j * p.S0 + ph], cs = binCol[j * p.S1 + pw];
    int const hs = (int)(rs & 0xFFFFu), he = (int)(rs >> 16), ws = (int)(cs & 0xFFFFu), we = (int)(cs >> 16);
    bool const empty = he <= hs || we <= ws;
    float const v0 = kMax && !empty ? -INFINITY : 0.f;
    float4 o = make_float4(v0, v0, v0, v0);
    for (int w = ws; w < we; ++w) {
      float4 const* const col = xs + w * p.H;
#pragma unroll 2
      for (int h = hs; h < he; ++h) {
        float4 const a = col[h];
        if (kMax) {
          o.x = o.x < a.x ? a.x : o.x; o.y = o.y < a.y ? a.y : o.y; o.z = o.z < a.z ? a.z : o.z; o.w = o.w < a.w ? a.w : o.w;
        } else {
          o.x = __fadd_rn(o.x, a.x); o.y = __fadd_rn(o.y, a.y); o.z = __fadd_rn(o.z, a.z); o.w = __fadd_rn(o.w, a.w);
        }
      }
    }
    if (!kMax && !empty) {
      float const inv = __fdiv_rn(1.f, (float)((he - hs) * (we - ws)));
      o.x = __fmul_rn(o.x, inv); o.y = __fmul_rn(o.y, inv); o.z = __fmul_rn(o.z, inv); o.w = __fmul_rn(o.w, inv);
    }
    float* const q = y + (size_t)bins * ((size_t)c0 + (size_t)p.C * roiIdx[j]) + t;
    q[0] = o.x;
    if (nc > 1) q[bins] = o.y;
    if (nc > 2) q[2 * bins] = o.z;
    if (nc > 3) q[3 * bins] = o.w;
  }
}

// ---- backward as a gather (see the header comment) ----
constexpr int kGatherThreads = 1024;
constexpr uint32_t kNoBin = 0xFFFFu;

// Shared-memory layout (bytes): slab float[CH*HW] (max only) | argmax uint16[RB*CH*S0*S1] (max only) |
// binRow uint32[RB*S0], binCol uint32[RB*S1]: start | end << 16 of every bin row / column of every ROI of the batch |
// rowMask uint32[H*words], colMask uint32[W*words]: bit j of word k set when ROI 32k+j of the batch covers that map row /
// column | rowTab uint16[RB*H], colTab uint16[RB*W]: lo | hi << 8, the bin rows / columns covering it, or kNoBin | roiIdx int[RB].
__host__ __device__ inline size_t gather_smem(int CH, int RB, int H, int W, int S0, int S1, bool isMax)
{
  int const words = (RB + 31) / 32;
  size_t b = isMax ? sizeof(float) * (size_t)CH * H * W : 0;
  b += isMax ? ((sizeof(uint16_t) * (size_t)RB * CH * S0 * S1 + 15) & ~(size_t)15) : 0;
  b += sizeof(uint32_t) * (size_t)RB * (S0 + S1);
  b += sizeof(uint32_t) * (size_t)words * (H + W);
  b += (sizeof(uint16_t) * (size_t)RB * (H + W) + 15) & ~(size_t)15;
  b += sizeof(int) * (size_t)RB;
  return b + 64;
}

template <bool kMax>
__global__ void __launch_bounds__(kGatherThreads, 1)
roipool_bwd_gather_kernel(float* __restrict__ dx, float const* __restrict__ x, float const* __restrict__ rois,
                          float const* __restrict__ dy, RoiParams p, int CH, int RB, int chunks)
{
  vlb::pdl_wait();
  extern __shared__ __align__(16) uint8_t sm[];
  __shared__ int sCount, sNext;
  int const HW = p.H * p.W, bins = p.S0 * p.S1, words = (RB + 31) / 32;
  int const img = blockIdx.x / chunks, c0 = (blockIdx.x % chunks) * CH;
  int const nch = min(CH, p.C - c0);
  int const tid = threadIdx.x, lane = tid & 31;
  uint8_t* q = sm;
  float* slab = reinterpret_cast<float*>(q);
  if (kMax) q += sizeof(float) * (size_t)CH * HW;
  uint16_t* am = reinterpret_cast<uint16_t*>(q);
  if (kMax) q += (sizeof(uint16_t) * (size_t)RB * CH * bins + 15) & ~(size_t)15;
  uint32_t* binRow = reinterpret_cast<uint32_t*>(q);
  uint32_t* binCol = binRow + (size_t)RB * p.S0;
  uint32_t* rowMask = binCol + (size_t)RB * p.S1;
  uint32_t* colMask = rowMask + (size_t)words * p.H;
  uint16_t* rowTab = reinterpret_cast<uint16_t*>(colMask + (size_t)words * p.W);
  uint16_t* colTab = rowTab + (size_t)RB * p.H;
  q = reinterpret_cast<uint8_t*>(rowTab) + ((sizeof(uint16_t) * (size_t)RB * (p.H + p.W) + 15) & ~(size_t)15);
  int* roiIdx = reinterpret_cast<int*>(q);

  size_t const slabOff = (size_t)HW * ((size_t)c0 + (size_t)p.C * img);
  if (kMax) {
    for (int i = tid; i < nch * HW; i += kGatherThreads) slab[i] = x[slabOff + i];
  }
  bool first = true;
  int base = 0;
  while (true) {
    __syncthreads();                                  // the previous batch's tables are no longer read
    if (tid < 32) {
      // the next RB ROIs of this image, in ascending order
      int cnt = 0, r = base;
      while (r < p.numROIs && cnt < RB) {
        int const rr = r + lane;
        bool mine = false;
        if (rr < p.numROIs) {
          int image = (int)rois[5 * (size_t)rr];
          mine = min(max(image - 1, 0), p.N - 1) == img;
        }
        unsigned const m = __ballot_sync(0xffffffffu, mine);
        int const pos = cnt + __popc(m & ((1u << lane) - 1u));
        if (mine && pos < RB) roiIdx[pos] = rr;
        int const tot = __popc(m);
        if (cnt + tot > RB) {                           // the batch is full inside this group of 32: resume behind its last member
          r += (int)__fns(m, 0, RB - cnt) + 1;
          cnt = RB;
          break;
        }
        cnt += tot; r += 32;
      }
      if (lane == 0) { sCount = cnt; sNext = min(r, p.numROIs); }
    }
    __syncthreads();
    int const nb = sCount;
    base = sNext;
    if (nb == 0) break;
    bin_tables(binRow, binCol, roiIdx, nb, rois, p);
    __syncthreads();
    // which bin rows cover map row h, which bin columns cover map column w
    for (int i = tid; i < nb * (p.H + p.W); i += kGatherThreads) {
      bool const isRow = i < nb * p.H;
      int const k = isRow ? i : i - nb * p.H;
      int const ext = isRow ? p.H : p.W, S = isRow ? p.S0 : p.S1;
      int const j = k / ext, pos = k - j * ext;
      uint32_t const* tab = (isRow ? binRow : binCol) + (size_t)j * S;
      uint32_t lo = kNoBin, hi = 0;
      for (int b = 0; b < S; ++b) {
        uint32_t const se = tab[b];
        if ((int)(se & 0xFFFFu) <= pos && pos < (int)(se >> 16)) { if (lo == kNoBin) lo = (uint32_t)b; hi = (uint32_t)b; }
      }
      (isRow ? rowTab : colTab)[k] = (uint16_t)(lo == kNoBin ? kNoBin : (lo | (hi << 8)));
    }
    if (kMax) {
      // arg-max of every bin: CPU scan order, first strictly greater, none for an empty or all -inf / NaN bin
      for (int b = tid; b < nb * nch * bins; b += kGatherThreads) {
        int const ph = b % p.S0;
        int t = b / p.S0;
        int const pw = t % p.S1; t /= p.S1;
        int const cc = t % nch, j = t / nch;
        uint32_t const rs = binRow[j * p.S0 + ph], cs = binCol[j * p.S1 + pw];
        int const hs = (int)(rs & 0xFFFFu), he = (int)(rs >> 16), ws = (int)(cs & 0xFFFFu), we = (int)(cs >> 16);
        float const* xz = slab + (size_t)cc * HW;
        float best = -INFINITY;
        uint32_t where = kNoBin;
        for (int w = ws; w < we; ++w)
          for (int h = hs; h < he; ++h) {
            float a = xz[w * p.H + h];
            if (a > best) { best = a; where = (uint32_t)(w * p.H + h); }
          }
        am[b] = (uint16_t)where;
      }
    }
    __syncthreads();
    // bit masks: the ROIs of the batch that cover a map row / column, so that a pixel visits only ROIs that contain it
    for (int i = tid; i < words * (p.H + p.W); i += kGatherThreads) {
      bool const isRow = i < words * p.H;
      int const k = isRow ? i : i - words * p.H;
      int const ext = isRow ? p.H : p.W;
      int const pos = k / words, wd = k - pos * words;
      uint16_t const* tab = isRow ? rowTab : colTab;
      uint32_t m = 0;
      for (int j = wd * 32; j < min(nb, wd * 32 + 32); ++j)
        if (tab[j * ext + pos] != kNoBin) m |= 1u << (j & 31);
      (isRow ? rowMask : colMask)[k] = m;
    }
    __syncthreads();
    for (int item = tid; item < nch * HW; item += kGatherThreads) {
      int const cc = item / HW, pix = item - cc * HW;
      int const w = pix / p.H, h = pix - w * p.H;
      float* const dst = dx + slabOff + item;
      float acc = first ? 0.f : *dst;
      for (int wd = 0; wd < words; ++wd) {
        uint32_t m = rowMask[h * words + wd] & colMask[w * words + wd];
        while (m) {
          int const j = wd * 32 + __ffs(m) - 1;          // ascending: the order of the CPU loop over the ROIs
          m &= m - 1;
          uint32_t const rt = rowTab[j * p.H + h], ct = colTab[j * p.W + w];
          float const* dyr = dy + (size_t)bins * ((size_t)(c0 + cc) + (size_t)p.C * roiIdx[j]);
          if (kMax) {
            uint16_t const* amr = am + (size_t)bins * (cc + (size_t)nch * j);
            for (uint32_t pw = ct & 255u; pw <= (ct >> 8); ++pw)
              for (uint32_t ph = rt & 255u; ph <= (rt >> 8); ++ph) {
                int const b = (int)(ph + p.S0 * pw);
                if (amr[b] == (uint32_t)pix) acc = __fadd_rn(acc, dyr[b]);
              }
          } else {
            // every bin that covers the pixel contributes dy / area (bits/nnroipooling.cu:74-90, acc_sum)
            for (uint32_t pw = ct & 255u; pw <= (ct >> 8); ++pw) {
              uint32_t const cs = binCol[j * p.S1 + pw];
              for (uint32_t ph = rt & 255u; ph <= (rt >> 8); ++ph) {
                uint32_t const rs = binRow[j * p.S0 + ph];
                int const area = (int)((rs >> 16) - (rs & 0xFFFFu)) * (int)((cs >> 16) - (cs & 0xFFFFu));
                acc = __fadd_rn(acc, __fmul_rn(dyr[ph + p.S0 * pw], __fdiv_rn(1.f, (float)area)));
              }
            }
          }
        }
      }
      *dst = acc;
    }
    first = false;
    if (base >= p.numROIs) break;
  }
  if (first) {
    // no ROI of this image: the slab of dX is zero
    for (int i = tid; i < nch * HW; i += kGatherThreads) dx[slabOff + i] = 0.f;
  }
}

// ---- backward (max): arg-max of every bin in parallel, four channels at a time, then one warp per channel adds the bins' derivatives to
// their pixels in bin order (see the header comment) ----
constexpr int kOrdThreads = 512;

// Shared memory (bytes): plane float4[HW] | dxs float[4*HW] | binRow uint32[RB*S0] | binCol uint32[RB*S1] | roiIdx int[RB] |
// am uint16[4*RB*bins]
__host__ __device__ inline size_t ordered_smem(int RB, int HW, int S0, int S1)
{ return 32 * (size_t)HW + 4 * (size_t)RB * (S0 + S1) + 4 * (size_t)RB + 8 * (size_t)RB * S0 * S1 + 64; }

// Bound by latency: the scans of the bins, then the chain of additions.  With one channel at a time and one warp per channel for the additions
// (38 x 50 x 512 x 2, 256 ROIs, 7 x 7 bins) 190 us; four channels per scan, and a step's additions without
// a pass through memory for every lane: 124 us.  Two or four warps per channel, each for a part of the pixels, were no faster.
__global__ void __launch_bounds__(kOrdThreads)
roipool_bwd_ordered_kernel(float* __restrict__ dx, float const* __restrict__ x, float const* __restrict__ rois,
                           float const* __restrict__ dy, RoiParams p, int RB, int quads)
{
  vlb::pdl_wait();
  extern __shared__ __align__(16) uint8_t sm[];
  __shared__ int sCount, sNext;
  int const HW = p.H * p.W, bins = p.S0 * p.S1;
  int const img = blockIdx.x / quads, c0 = (blockIdx.x % quads) * 4;
  int const nch = min(4, p.C - c0);
  int const tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float4* const plane = reinterpret_cast<float4*>(sm);
  float* const dxs = reinterpret_cast<float*>(plane + HW);
  uint32_t* const binRow = reinterpret_cast<uint32_t*>(dxs + 4 * (size_t)HW);
  uint32_t* const binCol = binRow + (size_t)RB * p.S0;
  int* const roiIdx = reinterpret_cast<int*>(binCol + (size_t)RB * p.S1);
  uint16_t* const am = reinterpret_cast<uint16_t*>(roiIdx + RB);
  float const invBins = 1.f / (float)bins, invS0 = 1.f / (float)p.S0;

  for (int i = tid; i < nch * HW; i += kOrdThreads) dxs[i] = 0.f;
  int base = 0;
  while (true) {
    __syncthreads();
    if (tid < 32) {
      // the next RB ROIs of this image, in ascending order
      int cnt = 0, r = base;
      while (r < p.numROIs && cnt < RB) {
        int const rr = r + lane;
        bool mine = false;
        if (rr < p.numROIs) {
          int image = (int)rois[5 * (size_t)rr];
          mine = min(max(image - 1, 0), p.N - 1) == img;
        }
        unsigned const m = __ballot_sync(0xffffffffu, mine);
        int const pos = cnt + __popc(m & ((1u << lane) - 1u));
        if (mine && pos < RB) roiIdx[pos] = rr;
        int const tot = __popc(m);
        if (cnt + tot > RB) {                           // the batch is full inside this group of 32: resume behind its last member
          r += (int)__fns(m, 0, RB - cnt) + 1;
          cnt = RB;
          break;
        }
        cnt += tot; r += 32;
      }
      if (lane == 0) { sCount = cnt; sNext = min(r, p.numROIs); }
    }
    __syncthreads();
    int const nb = sCount;
    base = sNext;
    if (nb == 0) break;
    bin_tables(binRow, binCol, roiIdx, nb, rois, p);
    vlb::stage_planes(plane, x + (size_t)HW * ((size_t)c0 + (size_t)p.C * img), HW, nch);
    __syncthreads();
    int const total = nb * bins;
    // arg-max of every bin, all threads: CPU scan order, first strictly greater, none for an empty or all -inf / NaN bin
    for (int b = tid; b < total; b += kOrdThreads) {
      // quotients by way of a float reciprocal: exact for these small operands, a fraction of the cost of integer division
      int const j = (int)(((float)b + 0.5f) * invBins), t = b - j * bins;
      int const pw = (int)(((float)t + 0.5f) * invS0), ph = t - pw * p.S0;
      uint32_t const rs = binRow[j * p.S0 + ph], cs = binCol[j * p.S1 + pw];
      int const hs = (int)(rs & 0xFFFFu), he = (int)(rs >> 16), ws = (int)(cs & 0xFFFFu), we = (int)(cs >> 16);
      float4 best = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
      uint32_t wx = kNoBin, wy = kNoBin, wz = kNoBin, ww = kNoBin;
      for (int w = ws; w < we; ++w)
#pragma unroll 2
        for (int h = hs; h < he; ++h) {
          uint32_t const at = (uint32_t)(w * p.H + h);
          float4 const a = plane[at];
          if (a.x > best.x) { best.x = a.x; wx = at; }
          if (a.y > best.y) { best.y = a.y; wy = at; }
          if (a.z > best.z) { best.z = a.z; wz = at; }
          if (a.w > best.w) { best.w = a.w; ww = at; }
        }
      uint16_t* const o = am + b;
      size_t const perCh = (size_t)RB * bins;
      o[0] = (uint16_t)wx; o[perCh] = (uint16_t)wy; o[2 * perCh] = (uint16_t)wz; o[3 * perCh] = (uint16_t)ww;
    }
    __syncthreads();
    // the planes have served: their room holds a word per pixel and channel, in which the lanes of a step meet
    for (int i = tid; i < HW; i += kOrdThreads) plane[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    // One warp per channel walks the bins in order -- ROI, bin column, bin row: the order of the CPU loop -- 32 at a time.  Among lanes whose
    // bins routed to the same pixel the first adds up for all, in lane order, and the pixel is read and written once a step.
    int const cc = warp;
    if (cc < nch) {
      uint16_t const* const amc = am + (size_t)cc * RB * bins;
      float* const acc = dxs + (size_t)cc * HW;
      unsigned* const mask = reinterpret_cast<unsigned*>(plane) + (size_t)cc * HW;
      // eight steps' derivatives are fetched together, so that their latency passes once per eight steps
      for (int b0 = 0; b0 < total; b0 += 32 * 8) {
        uint32_t wh[8];
        float vv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          int const b = b0 + 32 * u + lane;
          wh[u] = b < total ? amc[b] : kNoBin;
          vv[u] = 0.f;
          if (wh[u] != kNoBin) {
            int const j = (int)(((float)b + 0.5f) * invBins);
            vv[u] = __ldg(dy + (size_t)(b - j * bins) + (size_t)bins * ((size_t)(c0 + cc) + (size_t)p.C * roiIdx[j]));
          }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          uint32_t const where = wh[u];
          // the lanes of this step with the same pixel, for the first of them; 0 for the others
          unsigned m = 0;
          if (where != kNoBin) atomicOr(mask + where, 1u << lane);
          __syncwarp();
          if (where != kNoBin) m = mask[where];
          if ((m & ((1u << lane) - 1u)) != 0) m = 0;
          __syncwarp();
          if (m) mask[where] = 0;
          int const rounds = __reduce_max_sync(0xffffffffu, __popc(m));
          if (rounds == 0) continue;
          bool const first = m != 0;
          float sum = first ? acc[where] : 0.f;
          for (int r = 0; r < rounds; ++r) {
            float const v = __shfl_sync(0xffffffffu, vv[u], m ? __ffs(m) - 1 : 0);
            if (m) sum = __fadd_rn(sum, v);
            m &= m - 1;
          }
          if (first) acc[where] = sum;
          __syncwarp();
        }
      }
    }
    if (base >= p.numROIs) break;
  }
  __syncthreads();
  // dX is written once: the sums, or zeros where no bin routed (and for an image that no ROI names)
  for (int i = tid; i < nch * HW; i += kOrdThreads) dx[(size_t)HW * ((size_t)c0 + (size_t)p.C * img) + i] = dxs[i];
}

int make_params(vlb_ctx* ctx, RoiParams* p, int H, int W, int C, int N, int numROIs, int S0, int S1,
                double const* tf, int method)
{
  VLB_REQUIRE(ctx, H > 0 && W > 0 && C > 0 && N > 0, "roipool: empty input");
  VLB_REQUIRE(ctx, numROIs >= 0, "roipool: negative ROI count");
  VLB_REQUIRE(ctx, S0 >= 1 && S1 >= 1, "roipool: SUBDIVISIONS has a dimension smaller than 1");
  VLB_REQUIRE(ctx, tf != nullptr, "roipool: null transform");
  VLB_REQUIRE(ctx, method == VLB_POOL_MAX || method == VLB_POOL_AVG, "roipool: unknown method");
  p->H = H; p->W = W; p->C = C; p->N = N; p->numROIs = numROIs; p->S0 = S0; p->S1 = S1;
  for (int i = 0; i < 6; ++i) p->tf[i] = tf[i];
  return VLB_Success;
}

}  // namespace

extern "C" {

int vlb_roipool_bounds(vlb_ctx* ctx, int* bounds, int* images, float const* rois, int H, int W, int N,
                       int numROIs, int S0, int S1, double const* transform)
{
  if (!ctx) return VLB_IllegalArgument;
  RoiParams p;
  int rc = make_params(ctx, &p, H, W, 1, N, numROIs, S0, S1, transform, VLB_POOL_MAX);
  if (rc) return rc;
  VLB_REQUIRE(ctx, bounds && rois, "roipool_bounds: null tensor");
  if (numROIs == 0) return VLB_Success;
  vlb::launch(ctx->stream, roipool_bounds_kernel, vlb::grid_for((size_t)S0 * S1 * numROIs, kThreads), kThreads, 0, bounds, images, rois, p);
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, "vlb_roipool_bounds");
}

int vlb_roipool_forward(vlb_ctx* ctx, float* Y, float const* X, float const* rois, int H, int W, int C, int N,
                        int numROIs, int S0, int S1, double const* transform, int method)
{
  if (!ctx) return VLB_IllegalArgument;
  RoiParams p;
  int rc = make_params(ctx, &p, H, W, C, N, numROIs, S0, S1, transform, method);
  if (rc) return rc;
  VLB_REQUIRE(ctx, Y && X && rois, "roipool_forward: null tensor");
  if (numROIs == 0) return VLB_Success;
  {
    // planes in shared memory, where they fit (with room for three blocks per SM, or at least one for large maps) and the quotients by way of a float
    // reciprocal are exact (fewer than 2^18 bins a block, 2^12 a ROI).  64 ROIs per block pay for the staging of the planes; fewer
    // where that leaves the chip short of blocks.
    int const quads = vlb::ceil_div(C, 4);
    int RB = 64;
    while (RB > 8 && (long long)N * quads * vlb::ceil_div(numROIs, RB) < 4LL * ctx->smCount) RB /= 2;
    long long const HW = (long long)H * W, blocks = (long long)N * quads * vlb::ceil_div(numROIs, RB);
    if (H < 65535 && W < 65535 && HW < (1 << 20) && S0 <= 4096 && S1 <= 4096 && S0 * S1 <= 4096 && fwd_smem(RB, HW, S0, S1) <= 220 * 1024 && blocks < (1LL << 31)) {
      static bool attrDone[64] = {};
      if (!(ctx->device < 64 && attrDone[ctx->device])) {
        cudaError_t ea = vlb::allow_max_dynamic_smem(roipool_fwd_planes_kernel<true>);
        if (ea == cudaSuccess) ea = vlb::allow_max_dynamic_smem(roipool_fwd_planes_kernel<false>);
        if (ea != cudaSuccess) { cudaGetLastError(); return vlb::set_error(ctx, VLB_Cuda, cudaGetErrorString(ea)); }
        if (ctx->device < 64) attrDone[ctx->device] = true;
      }
      size_t const smem = fwd_smem(RB, HW, S0, S1);
      int const parts = vlb::ceil_div(numROIs, RB);
      if (method == VLB_POOL_MAX) vlb::launch(ctx->stream, roipool_fwd_planes_kernel<true>, (unsigned)blocks, kFwdThreads, smem, Y, X, rois, p, RB, parts, quads);
      else                        vlb::launch(ctx->stream, roipool_fwd_planes_kernel<false>, (unsigned)blocks, kFwdThreads, smem, Y, X, rois, p, RB, parts, quads);
      VLB_LAUNCHED(ctx, 1);
      return vlb::check_launch(ctx, "vlb_roipool_forward");
    }
  }
  size_t total = (size_t)S0 * S1 * C * numROIs;
  unsigned grid = vlb::grid_for(total, kThreads, ctx->smCount * 16);
  if (method == VLB_POOL_MAX) vlb::launch(ctx->stream, roipool_kernel<true, false>, grid, kThreads, 0, Y, X, rois, nullptr, p);
  else                        vlb::launch(ctx->stream, roipool_kernel<false, false>, grid, kThreads, 0, Y, X, rois, nullptr, p);
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, "vlb_roipool_forward");
}

int vlb_roipool_backward(vlb_ctx* ctx, float* dX, float const* X, float const* rois, float const* dY, int H, int W,
                         int C, int N, int numROIs, int S0, int S1, double const* transform, int method)
{
  if (!ctx) return VLB_IllegalArgument;
  RoiParams p;
  int rc = make_params(ctx, &p, H, W, C, N, numROIs, S0, S1, transform, method);
  if (rc) return rc;
  VLB_REQUIRE(ctx, dX && X && rois && dY, "roipool_backward: null tensor");
  {
    // the gather: slabs of about 64 KB per CTA, at least as many CTAs as SMs where the channels allow, and as many ROIs
    // per batch as the rest of the shared memory holds
    bool const isMax = method == VLB_POOL_MAX;
    long long const HW = (long long)H * W;
    size_t const budget = 200 * 1024;
    if (isMax && HW < 65535 && S0 <= 255 && S1 <= 255 && numROIs > 0) {
      // as many ROIs per batch as shared memory holds: two blocks per SM where that leaves room for 64 or for all, else one
      int const quads = vlb::ceil_div(C, 4);
      size_t const fixed = ordered_smem(0, (int)HW, S0, S1), perRoi = ordered_smem(1, (int)HW, S0, S1) - fixed;
      auto fit = [&](size_t budget) { return fixed < budget ? std::min<long long>((long long)((budget - fixed) / perRoi), numROIs) : 0LL; };
      long long RB = fit(112 * 1024);
      if (RB < 64 && RB < numROIs) RB = fit(224 * 1024);
      if ((RB >= 8 || RB == numROIs) && (long long)S0 * S1 <= 4096) {
        size_t const smem = ordered_smem((int)RB, (int)HW, S0, S1);
        static bool attrDone[64] = {};
        if (!(ctx->device < 64 && attrDone[ctx->device])) {
          cudaError_t ea = vlb::allow_max_dynamic_smem(roipool_bwd_ordered_kernel);
          if (ea != cudaSuccess) { cudaGetLastError(); return vlb::set_error(ctx, VLB_Cuda, cudaGetErrorString(ea)); }
          if (ctx->device < 64) attrDone[ctx->device] = true;
        }
        vlb::launch(ctx->stream, roipool_bwd_ordered_kernel, (unsigned)(N * quads), kOrdThreads, smem, dX, X, rois, dY, p, (int)RB, quads);
        VLB_LAUNCHED(ctx, 1);
        return vlb::check_launch(ctx, "vlb_roipool_backward");
      }
    }
    if (HW < 65535 && S0 <= 255 && S1 <= 255 && numROIs > 0) {
      int CH = (int)((64 * 1024) / (4 * HW));
      if (CH > C) CH = C;
      while (CH > 1 && (long long)N * vlb::ceil_div(C, CH) < ctx->smCount) --CH;
      if (CH >= 1) {
        size_t const fixed = gather_smem(CH, 0, H, W, S0, S1, isMax);
        size_t const perRoi = gather_smem(CH, 1, H, W, S0, S1, isMax) - fixed + 32;
        long long RB = fixed < budget ? (long long)((budget - fixed) / perRoi) : 0;
        if (RB > numROIs) RB = numROIs;
        if (RB >= 8 || RB == numROIs) {
          int const chunks = vlb::ceil_div(C, CH);
          size_t const smem = gather_smem(CH, (int)RB, H, W, S0, S1, isMax) + 64;
          static bool attrDone[2][64] = {};
          if (!(ctx->device < 64 && attrDone[isMax][ctx->device])) {
            cudaError_t ea = isMax ? vlb::allow_max_dynamic_smem(roipool_bwd_gather_kernel<true>)
                                   : vlb::allow_max_dynamic_smem(roipool_bwd_gather_kernel<false>);
            if (ea != cudaSuccess) { cudaGetLastError(); return vlb::set_error(ctx, VLB_Cuda, cudaGetErrorString(ea)); }
            if (ctx->device < 64) attrDone[isMax][ctx->device] = true;
          }
          unsigned const grid = (unsigned)(N * chunks);
          if (isMax) vlb::launch(ctx->stream, roipool_bwd_gather_kernel<true>, grid, kGatherThreads, smem, dX, X, rois, dY, p, CH, (int)RB, chunks);
          else       vlb::launch(ctx->stream, roipool_bwd_gather_kernel<false>, grid, kGatherThreads, smem, dX, X, rois, dY, p, CH, (int)RB, chunks);
          VLB_LAUNCHED(ctx, 1);
          return vlb::check_launch(ctx, "vlb_roipool_backward");
        }
      }
    }
  }
  // maps too large for a shared-memory slab: zero fill and scatter with atomics
  cudaError_t e = cudaMemsetAsync(dX, 0, sizeof(float) * (size_t)H * W * C * N, ctx->stream);
  if (e != cudaSuccess) return vlb::set_error(ctx, VLB_Cuda, cudaGetErrorString(e));
  if (numROIs == 0) return VLB_Success;
  size_t total = (size_t)S0 * S1 * C * numROIs;
  unsigned grid = vlb::grid_for(total, kThreads, ctx->smCount * 16);
  if (method == VLB_POOL_MAX) vlb::launch(ctx->stream, roipool_kernel<true, true>, grid, kThreads, 0, dX, X, rois, dY, p);
  else                        vlb::launch(ctx->stream, roipool_kernel<false, true>, grid, kThreads, 0, dX, X, rois, dY, p);
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, "vlb_roipool_backward");
}

}  // extern "C"
