// What the tensor-core contractions have in common (conv_tc.cu, conv_half.cu): parameters of a contraction, PTX wrappers for tensor memory, mbarriers
// and bulk copies, the places of a tile's rows and columns in the output, the cut of a reduction into ranges.  Every translation unit has its own copy.
#pragma once
#include "conv_internal.cuh"
#include <cuda.h>
#include <stdlib.h>
#include <string.h>
#include <algorithm>
#include <type_traits>

namespace {

using vlb::ConvGeom;
using vlb::ProfScope;
using vlb::kProfFprop; using vlb::kProfDgrad; using vlb::kProfWgrad; using vlb::kProfFc;

constexpr int BM = 128;          // output rows per CTA (TMEM lanes)
constexpr long long kWaitCycles = 200000000LL;    // default bound on any single barrier wait (about 0.1 s)
__constant__ long long gWaitCycles = kWaitCycles; // the bound in force on this device (vlb_ctx_set_wait_limit)

struct Operand {
  float const* ptr;
  long long ld, bs;
  int P;               // run length of contiguous reduction indices (DENSE_K, batched); 0 = unbatched
  int rows;            // valid extent of the row (M or N) index
  int vec;             // 1 when 16-byte loads are legal for this operand
  int fast;            // gather by tap tables: 1 aligned windows, 2 element-wise (any geometry), 0 filter too large for the tables (IM2COL, WGATHER)
  // convolution geometry (IM2COL, WGATHER)
  int H, W, C, FH, FW, Ho, Wo, sy, sx, pt, pl, dy, dx;
  long long imgStride;   // H*W*Ctotal
};

struct Epilogue {
  float* out;
  float const* bias;
  long long ldd;
  long long splitStride;
  float inMult, outMult;
  int P, Ktot;
  int relu;            // apply max(., 0) to the stored value (forward convolution followed by a ReLU layer)
  float const* mask;   // conv_ts_kernel, when non-null: laid out like out; the stored value is zeroed where mask is not positive
};

struct Params {
  Operand a, b;
  Epilogue e;
  int M, N, R;
  int BN;                 // tile columns: 16, 32, 64 or 128
  int numKb, kbPerSplit;
  int stages;
  int drainEvery;         // 3xTF32: k-blocks per tensor-core accumulation chain
  int tilesM, tilesN;     // conv_ts_kernel: the grid of output tiles its persistent CTAs walk
  int chanFast;           // conv_ts_kernel: reduction in blocks of 32 channels, r = c%32 + 32*(tap + taps*(c/32)); needs C % 32 == 0
  float const* bTiles;    // when non-null: B pre-split into shared-memory tile images, fetched with bulk copies
  int* status;
  int testSwitch;         // vlb_ctx_set_test_switch: bit 0 = conv_ts_kernel's filter-tile loader stays idle
  // conv_ts_kernel fed by tensor-map copies (tma != 0): an output tile is a box of bh x bw pixels of one image (tilesH x
  // tilesW boxes per image); its input window -- boxH rows (rowOff spare rows in front, so that the copy starts on a
  // 16-byte boundary) x boxW columns x 32 channels -- arrives in shared memory by one cp.async.bulk.tensor per channel block
  int tma, bh, bw, tilesH, tilesW, boxH, boxW, rowOff;
  int bStages;            // conv_ts_kernel: filter-tile stages in shared memory (4, or 3 where the input windows need the room)
  // conv_ts_kernel computing a filter gradient (wg != 0): D[(tap, c)][k] = sum over output pixels of x(pixel + tap, c) * dY(pixel, k).
  // A tile row is one channel of one filter tap: tapsPerTile taps x cPer channels = 128 rows, tapGroups x C/cPer row tiles; the
  // reduction (output pixels of the whole batch, kbTot k-blocks in the dY tile images) is cut into `splits` ranges of kbPerSplit
  // k-blocks, one work item per (range, row tile, column tile); the x runs arrive by tensor-map copies, xStages buffers.
  int wg, cPer, tapsPerTile, tapGroups, kbTot, splits, xStages;
  // conv_half_kernel, kMode 3: the gathered tensor split and laid out by split_chunks_kernel.  aHi[(image * C/8 + channel/8) * HW + pixel] are eight
  // channels of a pixel, the lo parts aLo further on; aExp[(image * C/64 + channel/64) * HW + pixel]; zero: sixteen zero bytes
  uint4 const* aHi;
  uint4 const* zero;
  int8_t const* aExp;
  long long aLo;
  int c64;                // blocks of 64 channels per image
  int const* bExp;        // conv_half_kernel: scale exponents of the tile images, [column tile][k-block]
  int8_t const* bOwn;     // and what single columns were scaled beyond them, [column tile][k-block][column]
  int chainShift;         // conv_ts_gen_kernel: 1 << chainShift own k-blocks per accumulation chain
  int fine;               // conv_ts_kernel, 128-column tiles: chains half as long, small terms first (kFine)
  int smemSum;            // conv_ts_kernel, kMode 0 / 1: keep the running sum of a tile in shared memory even for the tile widths that fit the
                          // drain warps' registers (one short tile per CTA, whose stores all warps share; test switch bit 3)
  int biasFirst;          // conv_ts_kernel: a tile's running sum starts at the bias (16-byte loads of it legal, no multiplier, columns in order)
  vlb::FastDiv31 dHo, dWo, dTilesN, dTilesM, dTaps;      // conv_ts_kernel: by a.Ho, a.Wo, tilesN, tilesM, a.FH * a.FW (set by ts_divisors)
  int plane;              // row mode: reduction indices per image in the tile images -- the plane's pixels rounded up to whole k-blocks
  // conv_ts_gen_kernel (general gather).  The reduction runs over units of `unit` channels of one filter tap, upk = 32 / unit of
  // them per k-block: unit number = tap + taps * (channel / unit).  Column tile nt belongs to filter group nt / tilesPerGroup;
  // a group has `cols` columns and reads a.C channels, aGroup elements further on.  Row (i, j) of an image is the output pixel
  // (oy + oys * i, ox + oxs * j) of a plane of outH x outW.  shufY > 0: column n of a group is channel n / (shufY * shufX) at the
  // output pixel moved by (n % shufY, n / shufY % shufX), outC channels per group.  ctaBeg, ctas: the CTAs that walk this problem.
  int unit, upk, tilesPerGroup, cols;
  // conv_half_kernel, kMode 4 and 5 (wg == 2): the filter gradient with the images along the reduction.  A k-block is 1 << gShift groups of eight images at
  // 8 >> gShift consecutive output rows of one column: k-block ((group of groups * Wo + column) * rowBlocks + row block).  aHi[((n/8 * W + w) * H + h) *
  // channels + channel] are eight images of a pixel (gShift < 3: four, and the other four aLo further on, fp32); aExp[(group of 64 images * W*H + pixel) *
  // channels + channel].
  int gShift, rowBlocks, nGroups, channels;
  int groups;             // tc_gemm_kernel, filter gradient: filter groups (0 counts as one), M rows and N columns each
  long long aGroup;
  int oy, ox, oys, oxs, outH, outW, shufY, shufX, outC, ctaBeg, ctas;
};

// Several contractions in one launch of conv_ts_gen_kernel (the residue classes of a strided data gradient), each with CTAs of its own.
// Launches pass the smallest block of parameters that holds the problems (with_capacity): one of 16 is 9.7 KB, which a launch of one
// problem then carries for nothing and reads its own through an index.  Always 16 / the smallest block: transposed convolution 35 x 47, stride 2 68.3 / 64.4 us,
// AlexNet step of 128 images 4480 / 4356, forward and gradients of 64 -> 40 channels in 4 groups, 1x1, stride 3 43.0 / 42.0 (a process in which the
// unchanged code took 42.0 and 43.0).
constexpr int kMaxTsProblems = 16;
template <int kMax> struct Problems { int n; Params p[kMax]; };
using TsProblems = Problems<kMaxTsProblems>;

// f(std::integral_constant<int, kMax>) for the smallest capacity that holds n: one (forward, stride 1, shuffled columns), the four classes of stride 2, 16.
template <class F>
inline void with_capacity(int n, F const& f)
{
  if (n <= 1) f(std::integral_constant<int, 1>{});
  else if (n <= 4) f(std::integral_constant<int, 4>{});
  else f(std::integral_constant<int, kMaxTsProblems>{});
}

template <int kMax>
inline Problems<kMax> first_problems(TsProblems const& b)
{
  Problems<kMax> q;
  q.n = b.n;
  std::copy(b.p, b.p + kMax, q.p);
  return q;
}

// ------------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(void const* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{ asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{ asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}" ::"r"(bar) : "memory"); }

// Bounded wait: false when the phase did not complete within gWaitCycles + extra.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, long long extra = 0)
{
  long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    // the thread is suspended by the hardware until the phase completes or the time hint (ns) runs out
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"(100000u) : "memory");
    if (ok) return true;
    if ((it & 15u) == 15u) {
      long long now = clock64();
      if (t0 == 0) t0 = now;
      else if (now - t0 > gWaitCycles + extra) return false;
    }
  }
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{ asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory"); }

// Bulk asynchronous copy global -> shared (both 16-byte aligned, size a multiple of 16); completion is
// signalled on the mbarrier as transaction bytes.  Source is always this GPU's own memory.
__device__ __forceinline__ void bulk_copy_g2s(uint32_t dstSmem, void const* src, uint32_t bytes, uint32_t bar)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dstSmem), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t dstSmem, uint32_t cols)
{
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dstSmem), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols)
{ asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory"); }

__device__ __forceinline__ void umma_tf32(uint32_t dTmem, uint64_t aDesc, uint64_t bDesc, uint32_t iDesc, uint32_t accumulate)
{
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}"
               ::"r"(dTmem), "l"(aDesc), "l"(bDesc), "r"(iDesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar)
{ asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory"); }

__device__ __forceinline__ void tmem_ld8_issue(uint32_t taddr, uint32_t* r)
{
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t* r)
{
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_st16(uint32_t taddr, uint32_t const (&r)[16])
{
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                 "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor (sm_100 format): start address, LBO, SBO in 16-byte
// units, version 1 at bit 46, layout type at bits 61-63: 2 = 128-byte swizzle (K-major tiles),
// 1 = 128-byte swizzle with 32-byte base (MN-major tiles of 32-bit elements).
__device__ __forceinline__ uint64_t make_desc(uint32_t addr, uint32_t lboBytes, uint32_t sboBytes, uint32_t layoutType = 2)
{
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lboBytes >> 4) << 16) | ((uint64_t)(sboBytes >> 4) << 32) |
         (1ull << 46) | ((uint64_t)layoutType << 61);
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes)
{ asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(bar), "r"(bytes) : "memory"); }

// 4-D tensor-map copy global -> shared (tile mode, one destination CTA; the map covers this GPU's own memory only); completion
// is signalled on the mbarrier as transaction bytes.  The innermost coordinate c0 must be a multiple of four elements.
__device__ __forceinline__ void tma_load_4d(uint32_t dstSmem, void const* map, int c0, int c1, int c2, int c3, uint32_t bar)
{
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
               ::"r"(dstSmem), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar) : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dstSmem, void const* map, int c0, int c1, int c2, uint32_t bar)
{
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               ::"r"(dstSmem), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}

__device__ __forceinline__ void lds128(uint32_t addr, float (&v)[4])
{
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(addr));
}

__device__ __forceinline__ float lds32(uint32_t addr)
{
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

// Bit f is set when position at + f * dilate lies inside [0, extent), f < taps (at most 32).
__device__ __forceinline__ uint32_t taps_inside(int at, int taps, int dilate, int extent)
{
  if (dilate == 1) {
    int const lo = max(-at, 0), hi = min(extent - at, taps);          // f in [lo, hi)
    return hi <= lo ? 0u : (0xffffffffu >> (32 - hi)) & (0xffffffffu << lo);
  }
  uint32_t m = 0;
  for (int f = 0; f < taps; ++f) if ((unsigned)(at + f * dilate) < (unsigned)extent) m |= 1u << f;
  return m;
}

// Where row `row` (0..127, = TMEM lane) of row tile `tm` lies in the output: image, pixel ho + Ho*wo, and whether it exists.
// Linear mode: the tile is 128 consecutive output pixels (ho fastest, images following one another).  Box mode (p.tma):
// the tile is a box of bh x bw pixels of one image, row = dh + bh*dw.
struct RowPos { int img, pix, split; bool valid; int h, w; };

template <bool kGen>
__device__ __forceinline__ RowPos row_pos(Params const& p, int tm, int row)
{
  RowPos r;
  r.h = r.w = 0;
  if (kGen) {
    r.split = p.dTilesM(tm); tm -= r.split * p.tilesM;
    int const m = tm * BM + row;
    r.valid = m < p.M;
    int const mm = min(m, p.M - 1), t = p.dHo(mm);
    r.img = p.dWo(t);
    r.h = p.oy + p.oys * (mm - t * p.a.Ho); r.w = p.ox + p.oxs * (t - r.img * p.a.Wo);
    r.pix = r.h + p.outH * r.w;
    return r;
  }
  if (p.wg == 2) {
    // tm = row tile + tilesM * reduction range; a row tile is four units of one filter group (tilesPerGroup tiles of it), a unit 32 channels of one filter tap
    int const split = p.dTilesM(tm), t = tm - split * p.tilesM, grp = t / p.tilesPerGroup;
    int const taps = p.a.FH * p.a.FW, u = (t - grp * p.tilesPerGroup) * 4 + (row >> 5), cb = p.dTaps(u), c = cb * 32 + (row & 31);
    r.valid = c < p.a.C;
    r.img = 0; r.pix = r.valid ? u - cb * taps + taps * c : 0; r.split = split;
    return r;
  }
  if (p.wg) {
    // tm = row tile + tilesM * reduction range; row tile = tap group + tapGroups * channel block; row = local tap * cPer + channel.
    // The "pixel" is the element of dF the row belongs to, fh + FH*(fw + FW*c), plus the offset of the range's partial result.
    int const split = tm / p.tilesM, t = tm - split * p.tilesM, cb = t / p.tapGroups, tg = t - cb * p.tapGroups;
    int const tl = row / p.cPer, c = cb * p.cPer + (row - tl * p.cPer), tap = tg * p.tapsPerTile + tl, taps = p.a.FH * p.a.FW;
    r.valid = tap < taps && c < p.a.C;
    r.img = 0; r.pix = r.valid ? tap + taps * c : 0; r.split = split;
    return r;
  }
  // tm = row tile + tilesM * reduction range (one range unless the caller cut the reduction)
  r.split = p.dTilesM(tm); tm -= r.split * p.tilesM;
  if (!p.tma) {
    int const m = tm * BM + row;
    r.valid = m < p.M;
    int const mm = min(m, p.M - 1);
    r.img = p.dWo(p.dHo(mm)); r.pix = mm - r.img * p.e.P;          // (a plane is a.Ho x a.Wo pixels)
  } else {
    int const per = p.tilesH * p.tilesW;
    int const n = tm / per, t = tm - n * per, wb = t / p.tilesH, hb = t - wb * p.tilesH;
    int const dw = row / p.bh, dh = row - dw * p.bh;
    int const h = hb * p.bh + dh, w = wb * p.bw + dw;
    r.valid = dw < p.bw && h < p.a.Ho && w < p.a.Wo;
    r.img = n; r.pix = r.valid ? h + p.a.Ho * w : 0;
  }
  return r;
}

// The columns of column tile nt: the first one among the output's columns, and how many of the tile's columns exist.
struct TileCols { int n0, cnt, grp; };

template <bool kGen>
__device__ __forceinline__ TileCols tile_cols(Params const& p, int nt)
{
  TileCols c;
  if (kGen) {
    c.grp = nt / p.tilesPerGroup;
    int const local = (nt - c.grp * p.tilesPerGroup) * p.BN;
    c.n0 = c.grp * p.cols + local; c.cnt = min(p.BN, p.cols - local);
  } else {
    c.grp = 0; c.n0 = nt * p.BN; c.cnt = min(p.BN, p.N - c.n0);
  }
  return c;
}

// Where the row of a tile that a thread stores goes.
struct TsDst { long long at; int row; bool valid; int h, w, img, split; };

template <bool kGen>
__device__ __forceinline__ TsDst ts_dst(Params const& p, int tm, int row)
{
  TsDst d;
  d.row = row;
  RowPos const rp = row_pos<kGen>(p, tm, row);
  d.valid = rp.valid; d.h = rp.h; d.w = rp.w; d.img = rp.img; d.split = rp.split;
  d.at = (long long)rp.split * p.e.splitStride + (long long)rp.img * p.e.Ktot * p.e.P + rp.pix;
  return d;
}

// Epilogue of conv_ts_kernel for what the direct store of the registers does not cover: the columns cBeg .. cBeg + cCnt - 1 of a tile from
// shared memory, P[column][row]: out[(image*Ktot + n)*P + pixel] = inMult*acc + bias[n] + outMult*old, then ReLU / mask.  Eight columns in flight.
// masked: the mask has been applied to P already.
template <bool kGen>
__device__ __forceinline__ void ts_store_cols(Params const& p, float const* P, TsDst const& d, TileCols const& tc, int cBeg, int cCnt, bool masked)
{
  int const nEnd = min(cCnt, tc.cnt - cBeg), n0 = tc.n0 + cBeg;
  if (!d.valid) return;
  float* const out = p.e.out + d.at;
  float const* const mask = masked ? nullptr : p.e.mask;
  P += d.row;
  if (kGen && p.shufY > 0) {
    // column n = moved by (ry, rx), channel c: the pixel is (h + ry, w + rx) where that lies inside the plane
    int const first = n0 - tc.grp * p.cols, per = p.shufY * p.shufX;
    int c = first / per, ry = (first - c * per) % p.shufY, rx = (first - c * per) / p.shufY;
    long long const plane = ((long long)d.img * p.e.Ktot + tc.grp * p.outC) * p.e.P;
    float* const base = p.e.out + (long long)d.split * p.e.splitStride;
#pragma unroll 4
    for (int k = 0; k < nEnd; ++k) {
      int const h = d.h + ry, w = d.w + rx;
      if ((unsigned)h < (unsigned)p.outH && (unsigned)w < (unsigned)p.outW) {
        long long const at = plane + (long long)c * p.e.P + (h + (long long)p.outH * w);
        float o = P[k * BM] + (p.e.bias ? p.e.bias[tc.grp * p.outC + c] : 0.f);
        if (mask && !(__ldg(mask + at) > 0.f)) o = 0.f;
        base[at] = o;
      }
      if (++ry == p.shufY) { ry = 0; if (++rx == p.shufX) { rx = 0; ++c; } }
    }
    return;
  }
  bool const hasBias = p.e.bias != nullptr && !p.biasFirst, hasOld = p.e.outMult != 0.f;
  float* o0 = out + (long long)n0 * p.e.P;
  for (int c0 = 0; c0 < nEnd; c0 += 8, o0 += 8LL * p.e.P) {
    float v[8], b[8], old[8], mk[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) { v[i] = P[min(c0 + i, nEnd - 1) * BM] * p.e.inMult; b[i] = 0.f; old[i] = 0.f; mk[i] = 1.f; }
    if (hasBias) {
#pragma unroll
      for (int i = 0; i < 8; ++i) b[i] = __ldg(p.e.bias + n0 + min(c0 + i, nEnd - 1));
    }
    if (hasOld) {
#pragma unroll
      for (int i = 0; i < 8; ++i) if (c0 + i < nEnd) old[i] = o0[(long long)i * p.e.P];
    }
    if (mask) {
#pragma unroll
      for (int i = 0; i < 8; ++i) if (c0 + i < nEnd) mk[i] = __ldg(mask + d.at + (long long)(n0 + c0 + i) * p.e.P);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float o = v[i];
      if (hasBias) o += b[i];
      if (hasOld) o += p.e.outMult * old[i];
      if (p.e.relu) o = o > 0.f ? o : 0.f;
      if (c0 + i < nEnd) o0[(long long)i * p.e.P] = mk[i] > 0.f ? o : 0.f;
    }
  }
}

constexpr int kMaxGenTaps = 128;                        // of the general gather (11 x 11 filters)

__device__ __forceinline__ void ldg32_if(float& x, float const* a, bool pred)
{
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %2, 0;\n @p ld.global.nc.f32 %0, [%1];\n}" : "+f"(x) : "l"(a), "r"((int)pred));
}

// ------------------------------------------------------------------ host side
inline int pick_bn(int N) { return N > 64 ? 128 : (N > 32 ? 64 : (N > 16 ? 32 : 16)); }

inline bool aligned16(void const* p) { return (((uintptr_t)p) & 15) == 0; }

// Registers per thread a kernel must have been compiled with (0: no requirement): those that redistribute registers between their warps (setmaxnreg) do
// so on the premise that every thread starts with exactly this many.
template <auto kKernel> constexpr int kRegsAtLaunch() { return 0; }

// The opt-in to more than 48 KB of dynamic shared memory, once per kernel and device instead of before every launch.
template <auto kKernel, int kRegs = kRegsAtLaunch<kKernel>()>
cudaError_t allow_large_smem(int device)
{
  static bool done[64] = {};
  if (device >= 0 && device < 64 && done[device]) return cudaSuccess;
  cudaError_t e = vlb::allow_max_dynamic_smem(kKernel);
  if (e == cudaSuccess && kRegs > 0) {
    // conv_ts_kernel redistributes registers between its warps (setmaxnreg) on the premise that every thread starts with
    // exactly this many; a build that gave it another count must not run (the hand-over would wait for registers for ever)
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, kKernel);
    if (e == cudaSuccess && attr.numRegs != kRegs) e = cudaErrorInvalidDeviceFunction;
  }
  if (e == cudaSuccess && device >= 0 && device < 64) done[device] = true;
  return e;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point query (the library does not link libcuda).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, cuuint64_t const*, cuuint64_t const*,
                                  cuuint32_t const*, cuuint32_t const*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled()
{
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)f;
    else
      cudaGetLastError();
  }
  return fn;
}

// The multiply-for-division constants of a launch, once its tiling is known: a thread's tile set-up (four divisions, a test per filter row and
// column) otherwise took the producers 2800 cycles per tile, in which the tensor core runs dry.
inline void ts_divisors(Params& p)
{
  p.dHo = vlb::FastDiv31(std::max(p.a.Ho, 1)); p.dWo = vlb::FastDiv31(std::max(p.a.Wo, 1));
  p.dTilesN = vlb::FastDiv31(p.tilesN); p.dTilesM = vlb::FastDiv31(p.tilesM); p.dTaps = vlb::FastDiv31(p.a.FH * p.a.FW);
}

// The cut of a filter gradient's reduction (numKb k-blocks, `tiles` output tiles) into ranges: the work items -- tiles x
// ranges -- should fill whole waves of the persistent CTAs, with ranges long enough that a tile's fixed cost stays small.
inline int pick_wg_splits(int smCount, int tiles, int numKb, int* kbPerSplit, int minKb)
{
  int best = 1; double bestEff = 0.0;
  for (int w = 1; w <= 6; ++w) {
    int s = std::max(1, (w * smCount) / tiles);
    s = std::min(s, std::max(1, numKb / minKb));
    int const per = vlb::ceil_div(numKb, s);
    s = vlb::ceil_div(numKb, per);
    long long const items = (long long)tiles * s;
    long long const perCta = (items + smCount - 1) / smCount;          // items of the busiest CTA
    // useful k-blocks per SM over the k-block slots the busiest CTA spends, a dozen k-blocks' worth of fixed cost per item
    double const eff = ((double)tiles * numKb / smCount) / ((double)perCta * (per + 12));
    if (eff > bestEff * 1.01) { bestEff = eff; best = s; }
  }
  *kbPerSplit = vlb::ceil_div(numKb, best);
  return vlb::ceil_div(numKb, *kbPerSplit);
}

// A forward or data-gradient contraction with fewer output tiles than SMs leaves most of the chip idle for the length of its whole reduction
// (one image through VGG-16's 28 x 28 layers: 28 tiles of 144 k-blocks): its reduction is cut into ranges as the filter gradients' are,
// and sum_parts adds them and applies the epilogue.  Returns the number of ranges; 1: left alone.  The lines, whole calls on 148 SMs:
//   tiles       8 of 144 k-blocks 90 -> 26 us, 100 93 -> 88, 124 and 148 level, 172 182 -> 147; of 36 k-blocks 172 53 -> 56.  Above the line
//               196 of 144 would gain (178 -> 150), of 36 lose (52 -> 55), 224 and more are level.
//   k-blocks    ranges of fewer than eight keep their sum in shared memory, and two of them cost more than one long reduction: 12 k-blocks in two
//               ranges 23.1 us, in one 14.1; 18 in three 19.2, in two 14.9, in one 15.3; 16 in two 18.0, in one 19.5.
inline int split_few_tiles(int smCount, int tiles, int numKb, int* kbPerSplit, int minKb)
{
  *kbPerSplit = numKb;
  if (tiles * 4 > smCount * 5 || numKb < 2 * minKb) return 1;
  return pick_wg_splits(smCount, tiles, numKb, kbPerSplit, minKb);
}

inline void conv_operand(Operand& o, ConvGeom const& g, float const* ptr, int channels)
{
  o.ptr = ptr;
  o.H = g.H; o.W = g.W; o.C = channels; o.FH = g.FH; o.FW = g.FW; o.Ho = g.Ho; o.Wo = g.Wo;
  o.sy = g.sy; o.sx = g.sx; o.pt = g.pt; o.pl = g.pl; o.dy = g.dy; o.dx = g.dx;
  o.imgStride = (long long)g.H * g.W * channels;
  o.ld = 0; o.bs = 0; o.P = 0; o.vec = 0;
  // 1: aligned windows (stride 1, extents multiples of 4); 2: element-wise gather, any geometry; 0: the filter does not fit the tap tables
  bool const lut = g.FH <= 32 && g.FW <= 32 && g.FH * g.FW <= 64;
  o.fast = !lut ? 0 : ((g.sy == 1 && g.sx == 1 && g.H % 4 == 0 && g.Ho % 4 == 0 && aligned16(ptr)) ? 1 : 2);
}

inline bool fits32(ConvGeom const& g)
{
  long long in = (long long)g.H * g.W * g.C * g.N, out = (long long)g.Ho * g.Wo * g.K * g.N;
  return in < (1LL << 31) - 256 && out < (1LL << 31) - 256 && (long long)g.FH * g.FW * g.FC * g.K < (1LL << 31);
}

// The geometry of a 1 x 1 convolution over a "plane" of `pixels` elements with `channels` channels (channel stride = pixels).
inline ConvGeom plane_geom(int pixels, int channels, int filters)
{
  ConvGeom t = {};
  t.H = pixels; t.W = 1; t.C = channels; t.N = 1; t.FH = 1; t.FW = 1; t.FC = channels; t.K = filters; t.Ho = pixels; t.Wo = 1;
  t.sy = 1; t.sx = 1; t.dy = 1; t.dx = 1; t.G = 1;
  return t;
}

// Channels per unit of the general gather: the least work, counting the gathered zeros (channels rounded up to units; kU = 3 leaves two of
// a k-block's 32 places empty) and the look-ups of small units (relative cost of a k-block, measured on 56 x 56 maps).
inline int gen_unit(int C)
{
  static int const unit[] = {32, 16, 8, 4, 3, 1};
  static double const cost[] = {1.0, 1.03, 1.1, 1.25, 1.35, 2.0};
  int best = 1; double bestCost = 1e30;
  for (int i = 0; i < 6; ++i) {
    double const c = cost[i] * (vlb::ceil_div(C, unit[i]) * unit[i]) * (32.0 / (32 / unit[i] * unit[i])) / C;
    if (c < bestCost) { bestCost = c; best = unit[i]; }
  }
  return best;
}

// Filter groups narrower than this (depthwise convolutions) leave a tensor-core tile nearly empty: CUDA cores.
constexpr int kMinGroupCols = 4;

inline bool gen_taps_ok(int FH, int FW) { return FH <= 32 && FW <= 32 && FH * FW <= kMaxGenTaps; }

// Time of a problem's k-blocks in units of a 128-column k-block, for comparing routes: narrower tiles save less than they drop columns.
inline double gen_cost(int tiles, int numKb, int BN)
{
  double const kb = BN == 128 ? 1.0 : (BN == 64 ? 0.62 : 0.5);
  return (double)tiles * (numKb + 6) * kb;
}

// Below kFineV positions the other kernel was the rule, whose chains hold large terms alone; conv_ts_kernel takes such a layer in its fine form,
// which is no further from the exact sums than that (256 images, forward / weights: 6.4e-7 there, 9.2e-7 in long chains, 3.9e-7 / 3.7e-7 in
// fine ones, which take 1 to 2% longer).
constexpr int kFineV = 128 * 64;

inline bool is_fc(ConvGeom const& g)
{
  return g.Ho == 1 && g.Wo == 1 && g.FH == g.H && g.FW == g.W && g.FC == g.C && g.sy == 1 && g.sx == 1 && g.pt == 0 &&
         g.pb == 0 && g.pl == 0 && g.pr == 0 && g.dy == 1 && g.dx == 1;
}

// The 3-D tensor map (run, rows, planes) of launch_rows; false when the driver refuses it.
inline bool rows_map(CUtensorMap* map, float const* ptr, long long run, long long rows, long long planes, int words, int cPer)
{
  EncodeTiledFn const encode = encode_tiled();
  if (!encode) return false;
  memset(map, 0, sizeof(*map));
  cuuint64_t const dims[3] = {(cuuint64_t)run, (cuuint64_t)rows, (cuuint64_t)planes};
  cuuint64_t const strides[2] = {(cuuint64_t)run * 4, (cuuint64_t)run * rows * 4};
  cuuint32_t const box[3] = {(cuuint32_t)words, (cuuint32_t)cPer, 1u};
  cuuint32_t const estr[3] = {1u, 1u, 1u};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One dimension of a data gradient's residue class: the input positions h with (h + pad) % stride == r, and the filter taps that reach
// them.  Positions are h0 + stride * i, i < count; tap f0 + step * (taps - 1 - f') of the filter meets position i at output
// position i + f' * dil - pad: a stride-1 convolution of the output derivative with `taps` taps.
struct ClassDim { int h0, count, taps, f0, step, dil, pad; };

inline ClassDim class_dim(int r, int H, int FH, int stride, int pad, int dilate)
{
  ClassDim c = {};
  c.h0 = ((r - pad) % stride + stride) % stride;
  c.count = c.h0 < H ? (H - 1 - c.h0) / stride + 1 : 0;
  int a = stride, d = dilate;
  while (d) { int const t = a % d; a = d; d = t; }                   // a = gcd(stride, dilate)
  c.step = stride / a; c.dil = dilate / a;
  c.f0 = -1;
  for (int f = 0; f < c.step && f < FH; ++f) if ((f * dilate) % stride == r) c.f0 = f;
  c.taps = c.f0 < 0 ? 0 : (FH - 1 - c.f0) / c.step + 1;
  // output position of tap f0 + step*j at position h: (h + pad - (f0 + step*j)*dilate) / stride = i + first - j*dil
  int const first = c.f0 < 0 ? 0 : (c.h0 + pad - c.f0 * dilate) / stride;          // exact: the numerator is a multiple of the stride
  c.pad = (c.taps - 1) * c.dil - first;
  return c;
}

// Whether the gathered tensor (chPerGroup channels in each of `groups` groups, read once per filter tap and column tile: `readings`) is split beforehand.  A k-block
// of the gather that splits as it goes takes 2000 cycles, one of split chunks 1150; a filter group has to be whole blocks of 64 channels, and a
// single one may be filled up with zeros to at most half as much again.  One reading costs more to split (8 bytes per element) than it saves:
// 1x1, 512 -> 128 channels, 28 x 28 x 64: 65 us against 60.
inline bool split_pays(int chPerGroup, int groups, int readings)
{
  return readings >= 2 && (groups == 1 ? (chPerGroup + 63) / 64 * 128 <= 3 * chPerGroup : chPerGroup % 64 == 0);
}

// Data gradient of a strided or grouped convolution, or one whose filters are no multiple of 32, through the general gather.  Two forms:
//   classes   one problem per residue class of the input pixel modulo the stride, each a stride-1 convolution of dY with the taps that
//             reach the class: no product with a structural zero, but C columns each;
//   shuffled  (dilation 1) one problem over the stride-sized blocks of input pixels whose columns are (pixel of the block, channel):
//             the classes' taps padded to the largest class, C * strideY * strideX columns -- for few channels, whose class
//             tiles would be mostly empty columns (11 x 11 stride 4 onto 3 channels: one 48-column problem instead of 16 with 3).
//
// Route is the kernel: kblocks(taps), problem(p, t, columns, BN), prep(p), launch(problems, tile images' description, scalar epilogue, covered).
template <class PrepBatch, class Route>
int dgrad_forms(vlb_ctx* ctx, vlb::ConvGeom const& g, float* dX, Route const& route)
{
  int const C = g.FC, nc = g.sy * g.sx;
  vlb::ConvGeom t = g;
  t.H = g.Ho; t.W = g.Wo; t.N = g.N; t.sy = t.sx = 1;
  ClassDim ch[kMaxTsProblems], cw[kMaxTsProblems];
  bool const classesOk = g.sy <= kMaxTsProblems && g.sx <= kMaxTsProblems && nc <= kMaxTsProblems;
  double classCost = 1e30;
  bool holes = false;               // classes that no tap reaches: zeros
  if (classesOk) {
    classCost = 0;
    for (int r = 0; r < g.sy; ++r) ch[r] = class_dim(r, g.H, g.FH, g.sy, g.pt, g.dy);
    for (int r = 0; r < g.sx; ++r) cw[r] = class_dim(r, g.W, g.FW, g.sx, g.pl, g.dx);
    int const BN = pick_bn(C);
    for (int y = 0; y < g.sy; ++y)
      for (int x = 0; x < g.sx; ++x) {
        int const taps = ch[y].taps * cw[x].taps, pix = ch[y].count * cw[x].count;
        if (pix == 0) continue;
        if (taps == 0) { holes = true; continue; }
        classCost += gen_cost(vlb::ceil_div((long long)pix * g.N, BM) * g.G * vlb::ceil_div(C, BN), route.kblocks(taps), BN);
      }
  }
  TsProblems ts = {};
  PrepBatch prep = {};
  vlb::SumEpilogue fin;
  fin.mask = ctx->reluMask;
  fin.bias = ctx->dgradBias; fin.P = g.H * g.W; fin.K = g.C;
  // shuffled form
  int const FHm = vlb::ceil_div(g.FH, g.sy), FWm = vlb::ceil_div(g.FW, g.sx);
  int const iy = g.pt / g.sy, ix = g.pl / g.sx, Hm = (g.H - 1 + g.pt) / g.sy - iy + 1, Wm = (g.W - 1 + g.pl) / g.sx - ix + 1;
  if (nc > 1 && g.dy == 1 && g.dx == 1 && gen_taps_ok(FHm, FWm)) {
    int const cols = C * nc, BN = pick_bn(cols);
    double const cost = gen_cost(vlb::ceil_div((long long)Hm * Wm * g.N, BM) * g.G * vlb::ceil_div(cols, BN), route.kblocks(FHm * FWm), BN);
    if (cost < classCost) {
      t.FH = FHm; t.FW = FWm; t.Ho = Hm; t.Wo = Wm; t.pt = FHm - 1 - iy; t.pl = FWm - 1 - ix;
      ts.n = 1;
      Params& p = ts.p[0];
      route.problem(p, t, cols, BN);
      p.oys = g.sy; p.oxs = g.sx; p.oy = g.sy * iy - g.pt; p.ox = g.sx * ix - g.pl; p.outH = g.H; p.outW = g.W;
      p.shufY = g.sy; p.shufX = g.sx; p.outC = C;
      p.e.inMult = 1.f; p.e.P = g.H * g.W; p.e.Ktot = g.C;
      auto& q = prep.p[0] = route.prep(p);
      q.bh = g.sy * (FHm - 1); q.ah = -g.sy; q.bw = g.sx * (FWm - 1); q.aw = -g.sx;
      q.sn = 1; q.sq = C; q.gs = (long long)C * g.Kg;
      int const rc = route.launch(ts, prep, fin, true);
      if (rc == VLB_Success) { ctx->maskDone = ctx->reluMask != nullptr; ctx->biasDone = true; }      // (a refused launch applies neither)
      return rc;
    }
  }
  if (!classesOk) return VLB_Unsupported;
  for (int y = 0; y < g.sy; ++y) for (int x = 0; x < g.sx; ++x) if (ch[y].taps * cw[x].taps > 0 && !gen_taps_ok(ch[y].taps, cw[x].taps)) return VLB_Unsupported;
  if (holes) {
    cudaError_t const e = cudaMemsetAsync(dX, 0, sizeof(float) * (size_t)g.H * g.W * g.C * g.N, ctx->stream);
    if (e != cudaSuccess) { cudaGetLastError(); return vlb::set_error(ctx, VLB_Cuda, cudaGetErrorString(e)); }
  }
  ts.n = 0;
  for (int y = 0; y < g.sy; ++y)
    for (int x = 0; x < g.sx; ++x) {
      ClassDim const& h = ch[y];
      ClassDim const& w = cw[x];
      if (h.taps * w.taps == 0 || h.count * w.count == 0) continue;
      t.FH = h.taps; t.FW = w.taps; t.Ho = h.count; t.Wo = w.count; t.pt = h.pad; t.pl = w.pad; t.dy = h.dil; t.dx = w.dil;
      Params& p = ts.p[ts.n];
      route.problem(p, t, C, pick_bn(C));
      p.oys = g.sy; p.oxs = g.sx; p.oy = h.h0; p.ox = w.h0; p.outH = g.H; p.outW = g.W;
      p.e.inMult = 1.f; p.e.P = g.H * g.W; p.e.Ktot = g.C;
      auto& q = prep.p[ts.n] = route.prep(p);
      q.bh = h.f0 + h.step * (h.taps - 1); q.ah = -h.step; q.bw = w.f0 + w.step * (w.taps - 1); q.aw = -w.step;
      q.sn = 1; q.sq = C; q.gs = (long long)C * g.Kg;
      ++ts.n;
    }
  if (holes) fin.bias = nullptr;                    // (the zeros of the classes without a tap would miss it)
  // (ts.n == 0: no tap reaches any pixel; all zeros, written above)
  int const rc = ts.n == 0 ? VLB_Success : route.launch(ts, prep, fin, !holes);
  if (rc == VLB_Success) { ctx->maskDone = ctx->reluMask != nullptr; ctx->biasDone = !holes; }
  return rc;
}

}  // namespace
