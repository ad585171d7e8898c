// Data gradients, filter gradients and convolution transposes on tcgen05 / TMEM with scaled half-precision operands
// (reference bits/nnconv.cu:120-317, bits/nnfullyconnected.cu:120-185, bits/nnconvt).
#include "tc_common.cuh"

namespace {

// D[m][n] = sum_r A(m,r) * B(n,r) as in conv_ts_kernel (conv_tc.cu), which keeps the forward passes: A goes to tensor memory, only the tiles of B to shared
// memory (bulk copies of ready-made tile images), fp32 accumulators in tensor memory.
//
// Arithmetic: scaled half-precision pairs.  The tensor core multiplies half-precision operands twice as fast as TF32 ones, and the two
// formats have the same 11 significant bits; what half precision lacks is range, and that is given back by scaling.  A k-block is 64
// reduction indices.  Each row of A takes the power of two that brings the largest magnitude of its values in the k-block into [2^14, 2^15), each tile of B one for
// 32 or 64 columns, and a column whose own largest magnitude is more than 2^16 below theirs one of its own; then x * s = hi + lo / 2048 with hi = half(x*s)
// and lo = half((x*s - hi) * 2048): 22 significant bits for every value of a row of A down to 2^-28 of the row's largest in the k-block, below that an absolute
// error of 2^-50 of that one; of a column of B down to 2^-12, 2^-34 at worst.  (Two TF32 values hold 22 bits as well, whatever stands beside them.)  Per k-block the accumulator T takes the small terms lo*hi + hi*lo first, which carry the 2048, then
// hi*hi with the accumulator scaled by 2^-11 (the MMA's scale-input-d); lo*lo (2^-22) is dropped.  Products of two halves are exact and the sums
// are fp32, as with TF32.  The drain warps add T * 2^-(row's + tile's exponent) to the fp32 running sum: one k-block per accumulation chain, so
// that the tensor core's truncating additions have no time to pile up (12 MMAs 16 deep; conv_ts_kernel has chains of up to 48 MMAs 8 deep).
// 3x3, 512 -> 512 channels, 28 x 28 x 64, against float64: 2.0e-7 (conv_ts_kernel 9e-7); data gradient 956 us there, 565 here.
// VLB_PRECISION_TF32 issues hi*hi alone: operands rounded to 11 bits as TF32 does, down to 2^-28 of the row's largest magnitude in the k-block (2^-12 of the
// column's), where the subnormal halves begin; below that an absolute error of 2^-39 (2^-23) of it.
// Why the forward passes stay where they are: their sums decide what ReLU and pooling let through.  Other sums, however near, decide some ties of
// existing networks the other way; a backward pass decides nothing.
//
// How A's rows get to tensor memory (kMode):
//   0  a thread per row gathers fp32 values, finds their largest, converts them (few channels, 1x1 filters): 2000 cycles per k-block
//   1  the same from input windows that tensor-map copies brought to shared memory
//   2  the same from runs along the planes (filter gradient; rows are (tap, channel))
//   3  sixteen 16-byte loads from a copy of the tensor that split_chunks_kernel has converted: 1150 cycles per k-block where the MMAs take 768.  No unit is saturated
//      (tensor pipe 73-77%, L2 24-30%, data banks of shared memory and L1 24-29%); by elimination it is the chain from a freed A stage over the loads to the next MMA
//   4  the same for filter gradients, chunks of eight images, a k-block being 64 images of a pixel
//   5  filter gradients of fewer images: a k-block is several rows of a column, wherever the filter tap puts them, so the chunks hold fp32 values, which a
//      thread converts as in the modes 0 to 2.  (Split beforehand they would need one power of two for all rows that some tap may put side by side, the
//      whole column: an infinity or a very large value in a row that a tap never reads would then cost that tap's sums their digits.)
// Warps: 0-7 drain and epilogue; 8, 9 MMA issue (one lane each; warp 8 also allocates TMEM), issuer q takes every other k-block; 10 loader of B's tiles; 11
// forwarder (when the tile of a k-block has landed it arrives on that k-block's A-stage barrier, so that an MMA thread waits on one barrier for both);
// 12-19 producers, two groups of four warps (one per TMEM lane quarter), group g fills the A stages of the k-blocks g, g + 2, ...
constexpr int kTsK = 64;                // reduction elements per k-block: one 128-byte swizzle row of halves
constexpr int kTsRowBytes = kTsK * 2;
constexpr int kTsGroups = 2;
constexpr int kTsDrainWarps = 8;        // two per lane quarter, each with half of the tile's columns
constexpr int kTsIssueWarp = kTsDrainWarps;
constexpr int kTsLoaderWarp = kTsDrainWarps + 2;
constexpr int kTsForwardWarp = kTsDrainWarps + 3;
constexpr int kTsFirstProducer = kTsDrainWarps + 4;
constexpr int kTsThreads = (kTsFirstProducer + 4 * kTsGroups) * 32;      // 640: five warpgroups, 96 registers per thread at launch
constexpr int kTsRunWarp = kTsFirstProducer + 4 * kTsGroups;             // row mode only: warp 20 issues the runs (tensor-map copies)
constexpr int kTsThreadsRows = (kTsRunWarp + 4) * 32;                    // 768: warp 20's warpgroup is launched whole (warps 21-23 idle), so that it can hand its registers over
constexpr int kTsBStages = 6;           // at most; Params::bStages are in use
constexpr int kTsStatic = 3072;         // upper bound of the kernel's static shared memory

// kind::f16 instruction descriptor: D = F32, A and B = F16 (0), both K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__device__ __forceinline__ uint32_t make_idesc_f16(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24); }

__device__ __forceinline__ void umma_f16_ts(uint32_t dTmem, uint32_t aTmem, uint64_t bDesc, uint32_t iDesc, uint32_t accumulate)
{
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
               ::"r"(dTmem), "r"(aTmem), "l"(bDesc), "r"(iDesc), "r"(accumulate) : "memory");
}
// D = A*B + D * 2^-11
__device__ __forceinline__ void umma_f16_ts_scaled(uint32_t dTmem, uint32_t aTmem, uint64_t bDesc, uint32_t iDesc)
{
  asm volatile("{\n .reg .pred p;\n setp.eq.b32 p, %3, %3;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, 11;\n}"
               ::"r"(dTmem), "r"(aTmem), "l"(bDesc), "r"(iDesc) : "memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, uint32_t const* r)
{
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// 32 columns from eight quads
__device__ __forceinline__ void tmem_st32(uint32_t taddr, uint4 const (&r)[8])
{
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
               "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
               ::"r"(taddr), "r"(r[0].x), "r"(r[0].y), "r"(r[0].z), "r"(r[0].w), "r"(r[1].x), "r"(r[1].y), "r"(r[1].z), "r"(r[1].w),
                 "r"(r[2].x), "r"(r[2].y), "r"(r[2].z), "r"(r[2].w), "r"(r[3].x), "r"(r[3].y), "r"(r[3].z), "r"(r[3].w),
                 "r"(r[4].x), "r"(r[4].y), "r"(r[4].z), "r"(r[4].w), "r"(r[5].x), "r"(r[5].y), "r"(r[5].z), "r"(r[5].w),
                 "r"(r[6].x), "r"(r[6].y), "r"(r[6].z), "r"(r[6].w), "r"(r[7].x), "r"(r[7].y), "r"(r[7].z), "r"(r[7].w) : "memory");
}

// A column of B whose largest magnitude lies more than 2^kOwnScale below the tile's takes a power of two of its own, 2^c beyond the tile's.  The closer the line
// lies to the tile's, the more k-blocks of ordinary values pay for it in the drain warps (rescale_columns; dense values never, a column with one value left by
// ReLU and pooling once in 25000 k-blocks, the cross terms of a normalisation layer in a fifth: AlexNet's filter gradients 522 -> 618 us); the further off, the fewer digits a column just above it keeps: at 2^16 its values have 22 bits (VLB_PRECISION_TF32:
// 11) down to 2^-12 of its largest.
constexpr int kOwnScale = 16;
constexpr int kMaxOwnScale = 100;       // (further down 22 bits until 2^-128 of the tile's largest magnitude)
constexpr int kOwnFlag = 1 << 16;       // added to an exponent word of the tile images: some column has one of its own

// Two fp32 values side by side in one 64-bit register pair, and the packed operations on them (one instruction for both).
__device__ __forceinline__ uint64_t pack2(float a, float b) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack2(uint64_t r, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ float max3(float a, float b, float c) { float r; asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }

// The scale exponent k of values whose largest magnitude is m: m * 2^k lies in [2^14, 2^15).  At most 116, so that 2^(k + 11) is a number
// (values below 2^-102 then stay smaller than they could be); -114 for infinity, whose row (or column) comes out as not-a-number in any case.
__device__ __forceinline__ int scale_exp(float m) { return min(141 - (int)(__float_as_uint(m) >> 23), 116); }
__device__ __forceinline__ float exp2i(int k) { return __uint_as_float((uint32_t)(127 + k) << 23); }      // -126 <= k <= 127

// A pair of values times s as half(x*s) and half((x*s - hi) * 2048); s2 = {s, s}, sl2 = {2048 s, 2048 s}.
template <bool kSplit>
__device__ __forceinline__ void split_pair(float a, float b, uint64_t s2, uint64_t sl2, uint32_t& hi, uint32_t& lo)
{
  uint64_t const x = pack2(a, b), xs = mul2(x, s2);
  float x0, x1;
  unpack2(xs, x0, x1);
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(x1), "f"(x0));
  if (kSplit) {
    float h0, h1, l0, l1;
    asm("{\n .reg .f16 a, b;\n mov.b32 {a, b}, %2;\n cvt.f32.f16 %0, a;\n cvt.f32.f16 %1, b;\n}" : "=f"(h0), "=f"(h1) : "r"(hi));
    unpack2(fma2(pack2(h0, h1), pack2(-2048.f, -2048.f), mul2(x, sl2)), l0, l1);
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(l1), "f"(l0));
  }
}

// The columns beg .. end - 1 of an accumulator (multiples of eight) times 2^-own[column], in tensor memory, so that the drain's own loop stays as it is.
// (5x5, 96 -> 256 channels in two groups, 27 x 27 x 128, such columns in a fifth of the k-blocks: 212 -> 260 us; with the factors in the drain's loop, whose unrolled code then
// has to be fetched for them, 220 -> 311; with one load for all exponents instead of one per eight columns 261.)
__device__ __forceinline__ void rescale_columns(uint32_t acc, int8_t const* own, int beg, int end)
{
#pragma unroll 1
  for (int c0 = beg; c0 < end; c0 += 8) {
    uint32_t r[8];
    tmem_ld8_issue(acc + (uint32_t)c0, r);
    uint2 const e = __ldg(reinterpret_cast<uint2 const*>(own + c0));
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * exp2i(-(int)(((j < 4 ? e.x : e.y) >> (8 * (j & 3))) & 255u)));
    tmem_st8(acc + (uint32_t)c0, r);
  }
  tmem_st_wait();
}

// kTma: the producers take the input windows from shared memory, where the loader thread has them delivered by tensor-map copies
// (one box of boxH x boxW pixels x 32 channels per channel block and tile, zero-filled outside the image by the copy
// engine, two buffers), instead of gathering them from global memory with per-thread loads.  xmap: the 4-D tensor map
// (H, W, C, N) of the gathered tensor; unused otherwise.
// kMode 2 (filter gradient): rows are (tap, channel), the reduction runs over the output pixels; the loader thread has the run of 64
// pixels (plus up to three in front, so that the copy starts on a 16-byte boundary) of every row delivered per k-block.
constexpr int kWgRowWords = kTsK + 4;                   // words per row of an x run in shared memory (272 bytes: 16-byte loads of 8 rows hit 32 banks)
constexpr int kWgRowBytes = kWgRowWords * 4;
constexpr int kWgStageBytes = BM * kWgRowBytes;         // 34816
constexpr int kTsXStages = 6;                           // at most
// "The MMAs of k-block j (numbered over the CTA's life) are through" is reported on barrier j % kTsDoneRing, phase j / kTsDoneRing,
// by the issuer's one commit per k-block.  Three parties wait for it: the producers of the A stage (for k-block j + kNA), the
// filter-tile loader (for k-block j + bStages) -- the filter stage is free at the same moment -- and the drain warps, whose accumulator
// is complete.  The ring is longer than any of them can fall behind (at most bStages - 1 <= 5 k-blocks can complete before the loader has
// looked, at most kNA - 1 before a producer has, at most kNT before the drain warps have), so a waiter never meets a barrier that is already a phase
// further.  (Waiting on the barriers of the kNA A stages instead
// was tried first: with six filter stages and four A stages the loader fell a whole phase behind on conv1_2 at batch 64 and then
// waited for a completion that needed its own copies -- the bounded wait ran out.)
constexpr int kTsDoneRing = 8;
static_assert(kTsBStages < kTsDoneRing, "the loader must not be able to fall a whole ring behind");

// Registers: 96 per thread at launch (640 threads, one CTA per SM); then the four issuing / loading warps keep 40, which leaves 128 x 56 for the others: the
// drain warps take 112 and the producers 104, or 120 and the 96 they have where the producers only carry chunks (kMode 3, 4) -- 256 x 24 either way, so
// the hand-over stays inside the registers the block was launched with and never waits.  (64 of the drain warps' hold half a row of the tile's running sum.)
// kMode 2 runs with another warp for its per-k-block tensor-map copies -- such a copy keeps the issuing warp busy for about
// a microsecond, so it cannot share a warp with the forwarding, the filter tiles or a producer (measured: 35-50% slower each way).
// Registers are handed over by whole warpgroups, so the kernel is launched with six of them (768 threads, 80 registers each; three warps have nothing
// to do): eight warps keep 40, the producers take 96, and the drain warps 104 here too (256 x 40 = 256 x 24 + 256 x 16).
// kNarrow: tiles of 64 columns or fewer (kMode 0, 1), which get more accumulators and A stages (below).
// kGen: the general gather (below) instead of the one that needs whole blocks of 32 channels.  cta, ctas: this CTA's place among
// those that walk the problem's tiles.
// A k-block is two sub-blocks of 32: sub-block s of a convolution is filter tap s % taps of the channel block s / taps, of the general gather the
// units upk * s .. upk * (s + 1) - 1.
template <bool kSplit, int kMode, bool kNarrow, bool kGen>
__device__ __forceinline__ void conv_half_body(Params const& p, CUtensorMap const* xmap, int const cta, int const ctas)
{
  constexpr bool kTma = kMode == 1, kWg = kMode == 2, kImages = kMode == 4 || kMode == 5;      // (0: per-thread gather, 3: gather of a tensor that was split beforehand)
  constexpr bool kChunks = kMode == 3 || kMode == 4;      // the producers only carry
  extern __shared__ uint8_t smemRaw[];
  __shared__ __align__(8) uint64_t fullA[4], doneK[kTsDoneRing], fullB[kTsBStages];
  __shared__ __align__(8) uint64_t tFree[4], turn[2], fullX[kTsXStages], emptyX[kTsXStages];
  __shared__ uint32_t tmemBase;
  __shared__ int2 tapLut[kGen ? kMaxGenTaps : 64];       // per filter tap fh + FH*fw: {element offset of the tap (in the input window when kTma), fh | fw << 5}
  // scale exponents of the A rows of k-block j at j % kTsDoneRing.  (The slot's previous k-block, eight before, has been drained: its accumulator
  // was handed to a k-block whose MMAs the producer has waited for.)
  __shared__ int8_t rowExp[kTsDoneRing][BM];

  uint8_t* smem = smemRaw + ((1024u - (smem_u32(smemRaw) & 1023u)) & 1023u);
  int const BN = p.BN;
  int const nB = p.bStages;
  uint32_t const bTileBytes = (uint32_t)BN * kTsRowBytes;
  uint32_t const bBytes = (kSplit ? 2u : 1u) * bTileBytes;
  uint32_t const tmemCols = 512;
  // Tensor memory: kNT accumulators of BN columns (k-block j in T[j % kNT]), then kNA A stages of 64 columns (32 hi, 32 lo).
  // 128-column tiles: three accumulators (two being accumulated while the third is drained and, at the end of a tile,
  // stored) and one A stage per issuer -- 512 columns.  Tiles of 64 columns or fewer have room for four accumulators and two
  // A stages per issuer: a stage is refilled while the MMAs of the issuer's other stage run, which is what these tiles, whose
  // MMAs are short, gain most from.
  constexpr int kNA = kNarrow ? 4 : 2, kAPer = kNA / 2, kAShift = kNA == 4 ? 1 : 0;      // kAPer = 1 << kAShift
  constexpr int kNT = kNarrow ? 4 : 3;
  uint32_t const colA = (uint32_t)(kNT * BN);
  float* const Psm = reinterpret_cast<float*>(smem + (size_t)nB * bBytes);      // patch of 32 columns for the stores that do not go straight from registers, [column][BM]
  // input windows (kTma) or runs (kWg) behind the patch
  uint32_t const xPlane = (uint32_t)(p.boxH * p.boxW), xTileBytes = kWg ? (uint32_t)kWgStageBytes : xPlane * 32u * 4u;
  uint32_t const xTile0 = smem_u32(Psm) + (uint32_t)min(BN, 32) * BM * 4u;

  int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int const numIter = p.kbPerSplit;                      // k-blocks per tile (work item: one range of the reduction of one output tile)
  int const numTiles = p.tilesM * p.tilesN * p.splits;
  // this CTA's tiles: cta, cta + ctas, ...; tile t = (row tile t / tilesN, column tile t % tilesN)
  int const myTiles = cta < numTiles ? (numTiles - 1 - cta) / ctas + 1 : 0;

  if (threadIdx.x == 0) {
    // an A stage is full when its four producer warps and the forwarder (filter tile landed) have arrived
    for (int s = 0; s < 4; ++s) mbar_init(smem_u32(&fullA[s]), 5);
    for (int s = 0; s < kTsDoneRing; ++s) mbar_init(smem_u32(&doneK[s]), 1);
    for (int s = 0; s < kTsBStages; ++s) mbar_init(smem_u32(&fullB[s]), 1);
    for (int b = 0; b < 4; ++b) mbar_init(smem_u32(&tFree[b]), kTsDrainWarps);
    mbar_init(smem_u32(&turn[0]), 1); mbar_init(smem_u32(&turn[1]), 1);
    // an input window is full when its copy has landed (one arrival with the byte count), empty when all eight producer warps are done with it
    // (filter gradient: a run belongs to one k-block, so only the four warps of the group that owns it let go of it)
    for (int b = 0; b < kTsXStages; ++b) { mbar_init(smem_u32(&fullX[b]), 1); mbar_init(smem_u32(&emptyX[b]), kWg ? 4 : 4 * kTsGroups); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kTsIssueWarp) tmem_alloc(smem_u32(&tmemBase), tmemCols);
  if (!kImages && (int)threadIdx.x < p.a.FH * p.a.FW) {
    int const fh = (int)threadIdx.x % p.a.FH, fw = (int)threadIdx.x / p.a.FH;
    if (kWg)       tapLut[threadIdx.x] = make_int2((fw * p.a.dx - p.a.pl) * p.a.H + fh * p.a.dy - p.a.pt, fh * p.a.dy - p.a.pt);   // {shift of the tap in the flattened plane, its row offset}
    else if (kTma) tapLut[threadIdx.x] = make_int2(fw * p.a.dx * p.boxH + fh * p.a.dy, fh | (fw << 5));
    else           tapLut[threadIdx.x] = make_int2((fw * p.a.dx - p.a.pl) * p.a.H + fh * p.a.dy - p.a.pt, fh | (fw << 5));
  }
  tc_fence_before();
  vlb::pdl_wait();        // (everything above touches this CTA's own shared and tensor memory only)
  __syncthreads();
  tc_fence_after();
  uint32_t const tmemAcc = tmemBase;

  if (warp < kTsDrainWarps) {
    // ============================== fp32 drain and epilogue ==============================
    // Every k-block's accumulator is added to the tile's running sum, times the k-block's power of two, and released at once.  The running
    // sum lives in registers (one TMEM lane = one output row per thread; a thread has half of the row's columns).  With four warps, each with whole
    // rows, the drain was what bounded the kernel: 1080 cycles per k-block, a quarter of them for the stores, where the MMAs take 768.
    if (kWg) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;" ::: "memory");
    else if (kChunks) asm volatile("setmaxnreg.inc.sync.aligned.u32 120;" ::: "memory");
    else     asm volatile("setmaxnreg.inc.sync.aligned.u32 112;" ::: "memory");
    uint32_t const lanes = tmemAcc + ((uint32_t)((warp & 3) * 32) << 16);
    int const row = (warp & 3) * 32 + lane, half = warp >> 2;
    auto drain = [&](auto kColsTag) {
      constexpr int kCols = decltype(kColsTag)::value;          // columns of this thread: half of the tile's
      constexpr int kStep = kWg ? (kCols < 16 ? kCols : 16) : (kCols < 32 ? kCols : 32);      // columns of the accumulator on the way at a time
      constexpr int kPatch = kCols < 16 ? kCols : 16;           // columns of its patch of shared memory
      int const col0 = half * kCols;
      float* const Pp = Psm + half * kPatch * BM;               // the patch, [column][BM]
      float* const Prow = Pp + row;
      uint64_t P2[kCols / 2];                                   // the running sum, two columns to a register pair
      bool const preMask = p.e.mask != nullptr && !(kGen && p.shufY > 0);
      uint32_t g = 0;                                   // k-blocks over the CTA's life
      int t = 0;                                        // g % kNT
      bool ok = true;
      for (int ts = 0; ts < myTiles && ok; ++ts) {
        int const tile = cta + ts * ctas;
        int const tm = p.dTilesN(tile);
        int nt = tile - tm * p.tilesN;                  // column tile
        TileCols tc = tile_cols<kGen>(p, nt);
        if (kImages) {
          int const grp = (tm - p.dTilesM(tm) * p.tilesM) / p.tilesPerGroup, local = nt * BN;
          tc.n0 = grp * p.cols + local; tc.cnt = min(BN, p.cols - local);
          nt += grp * p.tilesN;
        }
        int const n0 = tc.n0 + col0;
        // exponents of the tile images: one per 64 columns (this thread's, of a wide tile), per 32 where the images are along the reduction
        constexpr int kPer = kImages ? 32 : 64, kExps = kCols > kPer ? 2 : 1;
        int const perImage = max(BN / kPer, 1);
        size_t const image0 = (size_t)nt * p.kbTot + (size_t)p.dTilesM(tm) * numIter;
        int const* const bExp = p.bExp + image0 * perImage + col0 / kPer;
        int eB[kExps];
#pragma unroll
        for (int j = 0; j < kExps; ++j) eB[j] = __ldg(bExp + j);
#pragma unroll
        for (int j = 0; j < kCols; j += 4) {
          // (the bias is there long before the first k-block is)
          float4 const b = p.biasFirst && col0 + j < tc.cnt ? __ldg(reinterpret_cast<float4 const*>(p.e.bias + n0 + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
          P2[j / 2] = pack2(b.x, b.y); P2[j / 2 + 1] = pack2(b.z, b.w);
        }
        // ReLU mask of this thread's output row: sixteen columns are fetched before each of the tile's
        // first waits, so that their latency passes while the k-block is being computed, and kept as one bit each
        uint32_t mbits[2] = {0u, 0u};
        int const nEndT = min(kCols, tc.cnt - col0);    // columns of this thread that exist (may be none)
        float const* mkRow = p.e.mask;
        if (preMask) {
          RowPos const rp = row_pos<kGen>(p, tm, row);     // a row that does not exist reads (and discards) the mask of a pixel that does
          mkRow += ((long long)rp.img * p.e.Ktot + n0) * p.e.P + rp.pix;      // (a masked data gradient is never cut into ranges)
        }
        int lc = 0;                                     // batches of sixteen mask columns fetched so far
        for (int it = 0; it < numIter; ++it, ++g) {
          float mk[16];
          bool const fetch = preMask && 16 * lc < nEndT;
          if (fetch) {
#pragma unroll
            for (int j = 0; j < 16; ++j) mk[j] = __ldg(mkRow + (long long)min(16 * lc + j, nEndT - 1) * p.e.P);
          }
          ok = mbar_wait(smem_u32(&doneK[g & (kTsDoneRing - 1)]), (g / kTsDoneRing) & 1u);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) { if (lane == 0) atomicExch(p.status, 5); break; }
          if (fetch) {
            uint32_t b = 0;
#pragma unroll
            for (int j = 0; j < 16; ++j) b |= (mk[j] > 0.f ? 1u : 0u) << j;
            b <<= 16 * (lc & 1);
            if (lc < 2) mbits[0] |= b; else mbits[1] |= b;
            ++lc;
          }
          tc_fence_after();
          int const eA = (int)rowExp[g & (kTsDoneRing - 1)][row];
          int ex[kExps];
          bool odd = false;
#pragma unroll
          for (int j = 0; j < kExps; ++j) {
            ex[j] = -(eA + eB[j]);
            odd = odd || ex[j] < -126 || ex[j] > 127;
            if (it + 1 < numIter) eB[j] = __ldg(bExp + (it + 1) * perImage + j);
          }
          // a power of two outside the normal range (products of values around 1e-20 or 1e+20) is applied in two halves; kOwnFlag shows up here too, so that
          // the loop has one test for both
          bool far = __any_sync(0xffffffffu, odd);
          if (__builtin_expect(far, 0)) {
            int beg = kCols, end = 0;
#pragma unroll
            for (int j = 0; j < kExps; ++j)
              if (ex[j] < -kOwnFlag / 2) { ex[j] += kOwnFlag; beg = min(beg, j * kPer); end = min((j + 1) * kPer, kCols); }
            rescale_columns(lanes + (uint32_t)(t * 2 * kCols + col0), p.bOwn + (image0 + it) * BN + col0, beg, end);
          }
#pragma unroll
          for (int c0 = 0; c0 < kCols; c0 += kStep) {
            uint32_t t0[kStep < 16 ? 8 : kStep];
            uint32_t const at = lanes + (uint32_t)(t * 2 * kCols + col0 + c0);
            if constexpr (kStep == 8) tmem_ld8_issue(at, t0); else tmem_ld16_issue(at, t0);
            if constexpr (kStep == 32) tmem_ld16_issue(at + 16u, t0 + 16);
            int const e = ex[kExps == 2 ? c0 / 32 : 0], e1 = far ? e / 2 : 0;
            float const f = exp2i(e - e1), f1 = exp2i(e1);
            uint64_t const f2 = pack2(f, f);
            tmem_ld_wait();
            if (far) {
#pragma unroll
              for (int j = 0; j < kStep; ++j) t0[j] = __float_as_uint(__uint_as_float(t0[j]) * f1);
            }
#pragma unroll
            for (int j = 0; j < kStep; j += 2) {
              uint64_t& q = P2[(c0 + j) / 2];
              q = fma2(pack2(__uint_as_float(t0[j]), __uint_as_float(t0[j + 1])), f2, q);
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&tFree[t]));     // T[t] may be overwritten
          if (++t == kNT) t = 0;
        }
        if (!ok) break;
        for (; preMask && 16 * lc < nEndT; ++lc) {        // a tile of fewer k-blocks than batches: the rest of the mask
          uint32_t b = 0;
#pragma unroll
          for (int j = 0; j < 16; ++j) b |= (__ldg(mkRow + (long long)min(16 * lc + j, nEndT - 1) * p.e.P) > 0.f ? 1u : 0u) << j;
          b <<= 16 * (lc & 1);
          if (lc < 2) mbits[0] |= b; else mbits[1] |= b;
        }
        TsDst const dst = ts_dst<kGen>(p, tm, row);
        // The finished tile while the tensor core works on the next one.  Straight from the registers, a 4-byte store per column and
        // thread, coalesced along the rows: nothing here waits for anything.  (Every load of this phase -- a patch of shared memory, a
        // bias -- cost the drain warps its full latency plus a queue behind the producers' gathers: 4.4k cycles per 128-column tile through
        // 16-byte stores from a patch, 13k to 20k where planes of 13 x 13 or 27 x 27 pixels rule those out.)
        bool const direct = (p.e.bias == nullptr || p.biasFirst) && (p.e.mask == nullptr || preMask) && !(kGen && p.shufY > 0);
        if (preMask) {
#pragma unroll
          for (int j = 0; j < kCols; j += 2) {
            float a, b;
            unpack2(P2[j / 2], a, b);
            P2[j / 2] = pack2(((mbits[j / 32] >> (j & 31)) & 1u) ? a : 0.f, ((mbits[j / 32] >> ((j & 31) + 1)) & 1u) ? b : 0.f);
          }
        }
        if (direct) {
          float* o = p.e.out + dst.at + (long long)n0 * p.e.P;
#pragma unroll
          for (int j = 0; j < kCols; j += 2) {
            float a, b;
            unpack2(P2[j / 2], a, b);
            if (dst.valid && j < nEndT) *o = a;
            o += p.e.P;
            if (dst.valid && j + 1 < nEndT) *o = b;
            o += p.e.P;
          }
        } else {
          // sixteen columns at a time: registers -> patch[column][row] (shared memory, every thread its own row) -> global memory
          // (the loop over the columns has to run over shared memory: registers cannot be indexed)
#pragma unroll
          for (int c0 = 0; c0 < kCols; c0 += kPatch) {
            if (c0 < nEndT) {
#pragma unroll
              for (int j = 0; j < kPatch; j += 2) unpack2(P2[(c0 + j) / 2], Prow[j * BM], Prow[(j + 1) * BM]);
              ts_store_cols<kGen>(p, Pp, dst, tc, col0 + c0, kPatch, preMask);
            }
          }
        }
      }
    };
    // (each variant is compiled with the drain loops it can need only: the kernel's code has to stay small -- the variants for
    // 64-column tiles lost 10-30% whenever a few instructions were added to their roles)
    if constexpr (kNarrow) {
      if (BN == 64) drain(std::integral_constant<int, 32>{});
      else if (BN == 32) drain(std::integral_constant<int, 16>{});
      else drain(std::integral_constant<int, 8>{});
    } else if constexpr (kWg) {
      if (BN == 128) drain(std::integral_constant<int, 64>{});
      else if (BN == 64) drain(std::integral_constant<int, 32>{});
      else if (BN == 32) drain(std::integral_constant<int, 16>{});
      else drain(std::integral_constant<int, 8>{});
    } else {
      drain(std::integral_constant<int, 64>{});
    }
  } else if (warp < kTsFirstProducer) {
    // The issuers, the filter-tile loader and the forwarder work with one thread each and a handful of registers: the rest goes
    // to the others.  All four warps of the group execute this before anything else.
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;" ::: "memory");
    long long const total = (long long)myTiles * numIter;      // k-blocks of this CTA
    if (warp == kTsIssueWarp || warp == kTsIssueWarp + 1) {
    // ============================== MMA issue ==============================
    // Two issuing threads (in two warps, on two schedulers).  The tensor core's queue is about one MMA deep, so
    // while a thread waits on a barrier or commits, nothing of its own is in flight; with two threads the other
    // one's MMAs fill the gap.  Issuer q takes the k-blocks gi = q, q+2, ... (numbered over the CTA's life), which
    // live in A stage q (+ 2).  The k-blocks take the T buffers in turn, in the order the
    // drain warps will add them, so two are being accumulated while the third is drained; the two
    // issuers never touch the same tensor-memory columns, so no ordering between the two streams is needed.
    // Per k-block: a wait for the T buffer, a wait for the A stage (A written and B landed), twelve MMAs, one commit.
    if (lane == 0) {
      int const q = warp - kTsIssueWarp;
      uint32_t const idesc = make_idesc_f16(BN);
      uint64_t const descB0 = make_desc(smem_u32(smem), 16, 1024);
      uint32_t const stageStep = bBytes >> 4, loStep = bTileBytes >> 4;
      int sb = q, t = q;                             // filter stage, T buffer
      uint32_t tWraps = 0;                           // gi / kNT
      uint32_t own = 0;                              // this issuer's k-blocks so far: k-block `own` sits in A stage q + 2*(own % kAPer)
      uint32_t phTurn = q == 0 ? 1u : 0u;            // issuer 0 has the first turn (nothing to wait for)
      // measured: +5-13% on 128-column tiles, -5% on 64-column tiles (their MMAs are short and the extra wait shows), -1-5% in the
      // row mode (whose producers read shared memory and are never late)
      bool const takeTurns = !kNarrow && !kWg;
      for (long long gi = q; gi < total; gi += 2) {
        uint32_t const tAcc = tmemAcc + (uint32_t)(t * BN);
        // the k-block that sat in this T before must have been added to the running sum
        if (tWraps > 0 && !mbar_wait(smem_u32(&tFree[t]), (tWraps - 1) & 1u)) { atomicExch(p.status, 6); break; }
        int const sa = q + 2 * (int)(own & (uint32_t)(kAPer - 1));
        uint32_t const aHi = tmemAcc + colA + (uint32_t)(sa * 64), aLo = aHi + 32u;
        if (!mbar_wait(smem_u32(&fullA[sa]), (own >> kAShift) & 1u)) { atomicExch(p.status, 2); break; }

        // The issuers take turns: left to themselves they interleave their MMAs one by one, both k-blocks finish
        // together, both A stages are refilled together and the tensor core idles meanwhile.  In turns, the MMAs of
        // one k-block run while the other issuer's A stage (freed a whole k-block earlier) is being refilled.
        if (takeTurns) {
          if (!mbar_wait(smem_u32(&turn[q]), phTurn)) { atomicExch(p.status, 10); break; }
          phTurn ^= 1u;
        }
        tc_fence_after();
        uint64_t const dBh = descB0 + (uint64_t)((uint32_t)sb * stageStep), dBl = dBh + loStep;
        // The turn goes to the other issuer before the last MMAs of this k-block are queued: it needs about 200 cycles
        // (three MMAs) to wake up from its wait, and its MMAs, which use another A stage and another accumulator, may
        // queue up behind or between the remaining ones in any order.
        if (kSplit) {
#pragma unroll
          for (int k = 0; k < kTsK / 16; ++k) {
            umma_f16_ts(tAcc, aLo + 8u * k, dBh + 2u * k, idesc, k > 0 ? 1u : 0u);      // 0 = overwrite
            umma_f16_ts(tAcc, aHi + 8u * k, dBl + 2u * k, idesc, 1u);
          }
          umma_f16_ts_scaled(tAcc, aHi, dBh, idesc);
          if (takeTurns) mbar_arrive(smem_u32(&turn[q ^ 1]));
#pragma unroll
          for (int k = 1; k < kTsK / 16; ++k) umma_f16_ts(tAcc, aHi + 8u * k, dBh + 2u * k, idesc, 1u);
        } else {
#pragma unroll
          for (int k = 0; k < kTsK / 16; ++k) {
            umma_f16_ts(tAcc, aHi + 8u * k, dBh + 2u * k, idesc, k > 0 ? 1u : 0u);
            if (takeTurns && k == kTsK / 16 - 2) mbar_arrive(smem_u32(&turn[q ^ 1]));
          }
        }
        umma_commit(smem_u32(&doneK[(uint32_t)gi & (uint32_t)(kTsDoneRing - 1)]));
        ++own;
        sb += 2; if (sb >= nB) sb -= nB;
        t += 2; if (t >= kNT) { t -= kNT; ++tWraps; }
      }
    }
    __syncwarp();
    tc_fence_before();
  } else if (warp == kTsLoaderWarp) {
    // ============================== filter tiles: bulk copies ==============================
    if (lane == 0 && !(p.testSwitch & 1)) {
      int sb = 0;
      bool ok = true;
      long long gk = 0;                                  // k-blocks numbered over the CTA's life
      for (int ts = 0; ts < myTiles && ok; ++ts) {
        int const tile = cta + ts * ctas;
        int nt = tile % p.tilesN;
        if (kImages) nt += (tile / p.tilesN) % p.tilesM / p.tilesPerGroup * p.tilesN;
        uint8_t const* src = reinterpret_cast<uint8_t const*>(p.bTiles) + ((size_t)nt * p.kbTot + (size_t)(tile / p.tilesN / p.tilesM) * numIter) * bBytes;
        for (int it = 0; it < numIter; ++it, ++gk, src += bBytes) {
          // the stage held the filter tile of k-block gk - nB
          long long const j = gk - nB;
          if (j >= 0 && !mbar_wait(smem_u32(&doneK[j & (kTsDoneRing - 1)]), (uint32_t)((j / kTsDoneRing) & 1))) { atomicExch(p.status, 8); ok = false; break; }
          mbar_arrive_expect_tx(smem_u32(&fullB[sb]), bBytes);
          bulk_copy_g2s(smem_u32(smem + (size_t)sb * bBytes), src, bBytes, smem_u32(&fullB[sb]));
          if (++sb == nB) sb = 0;
        }
      }
    }
    __syncwarp();
  } else if (warp == kTsForwardWarp) {
    // ============================== forwarder; input windows: tensor-map copies ==============================
    // Forwarding: k-block gi (numbered over the CTA's life) uses A stage gi % kNA in that barrier's phase gi / kNA.  The arrival
    // for gi must fall into that phase, so the phase of gi - kNA has to be complete first (this thread arrived in it as well).
    // The windows of kTma (one per tile and block of 32 channels, xStages buffers) are numbered over the CTA's life and issued by
    // the same thread.
    if (lane == 0) {
      int const taps = p.a.FH * p.a.FW;
      int const perTile = kTma ? 2 * numIter / taps : 0;                     // windows per tile
      int const nXb = p.xStages;
      long long const wTotal = (long long)myTiles * perTile;
      long long wxs = 0;                                  // next window to issue
      int wts = 0, wsub = 0;                              // its tile (in this CTA's sequence) and its index inside the tile
      int ots = 0, osub = 0;                              // the same of the window nXb before it, once there is one
      int wbuf = 0; uint32_t wph = 1;                     // its buffer; first use of a buffer: nothing to wait for
      // Window w is issued when this thread has come to k-block wpos(w) (numbered over the CTA's life), after a wait for its buffer,
      // which the window v = w - nXb held: the group that gathers v's last sub-block, in k-block kl, lets go of it before that k-block's hand-over,
      // the other group before the hand-over of kl + 1.  At wpos = kl + 2 this thread has forwarded all that those two need, so the wait is
      // short and depends on nothing that this thread has yet to do.  The first nXb at once.
      auto windows = [&](long long gpos) -> bool {
        while (wxs < wTotal) {
          long long const wpos = wxs < nXb ? 0 : (long long)ots * numIter + ((osub + 1) * taps - 1) / 2 + 2;
          if (wpos > gpos) break;
          if (!mbar_wait(smem_u32(&emptyX[wbuf]), wph)) { atomicExch(p.status, 12); return false; }
          int const tmf = (cta + wts * ctas) / p.tilesN;
          int const split = tmf / p.tilesM, tm = tmf - split * p.tilesM;
          {
            int const per = p.tilesH * p.tilesW;
            int const n = tm / per, t = tm - n * per, wb = t / p.tilesH, hb = t - wb * p.tilesH;
            int const c0 = hb * p.bh - p.a.pt - p.rowOff, c1 = wb * p.bw - p.a.pl;      // c0 is a multiple of four: bh and pt + rowOff are
            mbar_arrive_expect_tx(smem_u32(&fullX[wbuf]), xTileBytes);
            tma_load_4d(xTile0 + (uint32_t)wbuf * xTileBytes, xmap, c0, c1, (split * perTile + wsub) * 32, n, smem_u32(&fullX[wbuf]));   // a range of the reduction is whole channel blocks
          }
          if (wxs >= nXb && ++osub == perTile) { osub = 0; ++ots; }
          ++wxs;
          if (++wbuf == nXb) { wbuf = 0; wph ^= 1u; }
          if (++wsub == perTile) { wsub = 0; ++wts; }
        }
        return true;
      };
      int sb = 0; uint32_t phB = 0;
      for (long long gi = 0; gi < total; ++gi) {
        int const sa = (int)(gi & (kNA - 1));
        if (gi >= kNA && !mbar_wait(smem_u32(&fullA[sa]), (uint32_t)(((gi >> (kAShift + 1)) - 1) & 1))) { atomicExch(p.status, 9); break; }
        if (kTma && !windows(gi)) break;
        if (!mbar_wait(smem_u32(&fullB[sb]), phB)) { atomicExch(p.status, 7); break; }
        mbar_arrive(smem_u32(&fullA[sa]));
        if (++sb == nB) { sb = 0; phB ^= 1u; }
      }
    }
    __syncwarp();
    }
  } else if (warp >= kTsRunWarp) {
    // ============================== row mode: runs by tensor-map copies ==============================
    // (this warpgroup exists in the row mode only and keeps a handful of registers, like the issuers')
    if (kWg) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;" ::: "memory");
    if (kWg && warp == kTsRunWarp && lane == 0) {
      // The run of k-block j (numbered over the CTA's life) -- 68 pixels x cPer channels per
      // tap of the tile, from the plane of image r / P starting at pixel r % P + shift of the tap, rounded down to four pixels (P:
      // the plane rounded up to whole k-blocks; the tile images hold zeros for the pixels added; pixels before the plane's first
      // or past its last one -- a tap that leaves the image to the left or right, a k-block past the end of the batch -- arrive as
      // zeros) -- goes into buffer j % xStages as soon as the producers have let go of the run of k-block j - xStages.
      int const taps = p.a.FH * p.a.FW, P = p.plane, nX = p.xStages;
      int buf = 0; uint32_t ph = 1;                        // first use of a buffer: nothing to wait for
      bool ok = true;
      for (int ts = 0; ts < myTiles && ok; ++ts) {
        int const tmf = (cta + ts * ctas) / p.tilesN;
        int const split = tmf / p.tilesM, t = tmf - split * p.tilesM, cb = t / p.tapGroups, tg = t - cb * p.tapGroups;
        int const tap0 = tg * p.tapsPerTile, nTaps = min(p.tapsPerTile, taps - tap0);
        long long const r0 = (long long)split * numIter * kTsK;
        int img = (int)(r0 / P), pix0 = (int)(r0 - (long long)img * P);
        for (int it = 0; it < numIter; ++it) {
          if (!mbar_wait(smem_u32(&emptyX[buf]), ph)) { atomicExch(p.status, 12); ok = false; break; }
          mbar_arrive_expect_tx(smem_u32(&fullX[buf]), (uint32_t)(nTaps * p.cPer * kWgRowBytes));
          for (int tl = 0; tl < nTaps; ++tl)
            tma_load_3d(xTile0 + (uint32_t)buf * xTileBytes + (uint32_t)(tl * p.cPer * kWgRowBytes), xmap,
                        pix0 + (tapLut[tap0 + tl].x & ~3), cb * p.cPer, img, smem_u32(&fullX[buf]));
          if (++buf == nX) { buf = 0; ph ^= 1u; }
          pix0 += kTsK; if (pix0 >= P) { pix0 -= P; ++img; }
        }
      }
    }
    __syncwarp();
  } else {
    // ============================== producers ==============================
    if (kWg) asm volatile("setmaxnreg.inc.sync.aligned.u32 96;" ::: "memory");
    else if (!kChunks) asm volatile("setmaxnreg.inc.sync.aligned.u32 104;" ::: "memory");      // (kMode 3, 4: the 96 of the launch)
    int const grp = (warp - kTsFirstProducer) >> 2;
    int const quarter = warp & 3;                       // the TMEM lanes this warp may access
    int const row = quarter * 32 + lane;
    int const HW = p.a.H * p.a.W, taps = p.a.FH * p.a.FW;
    uint32_t const aBase = tmemAcc + ((uint32_t)(quarter * 32) << 16) + colA;
    uint32_t own = 0;                                   // this group's k-blocks so far: k-block `own` goes into A stage grp + 2*(own % kAPer)
    long long gi = 0;                                   // k-blocks numbered over the CTA's life; this group takes gi % 2 == grp
    bool ok = true;

    // From the wait for the A stage to the arrival on its barrier; `store` writes this row's 32 columns of hi and of lo.
    auto stage_in = [&](auto store, int ke) -> bool {
      int const sa = grp + 2 * (int)(own & (uint32_t)(kAPer - 1));
      if (own >= (uint32_t)kAPer) {      // (first use of a stage: nothing to wait for) the stage's previous k-block, kNA before this one, must be through
        uint32_t const jp = 2u * (own - (uint32_t)kAPer) + (uint32_t)grp;
        if (!mbar_wait(smem_u32(&doneK[jp & (uint32_t)(kTsDoneRing - 1)]), (jp / (uint32_t)kTsDoneRing) & 1u)) { atomicExch(p.status, 1); return false; }
      }
      tc_fence_after();
      store(aBase + (uint32_t)(sa * 64));
      rowExp[(2u * own + (uint32_t)grp) & (uint32_t)(kTsDoneRing - 1)][row] = (int8_t)ke;
      ++own;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&fullA[sa]));
      return true;
    };

    // One k-block, from the 64 gathered values of this thread's row to the arrival on the A-stage barrier.
    auto hand_over = [&](float const* v) -> bool {
      // both parts are ready in registers before the wait, so that the stage is refilled as soon as it is free
      float m0 = 0.f, m1 = 0.f;                         // (fmax: a not-a-number counts as nothing and comes through the conversions as one)
#pragma unroll
      for (int k = 0; k < kTsK; k += 4) { m0 = max3(m0, fabsf(v[k]), fabsf(v[k + 1])); m1 = max3(m1, fabsf(v[k + 2]), fabsf(v[k + 3])); }
      float const m = fmaxf(m0, m1);
      int const ke = m > 0.f ? scale_exp(m) : 0;        // (a row of zeros keeps the powers of two in the normal range)
      float const s = exp2i(ke), sl = exp2i(ke + 11);
      uint64_t const s2 = pack2(s, s), sl2 = pack2(sl, sl);
      uint32_t hi[kTsK / 2], lo[kTsK / 2];
#pragma unroll
      for (int k = 0; k < kTsK / 2; ++k) split_pair<kSplit>(v[2 * k], v[2 * k + 1], s2, sl2, hi[k], lo[k]);
      return stage_in([&](uint32_t aAddr) {
        // (eight columns at a time: a wider store wants its registers in one piece, and hi and lo of a pair come out side by side)
#pragma unroll
        for (int k = 0; k < kTsK / 2; k += 8) {
          tmem_st8(aAddr + (uint32_t)k, hi + k);
          if (kSplit) tmem_st8(aAddr + 32u + (uint32_t)k, lo + k);
        }
      }, ke);
    };

    if (kWg) {
      // This thread's row: channel (row % cPer) of the tile's local tap row / cPer -- the same tap for the whole warp.  A k-block
      // is 64 consecutive output pixels; the row's 68-pixel run lies in shared memory, the wanted 64 start `s` pixels in.
      int const tl = (quarter * 32) / p.cPer;
      int const H = p.a.H, P = p.plane, real = p.a.Ho * p.a.Wo, nX = p.xStages;
      for (int ts = 0; ts < myTiles && ok; ++ts) {
        int const tmf = (cta + ts * ctas) / p.tilesN;
        int const split = tmf / p.tilesM, t = tmf - split * p.tilesM, tg = t % p.tapGroups;
        int const tap = tg * p.tapsPerTile + tl;
        bool const active = tap < taps;                                   // a tap the filter does not have: rows of zeros, never stored
        int2 const te = tapLut[active ? tap : 0];
        int const s = te.x & 3, dh = te.y;
        int const itFirst = (int)((gi ^ grp) & 1);
        int pb = (int)(((long long)split * numIter + itFirst) * kTsK % P);      // first pixel of the k-block inside its image
        for (int it = itFirst; it < numIter; it += kTsGroups) {
          uint32_t const xs = (uint32_t)(gi + it), use = xs / (uint32_t)nX;
          int const buf = (int)(xs - use * (uint32_t)nX);
          // With an odd number of buffers the buffer's previous run belongs to the other group, which may be behind: this run's phase can be told from
          // the one two before only once that run has been let go of.  (The run before it was this group's own.)
          if ((use > 0 && !mbar_wait(smem_u32(&emptyX[buf]), (use - 1u) & 1u)) ||
              !mbar_wait(smem_u32(&fullX[buf]), use & 1u)) { atomicExch(p.status, 11); ok = false; break; }
          uint32_t const src = xTile0 + (uint32_t)buf * xTileBytes + (uint32_t)(row * kWgRowBytes);
          float w[kWgRowWords];
#pragma unroll
          for (int j = 0; j < kWgRowWords / 4; ++j) lds128(src + 16u * j, *reinterpret_cast<float(*)[4]>(&w[4 * j]));
          // pixels whose tap row leaves the image above or below: output row ho + dh outside [0, H) -- the same for every lane's row -- and those that fill
          // the plane up to whole k-blocks, whose taps to the left still lie inside it (an infinity there times dY's zeros would be none)
          int const p0 = pb + lane, p1 = p0 + 32, ho0 = p0 % H, ho1 = p1 % H;
          pb += kTsGroups * kTsK; while (pb >= P) pb -= P;
          uint32_t const zm0 = active ? __ballot_sync(0xffffffffu, (unsigned)(ho0 + dh) >= (unsigned)H || p0 >= real) : 0xffffffffu;
          uint32_t const zm1 = active ? __ballot_sync(0xffffffffu, (unsigned)(ho1 + dh) >= (unsigned)H || p1 >= real) : 0xffffffffu;
          // the wanted 64, by two rounds of selects (s is uniform; a copy of the code per shift runs at the speed of instruction fetches)
          if (s != 0) {
            bool const s1 = (s & 1) != 0, s2 = (s & 2) != 0;
#pragma unroll
            for (int k = 0; k < kTsK + 2; ++k) w[k] = s1 ? w[k + 1] : w[k];
#pragma unroll
            for (int k = 0; k < kTsK; ++k) w[k] = s2 ? w[k + 2] : w[k];
          }
          if (zm0 | zm1) {
#pragma unroll
            for (int k = 0; k < kTsK; ++k) w[k] = (((k < 32 ? zm0 : zm1) >> (k & 31)) & 1u) ? 0.f : w[k];
          }
          ok = hand_over(w);
          if (!ok) break;
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&emptyX[buf]));     // this warp's loads from the run have completed (their values were used above)
        }
        gi += numIter;
      }
    } else if (kTma) {
      // This thread's pixel inside the input window: row dh + rowOff, column dw (a lane beyond the box reads the window's
      // first element; its row is never stored).  A sub-block is one filter tap and 32 channels: 32 loads from shared memory
      // one channel plane apart.
      int const dw = row / p.bh, dh = row - dw * p.bh;
      uint32_t const laneOff = dw < p.bw ? (uint32_t)(dw * p.boxH + dh + p.rowOff) * 4u : 0u;
      uint32_t const planeBytes = xPlane * 4u;
      int const perTile = 2 * numIter / taps, nX = p.xStages;
      // The window in hand, numbered over the CTA's life.  Every producer warp waits for and lets go of every window, whether or not one of its
      // k-blocks falls into it: a warp can then never arrive twice in one phase of the window's barrier.
      long long xs = -1, xsTile = 0;
      int buf = -1; uint32_t ph = 0;
      auto advance = [&](long long to) -> bool {
        while (xs < to) {
          __syncwarp();
          if (xs >= 0 && lane == 0) mbar_arrive(smem_u32(&emptyX[buf]));     // this warp's loads from the window have completed
          ++xs;
          if (++buf == nX) { buf = 0; ph ^= 1u; }
          if (!mbar_wait(smem_u32(&fullX[buf]), ph)) { atomicExch(p.status, 11); return false; }
        }
        return true;
      };
      for (int ts = 0; ts < myTiles && ok; ++ts, xsTile += perTile) {
        for (int it = (int)((gi ^ grp) & 1); it < numIter; it += kTsGroups) {
          float v[kTsK];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            int const sub = 2 * it + h, cb = p.dTaps(sub), tap = sub - cb * taps;
            if (cb < perTile) {
              if (!advance(xsTile + cb)) { ok = false; break; }
              uint32_t const src = xTile0 + (uint32_t)buf * xTileBytes + laneOff + (uint32_t)tapLut[tap].x * 4u;
#pragma unroll
              for (int k = 0; k < 32; ++k) v[32 * h + k] = lds32(src + (uint32_t)k * planeBytes);
            } else {
#pragma unroll
              for (int k = 0; k < 32; ++k) v[32 * h + k] = 0.f;
            }
          }
          if (!ok || !hand_over(v)) { ok = false; break; }
        }
        gi += numIter;
      }
    } else if (kImages) {
      // This warp's unit: 32 channels (a lane each) of one filter tap.  A k-block is eight chunks of eight images, 16 bytes for hi and 16 for lo (kMode 5:
      // for the first four and for the other four): one pixel (kMode 4), or 8 >> gShift output rows of a column.  Lanes are neighbours in memory, and which
      // pixels exist is the same for all of them.
      int const gShift = kMode == 4 ? 3 : p.gShift, g = 1 << gShift, rows = 8 >> gShift, W = p.a.W, H = p.a.H;
      for (int ts = 0; ts < myTiles && ok; ++ts) {
        int const tmf = p.dTilesN(cta + ts * ctas), split = p.dTilesM(tmf), t = tmf - split * p.tilesM, fg = t / p.tilesPerGroup;
        int const u = (t - fg * p.tilesPerGroup) * 4 + quarter, cb = p.dTaps(u), tap = u - cb * taps, c = cb * 32 + lane;
        bool const active = c < p.a.C;
        int const fw = tap / p.a.FH, fh = tap - fw * p.a.FH, dw = fw * p.a.dx - p.a.pl, dh = fh * p.a.dy - p.a.pt;
        uint4 const* const xq = p.aHi + (fg * p.a.C + c);
        int8_t const* const eq = p.aExp + (fg * p.a.C + c);
        for (int it = (int)((gi ^ grp) & 1); it < numIter; it += kTsGroups) {
          int const kb = split * numIter + it, col = p.dHo(kb), rb = kb - col * p.rowBlocks, n = p.dWo(col);      // (dHo, dWo: by rowBlocks and Wo)
          int const wx = (col - n * p.a.Wo) * p.a.sx + dw, h0 = rb * rows;
          bool const colOn = active && (unsigned)wx < (unsigned)W && n < p.nGroups;
          auto chunk = [&](int j, bool& on) -> uint4 const* {
            int const ho = h0 + (j >> gShift), hx = ho * p.a.sy + dh;
            on = colOn && ho < p.a.Ho && (unsigned)hx < (unsigned)H;
            return on ? xq + (((long long)(n * g + (j & (g - 1))) * W + wx) * H + hx) * p.channels : p.zero;
          };
          if constexpr (kMode == 4) {
            uint4 h[8], l[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              bool on;
              uint4 const* const q = chunk(j, on);
              h[j] = __ldg(q);
              if (kSplit) l[j] = __ldg(on ? q + p.aLo : p.zero);
            }
            int const hx = h0 * p.a.sy + dh;
            int const ke = colOn && (unsigned)hx < (unsigned)H ? __ldg(eq + (((long long)n * W + wx) * H + hx) * p.channels) : 0;
            ok = stage_in([&](uint32_t aAddr) { tmem_st32(aAddr, h); if (kSplit) tmem_st32(aAddr + 32u, l); }, ke);
          } else {
            float v[kTsK];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              bool on;
              float4 const* const q = reinterpret_cast<float4 const*>(chunk(j, on));
              *reinterpret_cast<float4*>(v + 8 * j) = __ldg(q);
              *reinterpret_cast<float4*>(v + 8 * j + 4) = __ldg(on ? q + p.aLo : q);
            }
            ok = hand_over(v);
          }
          if (!ok) break;
        }
        gi += numIter;
      }
    } else if (kMode == 3) {
      // A k-block is one filter tap and 64 channels: eight 16-byte loads for hi, eight for lo, straight to tensor memory.
      for (int ts = 0; ts < myTiles && ok; ++ts) {
        int const tile = cta + ts * ctas;
        int const tmf = p.dTilesN(tile), split = p.dTilesM(tmf), kb0 = split * numIter;
        int const m = (tmf - split * p.tilesM) * BM + row;
        uint32_t hm = 0, wm = 0;
        uint4 const* xq = p.aHi;
        int8_t const* eq = p.aExp;
        if (m < p.M) {
          int const q = p.dHo(m), n = p.dWo(q), ho = m - q * p.a.Ho, wo = q - n * p.a.Wo;
          long long const pix = (long long)wo * p.a.sx * p.a.H + ho * p.a.sy;
          // (general gather: a.C channels per group, all groups' channels in the tensor, c64 blocks of 64)
          long long const first = (long long)n * p.c64 + (kGen ? (tile - tmf * p.tilesN) / p.tilesPerGroup * (p.a.C / 64) : 0);
          xq += first * 8 * HW + pix;
          eq += first * HW + pix;
          hm = taps_inside(ho * p.a.sy - p.a.pt, p.a.FH, p.a.dy, p.a.H); wm = taps_inside(wo * p.a.sx - p.a.pl, p.a.FW, p.a.dx, p.a.W);
        }
        for (int it = (int)((gi ^ grp) & 1); it < numIter; it += kTsGroups) {
          int const cb = p.dTaps(kb0 + it), tp = kb0 + it - cb * taps;
          int2 const te = tapLut[tp];
          uint32_t const e = (uint32_t)te.y;
          bool const on = ((hm >> (e & 31u)) & (wm >> (e >> 5)) & 1u) != 0 && cb * 64 < p.a.C;      // (cb * 64 >= C: padding of the last range)
          uint4 const* const q = on ? xq + ((long long)(cb * 8) * HW + te.x) : p.zero;
          long long const step = on ? (long long)HW : 0;
          uint4 h[8], l[8];
#pragma unroll
          for (int c = 0; c < 8; ++c) h[c] = __ldg(q + c * step);
          if (kSplit) {
            uint4 const* const ql = on ? q + p.aLo : p.zero;
#pragma unroll
            for (int c = 0; c < 8; ++c) l[c] = __ldg(ql + c * step);
          }
          int const ke = on ? __ldg(eq + (long long)cb * HW + te.x) : 0;
          ok = stage_in([&](uint32_t aAddr) { tmem_st32(aAddr, h); if (kSplit) tmem_st32(aAddr + 32u, l); }, ke);
          if (!ok) break;
        }
        gi += numIter;
      }
    } else {
      for (int ts = 0; ts < myTiles && ok; ++ts) {
        int const tile = cta + ts * ctas;
        int const tmf = p.dTilesN(tile), split = p.dTilesM(tmf), kb0 = split * numIter;     // this item's range starts at k-block kb0
        int const m = (tmf - split * p.tilesM) * BM + row;
        uint32_t hm = 0, wm = 0;                          // tap rows / columns inside the image for this pixel
        float const* xq = p.a.ptr;
        if (m < p.M) {
          int const q = p.dHo(m), n = p.dWo(q), ho = m - q * p.a.Ho, wo = q - n * p.a.Wo;
          xq += (long long)n * p.a.imgStride + (long long)wo * p.a.sx * p.a.H + ho * p.a.sy;
          hm = taps_inside(ho * p.a.sy - p.a.pt, p.a.FH, p.a.dy, p.a.H); wm = taps_inside(wo * p.a.sx - p.a.pl, p.a.FW, p.a.dx, p.a.W);
        }
        for (int it = (int)((gi ^ grp) & 1); it < numIter; it += kTsGroups) {
          float v[kTsK];
          bool on[2];
          // a sub-block is one filter tap and 32 consecutive channels: one validity test, constant stride.  The taps
          // of a channel block follow one another, so that the lines fetched for one tap are still in L1 for the next.
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            int const sub = 2 * (kb0 + it) + h, cb = p.dTaps(sub), tp = sub - cb * taps, c0 = cb * 32;
            int2 const te = tapLut[tp];
            uint32_t const e = (uint32_t)te.y;
            on[h] = ((hm >> (e & 31u)) & (wm >> (e >> 5)) & 1u) != 0 && c0 < p.a.C;      // (c0 >= C: padding of the last range)
            // unconditional loads (a pixel outside the image reads the channels' first pixel of the first image instead and discards it):
            // nothing for the compiler to predicate or branch around, all 64 in flight together
            float const* const q = on[h] ? xq + ((long long)c0 * HW + te.x) : p.a.ptr + (c0 < p.a.C ? (long long)c0 * HW : 0);
#pragma unroll
            for (int k = 0; k < 32; ++k) v[32 * h + k] = __ldg(q + (long long)k * HW);
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (!on[h]) {
#pragma unroll
              for (int k = 0; k < 32; ++k) v[32 * h + k] = 0.f;
            }
          }
          if (!hand_over(v)) { ok = false; break; }
        }
        gi += numIter;
      }
    }
  }

  __syncthreads();
  tc_fence_after();
  if (warp == kTsIssueWarp) tmem_dealloc(tmemAcc, tmemCols);
}

template <bool kSplit, int kMode, bool kNarrow>
__global__ void __launch_bounds__(kMode == 2 ? kTsThreadsRows : kTsThreads, 1)
conv_half_kernel(const __grid_constant__ Params p, const __grid_constant__ CUtensorMap xmap)
{
  conv_half_body<kSplit, kMode, kNarrow, false>(p, &xmap, (int)blockIdx.x, (int)gridDim.x);
}

// The same from chunks (kMode 3) for what the plain kernel does not cover: channels that are no multiple of 32, filter groups, and the residue
// classes of a strided data gradient (several problems in one launch, so that a small layer's classes share the chip).
template <bool kSplit, bool kNarrow, int kMax>
__global__ void __launch_bounds__(kTsThreads, 1) conv_half_gen_kernel(const __grid_constant__ Problems<kMax> b)
{
  int i = 0;
  if constexpr (kMax > 1) while (i + 1 < b.n && (int)blockIdx.x >= b.p[i + 1].ctaBeg) ++i;
  conv_half_body<kSplit, 3, kNarrow, true>(b.p[i], nullptr, (int)blockIdx.x - b.p[i].ctaBeg, b.p[i].ctas);
}

// ------------------------------------------------------------------ tile images
// The B operand of a contraction is small and the same for every CTA: it is split into hi / lo once and laid out as ready-made
// shared-memory tile images -- for n-tile t and k-block kb: [hi tile BN x 64 halves][lo tile BN x 64], K-major with the 128-byte swizzle,
// 16-byte chunk c of row r at chunk c ^ (r & 7) -- so that a stage of B is one bulk copy.  64 rows of an image share a power of two (32 of those of
// prep_image_tiles_kernel), so that the blocks that write them need not agree on one; the exponents go to exps[(t * numKb + kb) * max(BN / 64, 1) + row / 64].
// With kOwnFlag added to that word, own[(t * numKb + kb) * BN + row] is what each of those rows was scaled beyond it (the others' are not written).
struct TileOut {
  uint8_t* img;
  int* exps;
  int8_t* own;
};

// Largest finite magnitude so far (as bits): infinities and not-a-numbers spoil their own column only, not the scale of the others.
__device__ __forceinline__ void max_finite(uint32_t& m, float v)
{
  uint32_t const u = __float_as_uint(v) & 0x7fffffffu;
  if (u < 0x7f800000u) m = max(m, u);
}
__device__ __forceinline__ int tile_exp(uint32_t m) { return m ? scale_exp(__uint_as_float(m)) : 0; }

// The exponent of a set of columns and whether some of them need their own, from the largest magnitudes of the columns: hi is the largest of them, lo
// the smallest but for zeros, less one (all ones: none).  Both as bits.
struct TileScale { int k; bool own; };
__device__ __forceinline__ TileScale tile_scale(uint32_t hi, uint32_t lo)
{
  TileScale t;
  t.k = tile_exp(hi);
  t.own = lo != 0xffffffffu && scale_exp(__uint_as_float(lo + 1u)) - t.k > kOwnScale;
  return t;
}
__device__ __forceinline__ int tile_word(TileScale t) { return t.k + (t.own ? kOwnFlag : 0); }
// What a column whose largest magnitude is m is scaled beyond the tile's exponent k.
__device__ __forceinline__ int own_exp(uint32_t m, int k)
{
  int const c = m ? scale_exp(__uint_as_float(m)) - k : 0;
  return c > kOwnScale ? min(c, kMaxOwnScale) : 0;
}

// tile_scale over a block of kWarps warps whose threads hold hi and lo; red: 2 * kWarps words of shared memory, not touched again before the next block
// barrier but one.
template <int kWarps>
__device__ __forceinline__ TileScale block_scale(uint32_t hi, uint32_t lo, uint32_t* red)
{
  hi = __reduce_max_sync(0xffffffffu, hi);
  lo = __reduce_min_sync(0xffffffffu, lo);
  if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5] = hi; red[kWarps + (threadIdx.x >> 5)] = lo; }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kWarps; ++w) { hi = max(hi, red[w]); lo = min(lo, red[kWarps + w]); }
  return tile_scale(hi, lo);
}

// Eight consecutive reduction indices of one row: 16 bytes of the hi and of the lo tile.
template <bool kSplit>
__device__ __forceinline__ void store_chunk8(uint8_t* img, int BN, int row, int chunk, float const (&v)[8], int k)
{
  float const s = exp2i(k), sl = exp2i(k + 11);
  uint64_t const s2 = pack2(s, s), sl2 = pack2(sl, sl);
  uint32_t h[4], l[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) split_pair<kSplit>(v[2 * e], v[2 * e + 1], s2, sl2, h[e], l[e]);
  uint8_t* const at = img + (size_t)row * kTsRowBytes + ((chunk ^ (row & 7)) << 4);
  *reinterpret_cast<uint4*>(at) = make_uint4(h[0], h[1], h[2], h[3]);
  if (kSplit) *reinterpret_cast<uint4*>(at + (size_t)BN * kTsRowBytes) = make_uint4(l[0], l[1], l[2], l[3]);
}

// The gathered tensor of a convolution, split once instead of once per filter tap and column tile (conv_half_kernel, kMode 3).  A thread takes 64
// channels of a pixel: loads and stores of a warp are whole lines.  (x: 4 bytes in, 4 out per element.)
template <bool kSplit>
__global__ void __launch_bounds__(128)
split_chunks_kernel(uint4* __restrict__ hi, long long loOff, int8_t* __restrict__ exps, uint4* __restrict__ zero, float const* __restrict__ x,
                    int HW, int C, int c64, int pixels, vlb::FastDiv31 divHW)
{
  vlb::pdl_wait();
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *zero = make_uint4(0, 0, 0, 0);
  int const m = (int)blockIdx.x * 128 + (int)threadIdx.x, cb = (int)blockIdx.y;
  if (m >= pixels) return;
  int const img = divHW(m), pix = m - img * HW;
  float const* const src = x + ((long long)img * C + cb * 64) * HW + pix;
  float v[64];
#pragma unroll
  for (int k = 0; k < 64; ++k) v[k] = __ldg(src + (long long)min(k, C - 1 - cb * 64) * HW);
  if (cb * 64 + 64 > C) {                               // channels that do not exist (the last block's)
#pragma unroll
    for (int k = 0; k < 64; ++k) v[k] = cb * 64 + k < C ? v[k] : 0.f;
  }
  float m0 = 0.f, m1 = 0.f;
#pragma unroll
  for (int k = 0; k < 64; k += 4) { m0 = max3(m0, fabsf(v[k]), fabsf(v[k + 1])); m1 = max3(m1, fabsf(v[k + 2]), fabsf(v[k + 3])); }
  float const mx = fmaxf(m0, m1);
  int const ke = mx > 0.f ? scale_exp(mx) : 0;
  float const s = exp2i(ke), sl = exp2i(ke + 11);
  uint64_t const s2 = pack2(s, s), sl2 = pack2(sl, sl);
  uint4* const out = hi + ((long long)img * c64 + cb) * 8 * HW + pix;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) split_pair<kSplit>(v[8 * c + 2 * e], v[8 * c + 2 * e + 1], s2, sl2, h[e], l[e]);
    out[(long long)c * HW] = make_uint4(h[0], h[1], h[2], h[3]);
    if (kSplit) out[loOff + (long long)c * HW] = make_uint4(l[0], l[1], l[2], l[3]);
  }
  exps[((long long)img * c64 + cb) * HW + pix] = (int8_t)ke;
}

// The input of a filter gradient with the images along the reduction, laid out once instead of gathered per filter tap and column tile: chunks of
// eight images of one pixel and channel, channels next to one another.  No filter tap, stride or plane size then moves a chunk off its 16-byte boundary.
// A warp takes eight pixels by four channels: 32-byte pieces in, 64-byte pieces out.
// split_images_kernel (kMode 4): split, with one scale exponent for the 64 images of a pixel and channel, which a thread holds in registers.
// grid (columns of eight pixels * channel blocks of 32, groups of 64 images)
template <bool kSplit>
__global__ void __launch_bounds__(256, 2)
split_images_kernel(uint4* __restrict__ hi, long long loOff, int8_t* __restrict__ exps, uint4* __restrict__ zero, float const* __restrict__ x,
                    int HW, int C, int N, int cBlocks)
{
  vlb::pdl_wait();
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *zero = make_uint4(0, 0, 0, 0);
  int const lane = (int)threadIdx.x & 31, place = (int)blockIdx.x / cBlocks, ng = (int)blockIdx.y;
  int const c = ((int)blockIdx.x - place * cBlocks) * 32 + ((int)threadIdx.x >> 5) * 4 + (lane & 3);
  int const pix = place * 8 + (lane >> 2);
  if (c >= C || pix >= HW) return;
  float const* const src = x + ((long long)ng * 64 * C + c) * HW + pix;
  float v[64];
  long long const step = (long long)C * HW;
  if (ng * 64 + 64 <= N) {
#pragma unroll
    for (int k = 0; k < 64; ++k) v[k] = __ldg(src + k * step);
  } else {
#pragma unroll
    for (int k = 0; k < 64; ++k) v[k] = ng * 64 + k < N ? __ldg(src + k * step) : 0.f;
  }
  float m0 = 0.f, m1 = 0.f;
#pragma unroll
  for (int k = 0; k < 64; k += 4) { m0 = max3(m0, fabsf(v[k]), fabsf(v[k + 1])); m1 = max3(m1, fabsf(v[k + 2]), fabsf(v[k + 3])); }
  float const mx = fmaxf(m0, m1);
  int const ke = mx > 0.f ? scale_exp(mx) : 0;
  float const s = exp2i(ke), sl = exp2i(ke + 11);
  uint64_t const s2 = pack2(s, s), sl2 = pack2(sl, sl);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) split_pair<kSplit>(v[8 * i + 2 * e], v[8 * i + 2 * e + 1], s2, sl2, h[e], l[e]);
    long long const at = ((long long)(ng * 8 + i) * HW + pix) * C + c;
    hi[at] = make_uint4(h[0], h[1], h[2], h[3]);
    if (kSplit) hi[loOff + at] = make_uint4(l[0], l[1], l[2], l[3]);
  }
  exps[((long long)ng * HW + pix) * C + c] = (int8_t)ke;
}

// The same for kMode 5: fp32 values as they are, four images of a chunk at x8, the other four loOff further on.  grid (as above, groups of eight images)
__global__ void __launch_bounds__(256)
gather_images_kernel(float4* __restrict__ x8, long long loOff, uint4* __restrict__ zero, float const* __restrict__ x, int HW, int C, int N, int cBlocks)
{
  vlb::pdl_wait();
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *zero = make_uint4(0, 0, 0, 0);
  int const lane = (int)threadIdx.x & 31, place = (int)blockIdx.x / cBlocks, n0 = (int)blockIdx.y * 8;
  int const c = ((int)blockIdx.x - place * cBlocks) * 32 + ((int)threadIdx.x >> 5) * 4 + (lane & 3);
  int const pix = place * 8 + (lane >> 2);
  if (c >= C || pix >= HW) return;
  long long const step = (long long)C * HW;
  float const* const src = x + n0 * step + (long long)c * HW + pix;
  float v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = n0 + k < N ? __ldg(src + k * step) : 0.f;
  long long const at = ((long long)blockIdx.y * HW + pix) * C + c;
  x8[at] = make_float4(v[0], v[1], v[2], v[3]);
  x8[loOff + at] = make_float4(v[4], v[5], v[6], v[7]);
}

// dY of such a filter gradient as tile images, and the bias gradient from the same sweep.  A block takes 32 filters of a column tile and octets -- eight
// consecutive rows of an output column, the 8 * kG images of a group: kG k-blocks -- one after the other; a thread has one row and filter of it in registers
// (64 values with kG = 8), so that dY is read once.  32 columns of a k-block therefore share an exponent here, not all of the tile's; the drain warps, who
// take 32 columns at a time, have one for each.  (A block of all 128 columns, reading an octet a second time from L2: 196 us for 103 MB, now 55; a range of
// octets of its own per block 61; every octet inside one column 76; every place's image number and magnitude tested by itself 93.)
// A filter's sum: in double over a thread's octets, then over the rows, then (last ticket) over the blocks in block order.
// grid (octets dealt out in turn, blocks of 32 filters of the column tiles of all filter groups)
template <bool kSplit, int kG>
__global__ void __launch_bounds__(256, kG == 8 ? 2 : 3)
prep_image_tiles_kernel(TileOut out, float const* __restrict__ dy, int Ho, int Wo, int N, int K, int Kg, int tilesPerGroup, int BN, int nGroups, int rowBlocks, int kbTot,
                        int octets, float* __restrict__ db, float* __restrict__ dbPart, unsigned* __restrict__ tickets)
{
  vlb::pdl_wait();
  constexpr int kRows = 8 / kG;                         // rows of a k-block
  __shared__ uint2 red[2][8][8];                        // [turn][warp][row of the octet]: largest magnitude, smallest of a filter less one
  __shared__ double sums[256][4];
  __shared__ bool last;
  int const tid = (int)threadIdx.x, warp = tid >> 5, lane = tid & 31, px = lane & 7, f = warp * 4 + (lane >> 3);
  int const perTile = max(BN / 32, 1), tile = (int)blockIdx.y / perTile, fb = (int)blockIdx.y - tile * perTile;
  int const fg = tile / tilesPerGroup, local = (tile - fg * tilesPerGroup) * BN + fb * 32 + f, row = fb * 32 + f;      // row of the tile image
  bool const rowOn = row < BN, real = rowOn && local < Kg;
  int const P = Ho * Wo, perCol = (Ho + 7) / 8;
  long long const imgStep = (long long)K * P;
  float const* const mine = dy + (long long)(real ? fg * Kg + local : 0) * P;
  double acc = 0.0;
  // (blocks that run at the same time take neighbouring octets: with a range of its own for each, 64 images far apart times hundreds of places are more
  // pages than the address translation holds)
  int turn = 0;
  for (int o = (int)blockIdx.x; o < octets; o += (int)gridDim.x, turn ^= 1) {
    int const col = o / perCol, h8 = o - col * perCol, ng = col / Wo, w = col - ng * Wo, h = h8 * 8 + px;
    int const kbAt = h8 * kG + px / kRows, kb = col * rowBlocks + kbAt;
    bool const on = real && ng < nGroups && h < Ho;
    float const* const src = mine + (long long)ng * 8 * kG * imgStep + w * Ho + h;
    float v[8 * kG];
    if (!on) {
#pragma unroll
      for (int n = 0; n < 8 * kG; ++n) v[n] = 0.f;
    } else if (ng * 8 * kG + 8 * kG <= N) {
#pragma unroll
      for (int n = 0; n < 8 * kG; ++n) v[n] = __ldg(src + n * imgStep);
    } else {
#pragma unroll
      for (int n = 0; n < 8 * kG; ++n) v[n] = ng * 8 * kG + n < N ? __ldg(src + n * imgStep) : 0.f;
    }
    float m0 = 0.f, m1 = 0.f, sum = 0.f;
#pragma unroll
    for (int n = 0; n < 8 * kG; n += 8) {
      m0 = max3(m0, fabsf(v[n]), fabsf(v[n + 1])); m1 = max3(m1, fabsf(v[n + 2]), fabsf(v[n + 3]));
      m0 = max3(m0, fabsf(v[n + 4]), fabsf(v[n + 5])); m1 = max3(m1, fabsf(v[n + 6]), fabsf(v[n + 7]));
      sum += ((v[n] + v[n + 1]) + (v[n + 2] + v[n + 3])) + ((v[n + 4] + v[n + 5]) + (v[n + 6] + v[n + 7]));
    }
    acc += (double)sum;
    uint32_t m = __float_as_uint(fmaxf(m0, m1));
    if (m >= 0x7f800000u) {                             // an infinity among them (a not-a-number counts as nothing in the maximum): the largest finite one
      m = 0;
#pragma unroll
      for (int n = 0; n < 8 * kG; ++n) max_finite(m, v[n]);
    }
#pragma unroll
    for (int q = 1; q < kRows; q <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, q));
    uint32_t const fMax = m;                           // of this filter in the k-block
    uint32_t lo = m - 1u;
#pragma unroll
    for (int q = 8; q < 32; q <<= 1) { m = max(m, __shfl_xor_sync(0xffffffffu, m, q)); lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, q)); }
    uint2 (&r)[8][8] = red[turn];                       // (written again two octets on, with a barrier in between)
    if (lane < 8) r[warp][px] = make_uint2(m, lo);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) { uint2 const u = r[q][px]; m = max(m, u.x); lo = min(lo, u.y); }
    TileScale const ts = tile_scale(m, lo);
    int const own = ts.own ? own_exp(fMax, ts.k) : 0;
    float const s = exp2i(ts.k + own), sl = exp2i(ts.k + own + 11);
    uint64_t const s2 = pack2(s, s), sl2 = pack2(sl, sl);
    size_t const imgBytes = (kSplit ? 2 : 1) * (size_t)BN * kTsRowBytes;
    uint8_t* const rowAt = out.img + (size_t)tile * kbTot * imgBytes + (size_t)row * kTsRowBytes;
    bool const kbOn = rowOn && kbAt < rowBlocks && kb < kbTot;
    // Neighbouring chunks of an image row belong to one thread (two groups of images) where kG > 1.  Rows of pixels change hands in pairs, so that two threads
    // write them together, a whole 32-byte sector: the even thread takes the even chunks of both, the odd one the odd ones.
    bool const oddPx = (px & 1) != 0;
    int const kbO = __shfl_xor_sync(0xffffffffu, kb, 1);
    bool const kbOnO = __shfl_xor_sync(0xffffffffu, kbOn ? 1 : 0, 1) != 0;
    uint8_t* const at0 = rowAt + (size_t)(oddPx ? kbO : kb) * imgBytes;      // image row of the even pixel of the pair, of the odd one
    uint8_t* const at1 = rowAt + (size_t)(oddPx ? kb : kbO) * imgBytes;
    bool const on0 = oddPx ? kbOnO : kbOn, on1 = oddPx ? kbOn : kbOnO;
    auto put = [&](uint8_t* at, int chunk, uint4 const& h4, uint4 const& l4) {
      uint8_t* const c = at + ((chunk ^ (row & 7)) << 4);
      *reinterpret_cast<uint4*>(c) = h4;
      if (kSplit) *reinterpret_cast<uint4*>(c + (size_t)BN * kTsRowBytes) = l4;
    };
    auto halves = [&](int i, uint4& h4, uint4& l4) {
      split_pair<kSplit>(v[8 * i], v[8 * i + 1], s2, sl2, h4.x, l4.x); split_pair<kSplit>(v[8 * i + 2], v[8 * i + 3], s2, sl2, h4.y, l4.y);
      split_pair<kSplit>(v[8 * i + 4], v[8 * i + 5], s2, sl2, h4.z, l4.z); split_pair<kSplit>(v[8 * i + 6], v[8 * i + 7], s2, sl2, h4.w, l4.w);
    };
    auto swap4 = [&](uint4 const& a) {
      return make_uint4(__shfl_xor_sync(0xffffffffu, a.x, 1), __shfl_xor_sync(0xffffffffu, a.y, 1), __shfl_xor_sync(0xffffffffu, a.z, 1), __shfl_xor_sync(0xffffffffu, a.w, 1));
    };
    if constexpr (kG == 1) {
      uint4 h4, l4;
      halves(0, h4, l4);
      if (kbOn) put(rowAt + (size_t)kb * imgBytes, px, h4, l4);
    } else {
#pragma unroll
      for (int i = 0; i < kG; i += 2) {
        uint4 h0, l0, h1, l1;
        halves(i, h0, l0);
        halves(i + 1, h1, l1);
        uint4 const hr = swap4(oddPx ? h0 : h1), lr = kSplit ? swap4(oddPx ? l0 : l1) : hr;
        int const mine = i + (oddPx ? 1 : 0);             // this thread's chunk of both rows
        if (on0) put(at0, ((px & ~1) % kRows) * kG + mine, oddPx ? hr : h0, oddPx ? lr : l0);
        if (on1) put(at1, ((px | 1) % kRows) * kG + mine, oddPx ? h1 : hr, oddPx ? l1 : lr);
      }
    }
    if (kbOn && px % kRows == 0) {
      size_t const image = (size_t)tile * kbTot + kb;
      if (f == 0) out.exps[image * perTile + fb] = tile_word(ts);
      if (ts.own) out.own[image * BN + row] = (int8_t)own;
    }
  }
  if (db == nullptr) return;
#pragma unroll
  for (int q = 1; q < 8; q <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, q);
  if (px == 0) dbPart[((size_t)blockIdx.x * gridDim.y + blockIdx.y) * 32 + f] = (float)acc;
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(&tickets[blockIdx.y], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  int const c = tid & 7, gr = tid >> 3;                 // four filters; every 32nd block
  double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
  for (unsigned i = gr; i < gridDim.x; i += 32) {
    float4 const q = __ldcg(reinterpret_cast<float4 const*>(dbPart + ((size_t)i * gridDim.y + blockIdx.y) * 32) + c);
    t[0] += q.x; t[1] += q.y; t[2] += q.z; t[3] += q.w;
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) sums[tid][e] = t[e];
  __syncthreads();
  if (gr == 0) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      for (int j = 1; j < 32; ++j) t[e] += sums[j * 8 + c][e];
      int const n = (tile - fg * tilesPerGroup) * BN + fb * 32 + 4 * c + e;
      if (fb * 32 + 4 * c + e < BN && n < Kg) db[fg * Kg + n] = (float)t[e];
    }
  }
  if (tid == 0) tickets[blockIdx.y] = 0;      // ready for the next call
}

// Dense operands: kRows: B(n, r) = f[n*R + r]; else B(n, r) = f[n + N*r].  A block per image (blockIdx.x = tile * numKb + kb), 16-byte
// chunks dealt to the threads along the contiguous index.
template <bool kSplit, bool kRows>
__global__ void __launch_bounds__(256) prep_dense_tiles_kernel(TileOut out, float const* __restrict__ f, int N, int R, int BN, int numKb)
{
  vlb::pdl_wait();
  __shared__ uint32_t colMax[BM];                       // largest magnitude of each row of the image
  int const tid = (int)threadIdx.x, tile = (int)blockIdx.x / numKb, kb = (int)blockIdx.x - tile * numKb, items = BN * 8;
  if (tid < BM) colMax[tid] = 0u;
  float v[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int const it = tid + 256 * i;
    int const row = kRows ? it >> 3 : it % BN, chunk = kRows ? it & 7 : it / BN, n = tile * BN + row, r0 = kb * kTsK + chunk * 8;
#pragma unroll
    for (int e = 0; e < 8; ++e) v[i][e] = it < items && n < N && r0 + e < R ? __ldg(f + (kRows ? (size_t)n * R + r0 + e : (size_t)(r0 + e) * N + n)) : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int const it = tid + 256 * i;
    uint32_t m = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) max_finite(m, v[i][e]);
    if (it < items && m) atomicMax(&colMax[kRows ? it >> 3 : it % BN], m);
  }
  __syncthreads();
  uint32_t hi = 0, lo = 0xffffffffu;
  for (int c = tid & 31; c < BN; c += 32) { uint32_t const m = colMax[c]; hi = max(hi, m); lo = min(lo, m - 1u); }
  TileScale const ts = tile_scale(__reduce_max_sync(0xffffffffu, hi), __reduce_min_sync(0xffffffffu, lo));
  uint8_t* const img = out.img + (size_t)blockIdx.x * ((kSplit ? 2 : 1) * (size_t)BN * kTsRowBytes);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int const it = tid + 256 * i;
    if (it < items) {
      int const row = kRows ? it >> 3 : it % BN, chunk = kRows ? it & 7 : it / BN, own = ts.own ? own_exp(colMax[row], ts.k) : 0;
      store_chunk8<kSplit>(img, BN, row, chunk, v[i], ts.k + own);
      if (ts.own && chunk == 0) out.own[(size_t)blockIdx.x * BN + row] = (int8_t)own;
    }
  }
  int const perImage = max(BN / 64, 1);
  if (tid < perImage) out.exps[(size_t)blockIdx.x * perImage + tid] = tile_word(ts);
}

// Filter tile images for conv_half_kernel and conv_half_gen_kernel, for filter groups, tap subsets
// (residue classes of a strided data gradient) and shuffled columns of the general gather.  Row n of a tile is column n of its
// group; tap (fh', fw') of the problem is tap (bh + ah*fh', bw + aw*fw') of the filter bank, zero where that does not exist; the
// filter of (column channel n, reduction channel q) starts at F + FH*FW * (gs*group + sn*n + sq*q).
struct PrepFilters {
  TileOut out;
  float const* f;
  int BN, numKb, rows, tilesPerGroup, cols, tapsH, tapsW, C, FH, FW, bh, ah, bw, aw, shufY, shufX;
  int whole;                        // k-block kb is tap kb % taps of the 64 channels from 64 * (kb / taps) on (kMode 3), not two sub-blocks of one tap of 32
  long long sn, sq, gs;
  vlb::FastDiv31 divTaps, divTapsH;                 // by tapsH * tapsW and tapsH (set by launch_prep)
};
template <int kMax> struct PrepBatchOf { PrepFilters p[kMax]; };
using PrepBatch = PrepBatchOf<kMaxTsProblems>;

template <int kMax>
PrepBatchOf<kMax> first_preps(PrepBatch const& b)
{
  PrepBatchOf<kMax> q;
  std::copy(b.p, b.p + kMax, q.p);
  return q;
}

// A block takes 64 rows of an image (all of a narrower tile), a thread eight places of one row.  Grid (tiles * numKb * blocks per image, problems).  Bound by the
// scattered 4-byte reads, one request per place: with a block per image 7 us for 128 -> 128 channels, 3x3, with two 3.5.  (Through shared memory, in
// runs of the taps of sixteen channels: 15 us against 13 for 512 -> 512 channels.)
template <bool kSplit, int kMax>
__global__ void __launch_bounds__(512) prep_filters_kernel(const __grid_constant__ PrepBatchOf<kMax> b)
{
  vlb::pdl_wait();
  __shared__ uint32_t red[32];
  PrepFilters const& p = b.p[blockIdx.y];
  int const per = max(p.BN / 64, 1), img = (int)blockIdx.x / per, tile = img / p.numKb, kb = img - tile * p.numKb;
  if (tile * p.BN >= p.rows) return;
  int const grp = tile / p.tilesPerGroup, col0 = (tile - grp * p.tilesPerGroup) * p.BN;
  int const taps = p.tapsH * p.tapsW, FT = p.FH * p.FW;
  int const row = ((int)blockIdx.x - img * per) * 64 + ((int)threadIdx.x >> 3), chunk = (int)threadIdx.x & 7, col = col0 + row;
  float v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = 0.f;
  if (row < p.BN && col < p.cols) {
    int ry = 0, rx = 0, n = col;
    if (p.shufY > 0) { n = col / (p.shufY * p.shufX); int const t = col - n * p.shufY * p.shufX; rx = t / p.shufY; ry = t - rx * p.shufY; }
    float const* const fn = p.f + (long long)FT * (p.gs * grp + p.sn * n);
    // the chunk's eight places are channels of one tap
    int const un = p.whole ? kb : 2 * kb + (chunk >> 2), cb = p.divTaps(un), tap = un - cb * taps, q0 = p.whole ? cb * 64 + chunk * 8 : cb * 32 + (chunk & 3) * 8;
    int const tw = p.divTapsH(tap), th = tap - tw * p.tapsH, fh = p.bh + p.ah * th + ry, fw = p.bw + p.aw * tw + rx;
    if ((unsigned)fh < (unsigned)p.FH && (unsigned)fw < (unsigned)p.FW) {
#pragma unroll
      for (int e = 0; e < 8; ++e) if (q0 + e < p.C) v[e] = __ldg(fn + (long long)FT * p.sq * (q0 + e) + (fh + p.FH * fw));
    }
  }
  uint32_t m = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e) max_finite(m, v[e]);
#pragma unroll
  for (int q = 1; q < 8; q <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, q));      // (the eight threads of a row are neighbours)
  TileScale const ts = block_scale<16>(m, m - 1u, red);
  int const own = ts.own ? own_exp(m, ts.k) : 0;
  if (row < p.BN) {
    store_chunk8<kSplit>(p.out.img + (size_t)img * ((kSplit ? 2 : 1) * (size_t)p.BN * kTsRowBytes), p.BN, row, chunk, v, ts.k + own);
    if (ts.own && chunk == 0) p.out.own[(size_t)img * p.BN + row] = (int8_t)own;
  }
  if (threadIdx.x == 0) p.out.exps[blockIdx.x] = tile_word(ts);
}

// Launches the tile-image kernel for n problems whose output pointers are set.  The problems share the tile width.
void launch_prep(vlb_ctx* ctx, PrepBatch& prep, int n)
{
  bool const split3 = ctx->precision == VLB_PRECISION_3XTF32;
  long long images = 0;
  for (int i = 0; i < n; ++i) {
    PrepFilters& q = prep.p[i];
    q.divTaps = vlb::FastDiv31(q.tapsH * q.tapsW); q.divTapsH = vlb::FastDiv31(q.tapsH);
    images = std::max(images, (long long)q.rows / q.BN * q.numKb);
  }
  VLB_LAUNCHED(ctx, 1);
  dim3 const grid((unsigned)(images * std::max(prep.p[0].BN / 64, 1)), n, 1);
  with_capacity(n, [&](auto capacity) {
    constexpr int kMax = decltype(capacity)::value;
    if (split3) vlb::launch(ctx->stream, prep_filters_kernel<true, kMax>, grid, 512, 0, first_preps<kMax>(prep));
    else        vlb::launch(ctx->stream, prep_filters_kernel<false, kMax>, grid, 512, 0, first_preps<kMax>(prep));
  });
}

// dY of a filter gradient as tile images, B(n, r) = dY[pixel, n, image] with r = pixel + Pp*image (Pp: the plane's P pixels rounded up to whole
// k-blocks, the pixels added read as zeros), for planes of a multiple of four pixels on a 16-byte boundary: 16-byte loads along the pixels, and -- dY being read
// anyway -- the bias gradient db[n] = sum of dY over pixels and images (reference bits/nnconv.cu:141-149) on
// the way: per-block partial sums, and the block that takes a tile's last ticket adds them in block order,
// so the result does not depend on the scheduling.
// grid (ranges of k-blocks, column tiles).  A block takes `per` consecutive k-blocks of a tile: sixteen threads per row (64 pixels), sixteen rows per
// pass, BN / 16 passes; the next k-block's values are asked for before this one's maximum is agreed on.
template <bool kSplit, int kPasses>
__global__ void __launch_bounds__(256)
prep_pixel_tiles_kernel(TileOut out, float const* __restrict__ dy, int N, int images, int P, int Pp, int numKb, int per,
                        float* __restrict__ db, float* __restrict__ dbPart, unsigned* __restrict__ tickets)
{
  vlb::pdl_wait();
  constexpr int BN = 16 * kPasses;
  __shared__ uint32_t red[2][16];
  __shared__ double sums[256][4];
  __shared__ bool last;
  int const tid = (int)threadIdx.x, tile = (int)blockIdx.y, row0 = tid >> 4, c4 = tid & 15;
  int const kbBeg = (int)blockIdx.x * per, kbEnd = min(numKb, kbBeg + per), kbPer = Pp / kTsK;
  int const n0 = tile * BN + row0;
  float4 v[kPasses], w[kPasses];
  float inner[kPasses], outer[kPasses];
#pragma unroll
  for (int i = 0; i < kPasses; ++i) inner[i] = outer[i] = 0.f;
  int img = kbBeg / kbPer, kq = kbBeg - img * kbPer;
  auto fetch = [&](float4 (&d)[kPasses]) {
    int const pix = kq * kTsK + c4 * 4;
    bool const on = pix < P && img < images;
    float const* const src = dy + ((size_t)img * N + n0) * P + pix;
#pragma unroll
    for (int i = 0; i < kPasses; ++i)
      d[i] = on && n0 + 16 * i < N ? *reinterpret_cast<float4 const*>(src + (size_t)(16 * i) * P) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (++kq == kbPer) { kq = 0; ++img; }
  };
  if (kbBeg < kbEnd) fetch(w);
  for (int kb = kbBeg; kb < kbEnd; ++kb) {
#pragma unroll
    for (int i = 0; i < kPasses; ++i) v[i] = w[i];
    if (kb + 1 < kbEnd) fetch(w);
    uint32_t hi = 0, lo = 0xffffffffu;
    auto largest = [&](float4 const& a) { uint32_t m = 0; max_finite(m, a.x); max_finite(m, a.y); max_finite(m, a.z); max_finite(m, a.w); return m; };
#pragma unroll
    for (int i = 0; i < kPasses; ++i) {
      uint32_t const m = largest(v[i]);
      hi = max(hi, m); lo = min(lo, m - 1u);
      inner[i] += (v[i].x + v[i].y) + (v[i].z + v[i].w);
    }
    if (((kb - kbBeg) & 7) == 7) {      // (sums of eight, then of those: a long range keeps its digits)
#pragma unroll
      for (int i = 0; i < kPasses; ++i) { outer[i] += inner[i]; inner[i] = 0.f; }
    }
    // (four values of a row are the least: where they call for powers of their own, the rows' largest magnitudes decide)
    TileScale ts = block_scale<8>(hi, lo, red[kb & 1]);
    unsigned long long own = 0;                         // a byte for each pass
    if (ts.own) {
#pragma unroll
      for (int i = 0; i < kPasses; ++i) {
        uint32_t m = largest(v[i]);
        for (int o = 8; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        own |= (unsigned long long)own_exp(m, ts.k) << (8 * i);
      }
      ts.own = __syncthreads_or(own != 0) != 0;
      if (ts.own && c4 == 0) {
#pragma unroll
        for (int i = 0; i < kPasses; ++i) out.own[((size_t)tile * numKb + kb) * BN + row0 + 16 * i] = (int8_t)(own >> (8 * i));
      }
    }
    float const s = exp2i(ts.k), sl = exp2i(ts.k + 11);
    uint64_t s2 = pack2(s, s), sl2 = pack2(sl, sl);
    uint8_t* const at = out.img + ((size_t)tile * numKb + kb) * ((kSplit ? 2 : 1) * (size_t)BN * kTsRowBytes) + (size_t)row0 * kTsRowBytes +
                        (((c4 >> 1) ^ (row0 & 7)) << 4) + (c4 & 1) * 8;      // (rows 16 apart share the swizzle)
#pragma unroll
    for (int i = 0; i < kPasses; ++i) {
      uint2 h, l;
      if (ts.own) {
        int const k = ts.k + (int)((own >> (8 * i)) & 255u);
        s2 = pack2(exp2i(k), exp2i(k)); sl2 = pack2(exp2i(k + 11), exp2i(k + 11));
      }
      split_pair<kSplit>(v[i].x, v[i].y, s2, sl2, h.x, l.x);
      split_pair<kSplit>(v[i].z, v[i].w, s2, sl2, h.y, l.y);
      *reinterpret_cast<uint2*>(at + (size_t)(16 * i) * kTsRowBytes) = h;
      if (kSplit) *reinterpret_cast<uint2*>(at + (size_t)(BN + 16 * i) * kTsRowBytes) = l;
    }
    constexpr int kPerImage = BN >= 64 ? BN / 64 : 1;
    if (tid < kPerImage) out.exps[((size_t)tile * numKb + kb) * kPerImage + tid] = tile_word(ts);
  }
  if (db == nullptr) return;
  int const rows = (int)gridDim.y * BN;
#pragma unroll
  for (int i = 0; i < kPasses; ++i) {
    float s = outer[i] + inner[i];
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (c4 == 0) dbPart[(size_t)blockIdx.x * rows + n0 + 16 * i] = s;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(&tickets[tile], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // the tile's partial sums in block order: four rows per thread, BN / 4 threads side by side, the blocks dealt to the groups of BN / 4
  constexpr int kSide = BN / 4, kGroups = 256 / kSide;
  int const c = tid % kSide, gr = tid / kSide;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
  for (unsigned i = gr; i < gridDim.x; i += kGroups) {
    float4 const q = __ldcg(reinterpret_cast<float4 const*>(dbPart + (size_t)i * rows + tile * BN) + c);
    s[0] += q.x; s[1] += q.y; s[2] += q.z; s[3] += q.w;
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) sums[tid][e] = s[e];
  __syncthreads();
  if (gr == 0) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      for (int j = 1; j < kGroups; ++j) s[e] += sums[j * kSide + c][e];
      if (tile * BN + 4 * c + e < N) db[tile * BN + 4 * c + e] = (float)s[e];
    }
  }
  if (tid == 0) tickets[tile] = 0;      // ready for the next call
}

// The tile images of conv_half_kernel in the context's scratch: images, exponents, the columns' own ones, then the caller's bytes.
size_t ts_images_bytes(vlb_ctx* ctx, size_t images, int BN)      // (a multiple of 2048)
{ return images * (ctx->precision == VLB_PRECISION_3XTF32 ? 2 : 1) * (size_t)BN * kTsRowBytes; }

size_t ts_exps_bytes(size_t images, int BN) { return (images * std::max(BN / 32, 1) * sizeof(int) + 255) & ~(size_t)255; }

size_t ts_tiles_bytes(vlb_ctx* ctx, int rows, int BN, int numKb)
{
  size_t const images = (size_t)vlb::ceil_div(rows, BN) * (size_t)numKb;
  return ts_images_bytes(ctx, images, BN) + ts_exps_bytes(images, BN) + ((images * BN + 255) & ~(size_t)255);
}

TileOut ts_tiles_at(vlb_ctx* ctx, void* at, int rows, int BN, int numKb)
{
  size_t const images = (size_t)vlb::ceil_div(rows, BN) * (size_t)numKb;
  TileOut out;
  out.img = (uint8_t*)at;
  out.exps = (int*)(out.img + ts_images_bytes(ctx, images, BN));
  out.own = (int8_t*)out.exps + ts_exps_bytes(images, BN);
  return out;
}

constexpr int kMaxGridY = 65535;      // (blocks of 64 channels, groups of images; fully connected layers that fit 32-bit counting have 2^14 at most, the general gather 2^15)

// Scratch of the split form of a tensor of `elements` values in whole blocks of 64 channels.
size_t chunks_bytes(vlb_ctx* ctx, long long elements)
{
  return (size_t)elements * (ctx->precision == VLB_PRECISION_3XTF32 ? 4 : 2) + (((size_t)elements / 64 + 255) & ~(size_t)255) + 256;
}

// Splits p's gathered tensor (p.a, `images` of `channels`) into `at` and points p at it.
void split_chunks(vlb_ctx* ctx, Params& p, void* at, int images, int channels)
{
  bool const split3 = ctx->precision == VLB_PRECISION_3XTF32;
  p.c64 = vlb::ceil_div(channels, 64);
  long long const HW = (long long)p.a.H * p.a.W, elements = HW * p.c64 * 64 * images;
  uint4* const hi = (uint4*)at;
  p.aHi = hi; p.aLo = elements / 8;
  char* const behind = (char*)at + (size_t)elements * (split3 ? 4 : 2);
  p.zero = (uint4 const*)behind; p.aExp = (int8_t const*)(behind + 256);
  dim3 const grid((unsigned)vlb::ceil_div(HW * images, 128), (unsigned)p.c64, 1);
#define VLB_SC(split) vlb::launch(ctx->stream, split_chunks_kernel<split>, grid, 128, 0, hi, p.aLo, (int8_t*)(behind + 256), (uint4*)behind, p.a.ptr, (int)HW, channels, p.c64, (int)(HW * images), vlb::FastDiv31((int)HW))
  if (split3) VLB_SC(true); else VLB_SC(false);
#undef VLB_SC
  VLB_LAUNCHED(ctx, 1);
}

// Scratch for the images of p's B operand (p.N columns, p.numKb k-blocks) and `extraBytes` behind them for the caller (*extra); false: error set.
bool ts_tiles(vlb_ctx* ctx, Params& p, size_t extraBytes, TileOut* out, float** extra = nullptr)
{
  size_t const bytes = ts_tiles_bytes(ctx, p.N, p.BN, p.numKb);
  char* const ws = (char*)vlb::workspace(ctx, bytes + extraBytes);
  if (!ws) return false;
  *out = ts_tiles_at(ctx, ws, p.N, p.BN, p.numKb);
  p.bTiles = (float const*)out->img; p.bExp = out->exps; p.bOwn = out->own;
  if (extra) *extra = (float*)(ws + bytes);
  return true;
}

bool prep_dense_tiles(vlb_ctx* ctx, Params& p, float const* f, bool rows, size_t extraBytes = 0, float** extra = nullptr)
{
  TileOut out;
  if (!ts_tiles(ctx, p, extraBytes, &out, extra)) return false;
  unsigned const grid = (unsigned)(vlb::ceil_div(p.N, p.BN) * p.numKb);
#define VLB_PD(split, r) vlb::launch(ctx->stream, prep_dense_tiles_kernel<split, r>, grid, 256, 0, out, f, p.N, p.R, p.BN, p.numKb)
  if (ctx->precision == VLB_PRECISION_3XTF32) { if (rows) VLB_PD(true, true); else VLB_PD(true, false); }
  else                                        { if (rows) VLB_PD(false, true); else VLB_PD(false, false); }
#undef VLB_PD
  VLB_LAUNCHED(ctx, 1);
  return true;
}

// The filter bank of one group flipped and transposed, for the data gradient of a stride-1 convolution (conv_half_kernel).
// Where it pays and there is room for the chunks, the gathered tensor is split beforehand (kMode 3).
bool prep_flipped_tiles(vlb_ctx* ctx, Params& p, float const* f, vlb::ConvGeom const& g, size_t extraBytes, float** extra)
{
  PrepBatch prep = {};
  PrepFilters& q = prep.p[0];
  extraBytes = (extraBytes + 255) & ~(size_t)255;
  int const images = p.M / (p.a.Ho * p.a.Wo);
  long long const elements = (long long)p.a.H * p.a.W * vlb::ceil_div(p.a.C, 64) * 64 * images;
  int const chunkKb = vlb::ceil_div(p.a.FH * p.a.FW * vlb::ceil_div(p.a.C, 64), p.splits);
  bool const chunks = split_pays(p.a.C, 1, p.a.FH * p.a.FW * vlb::ceil_div(p.N, p.BN)) && vlb::ceil_div(p.a.C, 64) <= kMaxGridY &&
                      vlb::try_workspace(ctx, ts_tiles_bytes(ctx, p.N, p.BN, p.splits * chunkKb) + extraBytes + chunks_bytes(ctx, elements));
  if (chunks) p.numKb = p.splits * (p.kbPerSplit = chunkKb);
  float* behind = nullptr;
  if (!ts_tiles(ctx, p, extraBytes + (chunks ? chunks_bytes(ctx, elements) : 0), &q.out, &behind)) return false;
  if (extra) *extra = behind;
  if (chunks) split_chunks(ctx, p, (char*)behind + extraBytes, images, p.a.C);
  q.f = f; q.BN = p.BN; q.numKb = p.numKb; q.tilesPerGroup = vlb::ceil_div(p.N, p.BN); q.rows = q.tilesPerGroup * p.BN; q.cols = p.N;
  q.tapsH = q.FH = g.FH; q.tapsW = q.FW = g.FW; q.C = g.K;
  q.bh = g.FH - 1; q.bw = g.FW - 1; q.ah = q.aw = -1;
  q.sn = 1; q.sq = g.C; q.whole = p.aHi != nullptr;
  launch_prep(ctx, prep, 1);
  return true;
}

// B(n, r) = dY[pixel, n, image], r = pixel + p.plane * image, and, when db is given, the bias gradient from the same sweep.
bool prep_pixel_tiles(vlb_ctx* ctx, Params& p, float const* dY, int P, int images, size_t extraBytes, float** extra, float* db)
{
  int const tiles = vlb::ceil_div(p.N, p.BN);
  // three blocks per SM; a block's range at least four k-blocks where there are that many
  int const ranges = std::max(1, std::min(3 * ctx->smCount / tiles, vlb::ceil_div(p.numKb, 4)));
  int const per = vlb::ceil_div(p.numKb, ranges), gx = vlb::ceil_div(p.numKb, per);
  extraBytes = (extraBytes + 255) & ~(size_t)255;
  TileOut out;
  float* at = nullptr;
  if (!ts_tiles(ctx, p, extraBytes + (db ? sizeof(float) * (size_t)gx * tiles * p.BN : 0), &out, &at)) return false;
  if (extra) *extra = at;
  float* const dbPart = db ? (float*)((char*)at + extraBytes) : nullptr;
  unsigned* const tickets = (unsigned*)((char*)ctx->deviceStatus + 256);
  dim3 const grid((unsigned)gx, (unsigned)tiles, 1);
  bool const split3 = ctx->precision == VLB_PRECISION_3XTF32;
#define VLB_PP(split, passes) vlb::launch(ctx->stream, prep_pixel_tiles_kernel<split, passes>, grid, 256, 0, out, dY, p.N, images, P, p.plane, p.numKb, per, db, dbPart, tickets)
#define VLB_PPS(passes) do { if (split3) VLB_PP(true, passes); else VLB_PP(false, passes); } while (0)
  if (p.BN == 128) VLB_PPS(8); else if (p.BN == 64) VLB_PPS(4); else if (p.BN == 32) VLB_PPS(2); else VLB_PPS(1);
#undef VLB_PPS
#undef VLB_PP
  VLB_LAUNCHED(ctx, 1);
  return true;
}

template <> constexpr int kRegsAtLaunch<conv_half_kernel<true, 0, true>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<true, 0, false>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<true, 1, true>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<true, 1, false>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<true, 4, true>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<true, 4, false>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<false, 4, true>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<false, 4, false>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<true, 5, true>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<true, 5, false>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<false, 5, true>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<false, 5, false>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<true, 2, false>>() { return 80; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<true, 3, true>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<true, 3, false>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<false, 3, true>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<false, 3, false>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<false, 0, true>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<false, 0, false>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<false, 1, true>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<false, 1, false>>() { return 96; }
template <> constexpr int kRegsAtLaunch<conv_half_kernel<false, 2, false>>() { return 80; }

// Decides whether conv_half_kernel can take its input windows from tensor-map copies and, if so, fills the box geometry in p,
// the tensor map and the shared-memory size.  Needs: reduction in blocks of 32 channels, unit stride, input rows a multiple
// of four elements (every global stride of a tensor map is a multiple of 16 bytes) on a 16-byte aligned base, an output
// map that boxes of bh x bw <= 128 pixels (bh a multiple of four, so that every box's window starts on a 16-byte boundary)
// cover with at least 95% of the tile rows in use (measured: with 112 of 128 rows in use, as on 56 x 56 and 28 x 28 maps,
// the per-thread gather is the faster route by 10-15%; on 224 x 224 and 112 x 112 maps the copies win by up to 20% on
// 64-column tiles and draw level on 128-column tiles), and room in shared memory for two windows.
// Shared memory of conv_half_kernel for the stores that do not go straight from registers: a patch of 32 columns.
size_t p_bytes(int BN) { return sizeof(float) * (size_t)std::min(BN, 32) * BM; }

bool plan_windows(vlb_ctx* ctx, Params& p, CUtensorMap* map, size_t* smemBytes, bool split3)
{
  Operand const& a = p.a;
  if (ctx->testSwitch & 2) return false;
  if (!p.chanFast || a.sy != 1 || a.sx != 1 || a.H % 4 != 0 || !aligned16(a.ptr)) return false;
  if (p.splits > 1 && 2 * p.kbPerSplit % (a.FH * a.FW) != 0) return false;      // a range of the reduction must be whole channel blocks
  EncodeTiledFn const encode = encode_tiled();
  if (!encode) return false;
  int const Ho = a.Ho, Wo = a.Wo;
  int bestBh = 0, bestBw = 0;
  double bestUtil = 0.0;
  for (int bh = 4; bh <= 128 && bh < Ho + 4; bh += 4) {
    int const bw = std::min(128 / bh, Wo);
    // share of the 128 tile rows that are output pixels, over all boxes of an image
    double const util = (double)Ho * Wo / ((double)vlb::ceil_div(Ho, bh) * (double)vlb::ceil_div(Wo, bw) * 128.0);
    if (util >= bestUtil - 1e-9) { bestUtil = util; bestBh = bh; bestBw = bw; }      // on a tie the taller box: longer contiguous runs
  }
  if (bestBh == 0 || bestUtil < 0.95) return false;
  int const rowOff = (4 - a.pt % 4) % 4;
  int const boxH = (rowOff + bestBh + (a.FH - 1) * a.dy + 3) / 4 * 4, boxW = bestBw + (a.FW - 1) * a.dx;
  if (boxH > 256 || boxW > 256) return false;
  size_t const xTileBytes = (size_t)boxH * boxW * 32 * 4;
  size_t const bBytes = (size_t)(split3 ? 2 : 1) * p.BN * kTsRowBytes, pBytes = p_bytes(p.BN);
  size_t const limit = 227 * 1024 - kTsStatic;      // what one block may have, less the kernel's static shared memory
  // window buffers: two where a window serves a whole channel block of several taps; six for 1 x 1 filters, whose windows are
  // half k-blocks and must be on their way well before their turn.  Filter-tile stages: what is left, at least three.
  int const nX = a.FH * a.FW == 1 ? kTsXStages : 2;
  int nB = 0;
  for (int n = kTsBStages; n >= 3 && !nB; --n)
    if ((size_t)n * bBytes + pBytes + nX * xTileBytes + 1024 <= limit) nB = n;
  if (!nB) return false;
  long long const images = (long long)p.M / ((long long)Ho * Wo);
  cuuint64_t const dims[4] = {(cuuint64_t)a.H, (cuuint64_t)a.W, (cuuint64_t)a.C, (cuuint64_t)images};
  cuuint64_t const strides[3] = {(cuuint64_t)a.H * 4, (cuuint64_t)a.H * a.W * 4, (cuuint64_t)a.imgStride * 4};
  cuuint32_t const box[4] = {(cuuint32_t)boxH, (cuuint32_t)boxW, 32u, 1u};
  cuuint32_t const estr[4] = {1u, 1u, 1u, 1u};
  CUresult const r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(a.ptr), dims, strides, box, estr,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return false;
  p.tma = 1; p.bh = bestBh; p.bw = bestBw; p.tilesH = vlb::ceil_div(Ho, bestBh); p.tilesW = vlb::ceil_div(Wo, bestBw);
  p.boxH = boxH; p.boxW = boxW; p.rowOff = rowOff; p.bStages = nB; p.xStages = nX;
  p.tilesM = (int)(images * p.tilesH * p.tilesW);
  *smemBytes = (size_t)nB * bBytes + pBytes + nX * xTileBytes + 1024;
  return true;
}

// Stride-1 and fully connected gradients with the gathered operand in tensor memory (p.bTiles set, p.a a convolution operand).
int launch_ts(vlb_ctx* ctx, Params& p, char const* where)
{
  bool split3 = ctx->precision == VLB_PRECISION_3XTF32;
  p.status = ctx->deviceStatus;
  p.testSwitch = ctx->testSwitch;
  // at least 120 KB, so that two CTAs (each allocating all 512 TMEM columns) never share an SM
  // filter-tile stages: as many as fit beside the running sum's patch, six at most
  if (p.splits < 1) { p.splits = 1; p.kbPerSplit = p.numKb; }
  size_t const stageBytes = (split3 ? 2u : 1u) * (size_t)p.BN * kTsRowBytes, patchBytes = p_bytes(p.BN);
  p.bStages = (int)std::min<size_t>(kTsBStages, (227 * 1024 - kTsStatic - 1024 - patchBytes) / stageBytes);
  if (p.aHi) p.bStages = std::min(p.bStages, 4);
  size_t smemBytes = (size_t)p.bStages * stageBytes + patchBytes + 1024;
  p.tilesM = vlb::ceil_div(p.M, BM); p.tilesN = vlb::ceil_div(p.N, p.BN);
  p.kbTot = p.splits * p.kbPerSplit;       // what the tile images hold per column tile
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  bool const windows = p.aHi == nullptr && plan_windows(ctx, p, &map, &smemBytes, split3);
  p.biasFirst = p.e.bias != nullptr && aligned16(p.e.bias) && p.N % 4 == 0;
  ts_divisors(p);
  if (smemBytes < 120u * 1024u) smemBytes = 120u * 1024u;
  long long const numTiles = (long long)p.tilesM * p.tilesN * p.splits;
  if (numTiles >= (1LL << 31)) return VLB_Unsupported;
  // Persistent: one CTA per SM walks the tiles, so that the pipeline never drains between tiles and a tile is stored
  // while the next one is computed.
  dim3 grid((unsigned)std::min<long long>(numTiles, ctx->smCount), 1, 1);
  cudaError_t e;
  bool const narrow = p.BN <= 64;
  auto go = [&](auto kernel) {
    e = allow_large_smem<decltype(kernel)::value>(ctx->device);
    if (e == cudaSuccess) vlb::launch(ctx->stream, decltype(kernel)::value, grid, kTsThreads, smemBytes, p, map);
  };
#define VLB_TS(split, mode, nar) go(std::integral_constant<decltype(&conv_half_kernel<split, mode, nar>), &conv_half_kernel<split, mode, nar>>{})
  if (p.aHi) {
    if (split3) { if (narrow) VLB_TS(true, 3, true); else VLB_TS(true, 3, false); }
    else        { if (narrow) VLB_TS(false, 3, true); else VLB_TS(false, 3, false); }
  } else if (split3) {
    if (windows) { if (narrow) VLB_TS(true, 1, true); else VLB_TS(true, 1, false); }
    else         { if (narrow) VLB_TS(true, 0, true); else VLB_TS(true, 0, false); }
  } else {
    if (windows) { if (narrow) VLB_TS(false, 1, true); else VLB_TS(false, 1, false); }
    else         { if (narrow) VLB_TS(false, 0, true); else VLB_TS(false, 0, false); }
  }
#undef VLB_TS
  if (e != cudaSuccess) { cudaGetLastError(); return vlb::set_error(ctx, VLB_Cuda, cudaGetErrorString(e)); }
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, where);
}

// conv_half_kernel in its row mode (kMode 2): rows whose reduction index is contiguous in memory, delivered by the 3-D tensor map `map`
// (run of 68 elements x cPer rows x 1).  p holds the tiling (cPer, tapsPerTile, tapGroups, tilesM, tilesN, splits, kbPerSplit,
// kbTot), the operand geometry, the tile images and the epilogue.
int launch_rows(vlb_ctx* ctx, Params& p, CUtensorMap const& map, char const* where)
{
  bool const split3 = ctx->precision == VLB_PRECISION_3XTF32;
  // shared memory: filter-tile stages, the running sum, the runs
  size_t const bBytes = (size_t)(split3 ? 2 : 1) * p.BN * kTsRowBytes, pBytes = p_bytes(p.BN);
  size_t const limit = 227 * 1024 - kTsStatic;
  p.bStages = 0;
  for (int nb = kTsBStages; nb >= 3 && !p.bStages; --nb)
    for (int nx = kTsXStages; nx >= 3 && !p.bStages; --nx)
      if ((size_t)nb * bBytes + pBytes + (size_t)nx * kWgStageBytes + 1024 <= limit) { p.bStages = nb; p.xStages = nx; }
  if (!p.bStages) return vlb::set_error(ctx, VLB_Unsupported, where);
  size_t smemBytes = (size_t)p.bStages * bBytes + pBytes + (size_t)p.xStages * kWgStageBytes + 1024;
  if (smemBytes < 120u * 1024u) smemBytes = 120u * 1024u;      // two CTAs (each allocating all 512 TMEM columns) never share an SM
  p.wg = 1;
  ts_divisors(p);
  p.status = ctx->deviceStatus;
  p.testSwitch = ctx->testSwitch;
  p.chanFast = 1;
  long long const numTiles = (long long)p.tilesM * p.tilesN * p.splits;
  if (numTiles >= (1LL << 31)) return VLB_Unsupported;
  dim3 grid((unsigned)std::min<long long>(numTiles, ctx->smCount), 1, 1);
  cudaError_t e;
  auto go = [&](auto kernel) {
    e = allow_large_smem<decltype(kernel)::value>(ctx->device);
    if (e == cudaSuccess) vlb::launch(ctx->stream, decltype(kernel)::value, grid, kTsThreadsRows, smemBytes, p, map);
  };
#define VLB_TSR(split) go(std::integral_constant<decltype(&conv_half_kernel<split, 2, false>), &conv_half_kernel<split, 2, false>>{})
  if (split3) VLB_TSR(true); else VLB_TSR(false);
#undef VLB_TSR
  if (e != cudaSuccess) { cudaGetLastError(); return vlb::set_error(ctx, VLB_Cuda, cudaGetErrorString(e)); }
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, where);
}

// conv_half_kernel, kMode 4 (64 images of a pixel per k-block) or 5: p holds the tiling, the chunks, the tile images and the epilogue.
int launch_images(vlb_ctx* ctx, Params& p, char const* where)
{
  bool const split3 = ctx->precision == VLB_PRECISION_3XTF32;
  size_t const stageBytes = (size_t)(split3 ? 2 : 1) * p.BN * kTsRowBytes, patchBytes = p_bytes(p.BN);
  p.bStages = 4;                                       // (what shared memory leaves over is L1, which serves the taps of a column)
  size_t const smemBytes = std::max<size_t>(p.bStages * stageBytes + patchBytes + 1024, 120u * 1024u);      // two CTAs never share an SM
  ts_divisors(p);
  p.dHo = vlb::FastDiv31(p.rowBlocks);
  p.status = ctx->deviceStatus;
  p.testSwitch = ctx->testSwitch;
  long long const numTiles = (long long)p.tilesM * p.tilesN * p.splits;
  if (numTiles >= (1LL << 31)) return VLB_Unsupported;
  dim3 const grid((unsigned)std::min<long long>(numTiles, ctx->smCount), 1, 1);
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  cudaError_t e;
  auto go = [&](auto kernel) {
    e = allow_large_smem<decltype(kernel)::value>(ctx->device);
    if (e == cudaSuccess) vlb::launch(ctx->stream, decltype(kernel)::value, grid, kTsThreads, smemBytes, p, map);
  };
#define VLB_TSI(split, mode, nar) go(std::integral_constant<decltype(&conv_half_kernel<split, mode, nar>), &conv_half_kernel<split, mode, nar>>{})
#define VLB_TSIM(mode) do { \
    if (split3) { if (p.BN <= 64) VLB_TSI(true, mode, true); else VLB_TSI(true, mode, false); } \
    else        { if (p.BN <= 64) VLB_TSI(false, mode, true); else VLB_TSI(false, mode, false); } \
  } while (0)
  if (p.gShift == 3) VLB_TSIM(4); else VLB_TSIM(5);
#undef VLB_TSIM
#undef VLB_TSI
  if (e != cudaSuccess) { cudaGetLastError(); return vlb::set_error(ctx, VLB_Cuda, cudaGetErrorString(e)); }
  VLB_LAUNCHED(ctx, 1);
  return vlb::check_launch(ctx, where);
}

// Filter gradients in planes of rows (conv_wgrad_half below) need: a tap that is a constant shift of the flattened plane (Ho == H), planes of a multiple of four
// pixels (the 16-byte strides the tensor map wants) that whole k-blocks cover with at most a third more work, channels in blocks of 32.
bool wgrad_rows_ok(ConvGeom const& g)
{
  int const taps = g.FH * g.FW, P = g.Ho * g.Wo, Pp = (P + kTsK - 1) / kTsK * kTsK;
  if (g.G != 1 || g.sy != 1 || g.sx != 1 || g.Ho != g.H || P % 4 != 0 || (Pp - P) * 4 > Pp || g.H * g.W % 4 != 0 || taps > 64 || g.FH > 32 || g.FW > 32) return false;
  if (g.C % 32 != 0 || (g.C > 128 && g.C % 128 != 0) || (g.C < 128 && 128 % g.C != 0)) return false;
  if (g.K > 4096 || (g.FH - 1) * g.dy - g.pt >= g.H || g.pt >= g.H) return false;
  return (long long)Pp * g.N < (1LL << 31) - 4096;
}

// Whether the images along the reduction (kbs k-blocks in `tiles` output tiles, 8 << gShift images in each) beat the other route, in microseconds as measured on 148 SMs:
// a k-block of a tile takes 0.7 here (0.85 with fewer than 64 images in it, whose chunks are converted as they come), 1.05 in planes of rows, 1.9 (per 64 pixels) in
// tc_gemm_kernel; the input's chunks take 8 bytes per element at 5 TB/s, the tile images 3 more than the row mode's; one launch more than there 3 (nothing with fewer than
// 64 images: the row mode's first runs arrive that much later), two more than tc_gemm_kernel with its own producers 10.
// 64 images: 3x3, 512 -> 512, 14 x 14: 190 (planes of rows 331); 256 -> 256, 56 x 56: 920 (1003); 1x1, 512 -> 128, 28 x 28: 103 (62); 13 x 13, 256 -> 384, 128
// images: 161 (tc_gemm_kernel 260).  Fewer: 3x3, 256 -> 256, 14 x 14, 8 images 48 (planes of rows 62), 16 images 56 (66), 32 images 60 (73); 512 -> 512, 7 x 7, 8 images
// 32 (tc_gemm_kernel 28), 32 images 56 (71); 1x1, 512 -> 128, 28 x 28, 32 images 78 (planes of rows 54).
bool wgrad_images_pay(vlb_ctx* ctx, ConvGeom const& g, bool rows, long long kbs, int tiles, int gShift)
{
  int const V = g.FH * g.FW * g.FC;
  double const x = (double)g.H * g.W * g.C * g.N, y = (double)g.Ho * g.Wo * g.K * g.N, perSm = 1.0 / ctx->smCount;
  long long const P = (long long)g.Ho * g.Wo;
  double const other = rows ? 1.05 * vlb::ceil_div(V, BM) * vlb::ceil_div(g.K, pick_bn(g.K)) * (double)((P + kTsK - 1) / kTsK) * g.N * perSm
                            : 1.9 * vlb::ceil_div(V, BM) * vlb::ceil_div(g.Kg, pick_bn(g.Kg)) * (double)g.G * (double)P * g.N / kTsK * perSm;
  double const perKb = gShift == 3 ? 0.7 : 0.85, launches = !rows ? 10.0 : gShift == 3 ? 3.0 : 0.0;
  return perKb * tiles * (double)kbs * perSm + (x * 8 + y * (rows ? 3 : 0)) / 5e6 + launches < other;
}

// k-blocks of a reduction over `taps` filter taps of `channels` channels.
int gen_kblocks(int taps, int channels) { return taps * vlb::ceil_div(channels, 64); }

// One contraction of conv_half_gen_kernel: the stride / pad / dilation geometry t over src, `groups` groups of chPerGroup channels
// and `cols` output columns each.
void gen_problem(Params& p, ConvGeom const& t, float const* src, int chPerGroup, int groups, int cols, int BN)
{
  conv_operand(p.a, t, src, chPerGroup * groups);
  p.a.C = chPerGroup; p.aGroup = (long long)t.H * t.W * chPerGroup;
  p.M = t.Ho * t.Wo * t.N; p.N = cols * groups; p.R = t.FH * t.FW * chPerGroup; p.a.rows = p.M;
  p.numKb = gen_kblocks(t.FH * t.FW, chPerGroup);
  p.BN = BN; p.cols = cols; p.tilesPerGroup = vlb::ceil_div(cols, BN); p.tilesN = groups * p.tilesPerGroup; p.tilesM = vlb::ceil_div(p.M, BM);
  p.splits = 1; p.kbPerSplit = p.kbTot = p.numKb;
  p.oy = p.ox = 0; p.oys = p.oxs = 1; p.outH = t.Ho; p.outW = t.Wo; p.shufY = p.shufX = 0; p.outC = cols;
}

// The part of the filter tile images' description that follows from the problem.
PrepFilters gen_prep(Params const& p, ConvGeom const& g, float const* f)
{
  PrepFilters q = {};
  q.f = f; q.BN = p.BN; q.numKb = p.numKb; q.rows = p.tilesN * p.BN; q.tilesPerGroup = p.tilesPerGroup; q.cols = p.cols;
  q.whole = 1; q.tapsH = p.a.FH; q.tapsW = p.a.FW; q.C = p.a.C; q.FH = g.FH; q.FW = g.FW;
  q.ah = q.aw = 1; q.shufY = p.shufY; q.shufX = p.shufX;
  return q;
}

// Builds the tile images of all problems (one launch) and runs them (one launch).  The problems share the tile width.
// Where the problems' tiles are too few for the chip the reductions are cut, all into the same number of ranges, and `fin` (the epilogue,
// which the problems then do not apply themselves) goes to the sum over the ranges; they cover every element of the output then
// (`covered`).  -1: the gather that splits as it goes has it (a reduction too long; no room for the chunks).
int launch_ts_gen(vlb_ctx* ctx, TsProblems& b, PrepBatch& prep, float* out, size_t nOut, vlb::SumEpilogue const& fin, bool covered, char const* where)
{
  bool const split3 = ctx->precision == VLB_PRECISION_3XTF32;
  int const BN = b.p[0].BN;
  size_t const stageBytes = (split3 ? 2u : 1u) * (size_t)BN * kTsRowBytes, patchBytes = p_bytes(BN);
  size_t total = 0, offset[kMaxTsProblems];
  long long tiles = 0;
  double work = 0;
  int splits = 1;
  {
    long long t = 0, kb = 0;
    for (int i = 0; i < b.n; ++i) { long long const ti = (long long)b.p[i].tilesM * b.p[i].tilesN; t += ti; kb += ti * b.p[i].numKb; }
    int per;
    if (covered && t < (1 << 20)) splits = split_few_tiles(ctx->smCount, (int)t, (int)(kb / t), &per, 4);
  }
  for (int i = 0; i < b.n; ++i) {
    Params& p = b.p[i];
    p.splits = splits; p.kbPerSplit = vlb::ceil_div(p.numKb, splits);
    p.numKb = p.kbTot = p.splits * p.kbPerSplit;
    prep.p[i].numKb = p.numKb;
    p.e.out = out;
    if (splits > 1) p.e.splitStride = (long long)nOut;
    else { p.e.bias = fin.bias; p.e.mask = fin.mask; }
    offset[i] = total;
    total += ts_tiles_bytes(ctx, p.tilesN * BN, BN, p.numKb);
    if (p.numKb > 32767) return -1;
    long long const t = (long long)p.tilesM * p.tilesN * p.splits;
    tiles += t;
    work += (double)t * (p.kbPerSplit + 6);
    if (t >= (1LL << 31)) return VLB_Unsupported;
  }
  // all problems gather from one tensor, which is split beforehand
  Operand const& a0 = b.p[0].a;
  int const images = (int)(b.p[0].M / ((long long)a0.Ho * a0.Wo)), channels = (int)(a0.imgStride / ((long long)a0.H * a0.W));
  long long const elements = (long long)a0.H * a0.W * vlb::ceil_div(channels, 64) * 64 * images;
  size_t const partBytes = splits > 1 ? (sizeof(float) * nOut * splits + 255) & ~(size_t)255 : 0;
  char* const ws = (char*)vlb::try_workspace(ctx, total + partBytes + chunks_bytes(ctx, elements));
  if (!ws) return -1;
  float* const part = (float*)(ws + total);
  split_chunks(ctx, b.p[0], ws + total + partBytes, images, channels);
  // CTAs per problem: one per tile when all tiles fit, else shares of the chip in proportion to the work, the rest to the longest queues
  int given = 0;
  for (int i = 0; i < b.n; ++i) {
    Params& p = b.p[i];
    long long const t = (long long)p.tilesM * p.tilesN * p.splits;
    p.ctas = tiles <= ctx->smCount ? (int)t
             : (int)std::min<long long>(t, std::max(1, (int)((double)ctx->smCount * (double)t * (p.kbPerSplit + 6) / work)));
    given += p.ctas;
  }
  while (tiles > ctx->smCount && given < ctx->smCount) {
    int worst = -1; double most = 0;
    for (int i = 0; i < b.n; ++i) {
      Params const& p = b.p[i];
      long long const t = (long long)p.tilesM * p.tilesN * p.splits;
      double const queue = (double)((t + p.ctas - 1) / p.ctas) * (p.kbPerSplit + 6);
      if (p.ctas < t && queue > most) { most = queue; worst = i; }
    }
    if (worst < 0) break;
    ++b.p[worst].ctas; ++given;
  }
  int const stages = (int)std::min<size_t>(4, (227 * 1024 - kTsStatic - 1024 - patchBytes) / stageBytes);
  for (int i = 0, beg = 0; i < b.n; ++i) {
    Params& p = b.p[i];
    p.ctaBeg = beg; beg += p.ctas;
    prep.p[i].out = ts_tiles_at(ctx, ws + offset[i], p.tilesN * BN, BN, p.numKb);
    p.bTiles = (float const*)prep.p[i].out.img; p.bExp = prep.p[i].out.exps; p.bOwn = prep.p[i].out.own;
    if (splits > 1) p.e.out = part;
    p.c64 = b.p[0].c64; p.aHi = b.p[0].aHi; p.aLo = b.p[0].aLo; p.aExp = b.p[0].aExp; p.zero = b.p[0].zero;
    p.status = ctx->deviceStatus; p.testSwitch = ctx->testSwitch; p.chanFast = 1; p.bStages = stages;
    ts_divisors(p);
    p.biasFirst = p.e.bias != nullptr && aligned16(p.e.bias) && p.cols % 4 == 0 && p.shufY == 0;
  }
  launch_prep(ctx, prep, b.n);
  size_t const smemBytes = std::max<size_t>((size_t)stages * stageBytes + patchBytes + 1024, 120u * 1024u);      // two CTAs never share an SM
  cudaError_t e;
  with_capacity(b.n, [&](auto capacity) {
    constexpr int kMax = decltype(capacity)::value;
    auto go = [&](auto kernel) {
      e = allow_large_smem<decltype(kernel)::value, 96>(ctx->device);
      if (e == cudaSuccess) vlb::launch(ctx->stream, decltype(kernel)::value, given, kTsThreads, smemBytes, first_problems<kMax>(b));
    };
#define VLB_TSG(split, nar) go(std::integral_constant<decltype(&conv_half_gen_kernel<split, nar, kMax>), &conv_half_gen_kernel<split, nar, kMax>>{})
    if (split3) { if (BN <= 64) VLB_TSG(true, true); else VLB_TSG(true, false); }
    else        { if (BN <= 64) VLB_TSG(false, true); else VLB_TSG(false, false); }
#undef VLB_TSG
  });
  if (e != cudaSuccess) { cudaGetLastError(); return vlb::set_error(ctx, VLB_Cuda, cudaGetErrorString(e)); }
  VLB_LAUNCHED(ctx, 1);
  int const rc = vlb::check_launch(ctx, where);
  return rc || splits == 1 ? rc : vlb::sum_parts(ctx, out, part, nOut, nOut, splits, fin);
}

}  // namespace

namespace vlb {

// Filter gradient with the images along the reduction: any stride, dilation, padding, plane and channel count, filter groups.  What it needs is images:
// a k-block holds 8 << gShift of them at 8 >> gShift rows, and what is missing to a whole number of either is work for nothing.  -1: not eligible or not worth it.
int conv_wgrad_images(vlb_ctx* ctx, ConvGeom const& g, float* dF, float* db, float const* X, float const* dY, bool* dbDone, bool rows)
{
  int const taps = g.FH * g.FW, V = taps * g.FC;
  int gShift = 0;
  long long least = -1;
  for (int s = 0; s <= 3; ++s) {
    // (14 : 17, a k-block of split chunks : one of chunks that are converted as they come; 3x3, 256 -> 256, 14 x 14 maps of 100 images: 122 us in blocks of 64 images, 145 of 8)
    long long const images = (long long)ceil_div(g.N, 8 << s) * (8 << s), rows = (long long)ceil_div(g.Ho, 8 >> s) * (8 >> s), cost = images * rows * (s == 3 ? 14 : 17);
    if (least < 0 || cost <= least) { least = cost; gShift = s; }
  }
  if (taps > 4096 || g.K > 4096 || (g.G > 1 && g.Kg < 16)) return -1;
  Params p = {};
  int const units = taps * ceil_div(g.FC, 32);
  p.BN = pick_bn(g.Kg);
  p.tilesPerGroup = ceil_div(units, 4); p.tilesM = g.G * p.tilesPerGroup; p.tilesN = ceil_div(g.Kg, p.BN); p.cols = g.Kg;
  p.gShift = gShift; p.rowBlocks = ceil_div(g.Ho, 8 >> gShift); p.nGroups = ceil_div(g.N, 8 << gShift); p.channels = g.C;
  long long const kbs = (long long)p.nGroups * g.Wo * p.rowBlocks;
  if (kbs >= (1LL << 24) || (!(ctx->testSwitch & 16) && !wgrad_images_pay(ctx, g, rows, kbs, p.tilesM * p.tilesN, gShift))) return -1;
  p.splits = pick_wg_splits(ctx->smCount, p.tilesM * p.tilesN, (int)kbs, &p.kbPerSplit, 24);
  p.kbTot = p.splits * p.kbPerSplit; p.numKb = p.kbTot;
  conv_operand(p.a, g, X, g.C);
  p.a.C = g.FC;
  p.M = V; p.N = g.G * p.tilesN * p.BN; p.R = (int)((long long)g.Ho * g.Wo * g.N); p.a.rows = V; p.wg = 2;
  size_t const nF = (size_t)V * g.K;
  if ((long long)nF * p.splits >= (1LL << 31)) return -1;
  // (a block of the input's preparation per group of images on gridDim.y)
  if ((gShift == 3 ? p.nGroups : p.nGroups << gShift) > kMaxGridY) return -1;
  // scratch: tile images, partial results, the input's chunks (64 images per k-block: split, with exponents), the bias gradient's partial sums
  int const imgGroups = p.nGroups << gShift, tiles = g.G * p.tilesN;
  long long const chunks = (long long)imgGroups * g.H * g.W * g.C;
  bool const split3 = ctx->precision == VLB_PRECISION_3XTF32;
  size_t const partBytes = p.splits > 1 ? ((sizeof(float) * nF * p.splits + 255) & ~(size_t)255) : 0;
  size_t const chunkBytes = (size_t)chunks * (split3 || gShift < 3 ? 32 : 16);
  size_t const expBytes = gShift == 3 ? ((size_t)p.nGroups * g.W * g.H * g.C + 511) & ~(size_t)255 : 0;
  // (one pixel per k-block: the columns of a plane are one long one, whose octets lie on 32-byte boundaries where P does)
  int const oH = gShift == 3 ? g.Ho * g.Wo : g.Ho, oW = gShift == 3 ? 1 : g.Wo, oBlocks = gShift == 3 ? oH : p.rowBlocks;
  int const octets = ceil_div(p.kbTot, oBlocks) * ceil_div(oH, 8);
  int const fBlocks = tiles * std::max(p.BN / 32, 1);
  int const gx = std::max(1, std::min(4 * ctx->smCount / fBlocks, octets));
  size_t const extraBytes = partBytes + ((chunkBytes + 255) & ~(size_t)255) + 256 + expBytes + (db ? sizeof(float) * (size_t)gx * fBlocks * 32 : 0);
  if (!try_workspace(ctx, ts_tiles_bytes(ctx, p.N, p.BN, p.numKb) + extraBytes)) return -1;      // (the other kernels need no copy of the input)
  TileOut out;
  float* at = nullptr;
  ProfScope prof(ctx, kProfWgrad);
  prof.rec.flops = 2.0 * (double)V * (double)g.Kg * g.G * (double)p.R;
  if (!ts_tiles(ctx, p, extraBytes, &out, &at)) return ctx->lastError;
  float* const part = at;
  uint4* const hi = (uint4*)((char*)at + partBytes);
  uint4* const zero = (uint4*)((char*)hi + ((chunkBytes + 255) & ~(size_t)255));
  int8_t* const exps = (int8_t*)zero + 256;
  float* const dbPart = db ? (float*)((char*)exps + expBytes) : nullptr;
  unsigned* const tickets = (unsigned*)((char*)ctx->deviceStatus + 256);
  p.aHi = hi; p.aLo = chunks; p.aExp = exps; p.zero = zero;
  int const cBlocks = ceil_div(g.C, 32), HW = g.H * g.W;
  dim3 const gridX((unsigned)(ceil_div(HW, 8) * cBlocks), (unsigned)(gShift == 3 ? p.nGroups : imgGroups), 1), gridY((unsigned)gx, (unsigned)fBlocks, 1);
  if (gShift < 3)  vlb::launch(ctx->stream, gather_images_kernel, gridX, 256, 0, (float4*)hi, chunks, zero, X, HW, g.C, g.N, cBlocks);
  else if (split3) vlb::launch(ctx->stream, split_images_kernel<true>, gridX, 256, 0, hi, chunks, exps, zero, X, HW, g.C, g.N, cBlocks);
  else             vlb::launch(ctx->stream, split_images_kernel<false>, gridX, 256, 0, hi, chunks, exps, zero, X, HW, g.C, g.N, cBlocks);
#define VLB_IM(split, G8) vlb::launch(ctx->stream, prep_image_tiles_kernel<split, G8>, gridY, 256, 0, out, dY, oH, oW, g.N, g.K, g.Kg, p.tilesN, p.BN, p.nGroups, oBlocks, p.kbTot, octets, db, dbPart, tickets)
#define VLB_IMS(G8) do { if (split3) VLB_IM(true, G8); else VLB_IM(false, G8); } while (0)
  if (gShift == 3) VLB_IMS(8); else if (gShift == 2) VLB_IMS(4); else if (gShift == 1) VLB_IMS(2); else VLB_IMS(1);
#undef VLB_IMS
#undef VLB_IM
  VLB_LAUNCHED(ctx, 2);
  *dbDone = db != nullptr;
  p.e = Epilogue{};
  p.e.out = p.splits > 1 ? part : dF; p.e.splitStride = p.splits > 1 ? (long long)nF : 0; p.e.inMult = 1.f; p.e.P = V; p.e.Ktot = g.K;
  int const rc = launch_images(ctx, p, "conv_wgrad_images");
  if (rc) return rc;
  return p.splits > 1 ? sum_parts(ctx, dF, part, nF, nF, p.splits) : VLB_Success;
}

// Filter gradient of a convolution: with the images along the reduction where that pays, else, for a stride-1 convolution whose output has the input's height, through
// the row mode: rows (tap, channel) in tensor memory, dY as tile images.  Returns -1 when the layer is not eligible (the
// caller then takes tc_gemm_kernel), else an error code.
int conv_wgrad_half(vlb_ctx* ctx, ConvGeom const& g, float* dF, float* db, float const* X, float const* dY, bool* dbDone)
{
  if (ctx->testSwitch & 4) return -1;
  bool const rows = wgrad_rows_ok(g) && aligned16(X) && aligned16(dY);
  {
    int const rc = conv_wgrad_images(ctx, g, dF, db, X, dY, dbDone, rows);
    if (rc >= 0 || !rows) return rc;
  }
  int const taps = g.FH * g.FW, P = g.Ho * g.Wo, HW = g.H * g.W;
  int const Pp = (P + kTsK - 1) / kTsK * kTsK;       // planes are padded to whole k-blocks, so that no k-block straddles two images
  int const V = taps * g.C;
  long long const R = (long long)P * g.N;
  Params p = {};
  p.cPer = std::min(g.C, 128); p.tapsPerTile = 128 / p.cPer; p.tapGroups = vlb::ceil_div(taps, p.tapsPerTile);
  p.M = V; p.N = g.K; p.R = (int)R;
  p.BN = pick_bn(p.N);
  p.tilesM = p.tapGroups * (g.C / p.cPer); p.tilesN = vlb::ceil_div(p.N, p.BN);
  if (vlb::ceil_div(g.K, p.BN) * p.BN > 65535) return -1;
  int const numKb = (int)((long long)Pp * g.N / kTsK);
  p.plane = Pp;
  p.splits = pick_wg_splits(ctx->smCount, p.tilesM * p.tilesN, numKb, &p.kbPerSplit, 24);
  p.kbTot = p.splits * p.kbPerSplit;               // the tile images are padded with zeros to whole ranges
  p.numKb = p.kbTot;
  conv_operand(p.a, g, X, g.C);
  p.a.rows = V;
  size_t const nF = (size_t)V * g.K;
  if ((long long)nF * p.splits >= (1LL << 31)) return -1;
  size_t const partBytes = p.splits > 1 ? ((sizeof(float) * nF * p.splits + 255) & ~(size_t)255) : 0;
  CUtensorMap map;
  if (!rows_map(&map, X, HW, g.C, g.N, kWgRowWords, p.cPer)) return -1;

  ProfScope prof(ctx, kProfWgrad);      // includes the dY tile images (with the bias gradient) and the sum of the partial results
  prof.rec.flops = 2.0 * (double)V * (double)g.K * (double)R;
  float* part = nullptr;
  if (!prep_pixel_tiles(ctx, p, dY, P, g.N, partBytes, p.splits > 1 ? &part : nullptr, db)) return ctx->lastError;
  *dbDone = db != nullptr;
  p.e = Epilogue{};
  p.e.out = part ? part : dF; p.e.splitStride = part ? (long long)nF : 0; p.e.inMult = 1.f; p.e.P = V; p.e.Ktot = g.K;
  int const rc = launch_rows(ctx, p, map, "conv_wgrad_half");
  if (rc) return rc;
  return part ? vlb::sum_parts(ctx, dF, part, nF, nF, p.splits) : VLB_Success;
}

int fc_dgrad_half(vlb_ctx* ctx, ConvGeom const& g, float* dX, float const* F, float const* dY)
{
  int const V = g.FH * g.FW * g.FC;
  if ((ctx->testSwitch & 4) || V % 4 != 0 || g.K % 32 != 0 || !aligned16(F) || !aligned16(dY) || V < 128 * 16) return -1;
  Params p = {};
  p.M = V; p.N = g.N; p.R = g.K;
  ConvGeom const t = plane_geom(V, g.K, g.N);
  conv_operand(p.a, t, F, g.K);
  p.a.rows = V;
  p.BN = pick_bn(p.N);
  int const numKb = vlb::ceil_div(g.K, kTsK);
  p.splits = pick_wg_splits(ctx->smCount, vlb::ceil_div(V, BM) * vlb::ceil_div(p.N, p.BN), numKb, &p.kbPerSplit, 8);
  p.numKb = p.splits * p.kbPerSplit;
  p.chanFast = 1;
  size_t const nOut = (size_t)V * g.N;
  size_t const partBytes = p.splits > 1 ? sizeof(float) * nOut * p.splits : 0;
  ProfScope prof(ctx, kProfFc);
  prof.rec.flops = 2.0 * (double)V * (double)g.N * (double)g.K;
  // more than 128 images: several column tiles read the weights, from chunks then (256 images, V = 25088, K = 4096: 322 us -> 264, of
  // which 122 are the split, at the copy rate)
  size_t const partRoom = (partBytes + 255) & ~(size_t)255, chunkBytes = chunks_bytes(ctx, (long long)V * vlb::ceil_div(g.K, 64) * 64);
  bool const chunks = split_pays(g.K, 1, vlb::ceil_div(p.N, p.BN)) && try_workspace(ctx, ts_tiles_bytes(ctx, p.N, p.BN, p.numKb) + partRoom + chunkBytes);
  float* behind = nullptr;
  if (!prep_dense_tiles(ctx, p, dY, true, partRoom + (chunks ? chunkBytes : 0), &behind)) return ctx->lastError;      // B(n, k) = dY[k + K n]
  float* const part = p.splits > 1 ? behind : nullptr;
  if (chunks) split_chunks(ctx, p, (char*)behind + partRoom, 1, g.K);
  p.e = Epilogue{};
  p.e.out = part ? part : dX; p.e.splitStride = part ? (long long)nOut : 0; p.e.inMult = 1.f; p.e.P = V; p.e.Ktot = g.N;
  vlb::SumEpilogue epi;
  (part ? epi.mask : p.e.mask) = ctx->reluMask; ctx->maskDone = ctx->reluMask != nullptr;
  int rc = launch_ts(ctx, p, "fc_dgrad_half");
  return rc || !part ? rc : vlb::sum_parts(ctx, dX, part, nOut, nOut, p.splits, epi);
}

int fc_wgrad_half(vlb_ctx* ctx, ConvGeom const& g, float* dF, float const* X, float const* dY)
{
  int const V = g.FH * g.FW * g.FC;
  if ((ctx->testSwitch & 4) || V % 4 != 0 || g.N % 32 != 0 || !aligned16(X) || !aligned16(dY) || V < 128 * 16) return -1;
  if (V < kFineV && (long long)V * g.K < (1 << 23)) return -1;
  Params p = {};
  p.M = V; p.N = g.K; p.R = g.N;
  ConvGeom const t = plane_geom(V, g.N, g.K);
  conv_operand(p.a, t, X, g.N);
  p.a.rows = V;
  p.BN = pick_bn(p.N);
  p.numKb = vlb::ceil_div(g.N, kTsK); p.kbPerSplit = p.numKb; p.splits = 1;
  p.chanFast = 1;
  ProfScope prof(ctx, kProfFc);
  prof.rec.flops = 2.0 * (double)V * (double)g.K * (double)g.N;
  // the column tiles of the filters all read X, from chunks (eight images of an input) where the images fill blocks of 64 (V = 25088, K = 4096, 256 images:
  // 335 us -> 220; 64 images 207 -> 133, where the gradient's 411 MB take 63)
  size_t const chunkBytes = chunks_bytes(ctx, (long long)V * vlb::ceil_div(g.N, 64) * 64);
  bool const chunks = split_pays(g.N, 1, vlb::ceil_div(p.N, p.BN)) && try_workspace(ctx, ts_tiles_bytes(ctx, p.N, p.BN, p.numKb) + chunkBytes);
  float* behind = nullptr;
  if (!prep_dense_tiles(ctx, p, dY, false, chunks ? chunkBytes : 0, &behind)) return ctx->lastError;      // B(k, n) = dY[k + K n]
  if (chunks) split_chunks(ctx, p, behind, 1, g.N);
  p.e = Epilogue{};
  p.e.out = dF; p.e.inMult = 1.f; p.e.P = V; p.e.Ktot = g.K;
  return launch_ts(ctx, p, "fc_wgrad_half");
}

int conv_dgrad_gen_half(vlb_ctx* ctx, ConvGeom const& g, float* dX, float const* F, float const* dY)
{
  // dY is read once per filter tap and column tile, whichever class or column the tap belongs to
  if (!split_pays(g.Kg, g.G, g.FH * g.FW * ceil_div(g.FC, pick_bn(g.FC)))) return -1;
  struct {
    vlb_ctx* ctx; ConvGeom const& g; float* dX; float const* F; float const* dY;
    int kblocks(int taps) const { return gen_kblocks(taps, g.Kg); }
    void problem(Params& p, ConvGeom const& t, int cols, int BN) const { gen_problem(p, t, dY, g.Kg, g.G, cols, BN); }
    PrepFilters prep(Params const& p) const { return gen_prep(p, g, F); }
    int launch(TsProblems& ts, PrepBatch& prep, SumEpilogue const& fin, bool covered) const
    { return launch_ts_gen(ctx, ts, prep, dX, (size_t)g.H * g.W * g.C * g.N, fin, covered, "conv_dgrad_gen_half"); }
  } const route{ctx, g, dX, F, dY};
  return dgrad_forms<PrepBatch>(ctx, g, dX, route);
}

// Data gradient of a stride-1 convolution: dX = conv(dY, flipped and transposed filters) with padding (F-1)*dilate - pad.  -1: not eligible.
int conv_dgrad_half(vlb_ctx* ctx, ConvGeom const& g, float* dX, float const* F, float const* dY)
{
  ConvGeom t = g;
  t.H = g.Ho; t.W = g.Wo; t.C = g.K; t.FC = g.K; t.K = g.C; t.Ho = g.H; t.Wo = g.W;
  t.pt = (g.FH - 1) * g.dy - g.pt; t.pl = (g.FW - 1) * g.dx - g.pl;
  Params p = {};
  conv_operand(p.a, t, dY, g.K);
  if (!p.a.fast || g.K % 32 != 0) return -1;
  long long const M = (long long)g.H * g.W * g.N;
  p.M = (int)M; p.N = g.C; p.R = g.FH * g.FW * g.K;
  p.a.rows = p.M;
  p.BN = pick_bn(p.N);
  p.chanFast = 1;
  ProfScope prof(ctx, kProfDgrad);
  prof.rec.flops = 2.0 * (double)M * (double)g.C * (double)p.R;
  p.numKb = ceil_div(p.R, kTsK);
  p.splits = split_few_tiles(ctx->smCount, ceil_div(p.M, BM) * ceil_div(p.N, p.BN), p.numKb, &p.kbPerSplit, 4);
  p.numKb = p.splits * p.kbPerSplit;
  size_t const nOut = (size_t)p.M * g.C;
  float* part = nullptr;
  if (!prep_flipped_tiles(ctx, p, F, g, p.splits > 1 ? sizeof(float) * nOut * p.splits : 0, &part)) return ctx->lastError;
  p.e = Epilogue{}; p.e.out = dX; p.e.inMult = 1.f; p.e.P = g.H * g.W; p.e.Ktot = g.C;
  ctx->maskDone = ctx->reluMask != nullptr; ctx->biasDone = true;
  if (p.splits == 1) { p.e.mask = ctx->reluMask; p.e.bias = ctx->dgradBias; return launch_ts(ctx, p, "conv_dgrad_half"); }
  SumEpilogue epi;
  epi.mask = ctx->reluMask; epi.bias = ctx->dgradBias; epi.P = p.e.P; epi.K = g.C;
  p.e.out = part; p.e.splitStride = (long long)nOut;
  int const rc = launch_ts(ctx, p, "conv_dgrad_half");
  return rc ? rc : sum_parts(ctx, dX, part, nOut, nOut, p.splits, epi);
}

cudaError_t half_set_wait_limit(long long cycles, cudaStream_t stream)
{
  long long const v = cycles == 0 ? kWaitCycles : cycles;
  return cudaMemcpyToSymbolAsync(gWaitCycles, &v, sizeof(v), 0, cudaMemcpyHostToDevice, stream);
}

}  // namespace vlb
