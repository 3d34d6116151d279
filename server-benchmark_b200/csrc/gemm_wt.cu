// AWQ GEMM with the dequantised weights in tensor memory, one tile per pair of CTAs (any M).
//
//   D[n, m] = sum_k W[k, n] * x[m, k]          (the transposed product)
//
// The weights are the A operand of tcgen05.mma.cta_group::2.kind::f16 (M = 256 weight columns, 128
// per CTA, x K = 16) and live in TMEM: conversion warps take the packed words from shared memory
// with ldmatrix.trans, dequantise them in registers to (q - z) * s in fp16 and write the fragments
// with tcgen05.st.16x128b.  The activations are the B operand (up to 256 tokens, K-major, 128-byte
// swizzle) exactly as TMA delivers them, half of the tokens in each CTA's shared memory.
//
// Why this split: per 128-row stage a CTA moves 8 KB of packed words in and out of shared memory and
// N / 2 tokens x 256 B in and out (80 KB at N = 256 against 1024 tensor cycles), so shared memory
// does not bound it; N follows the tokens that are there (multiples of 16), so padding costs no
// tensor time; ldmatrix.trans pairs the rows (k, k + 1) of a halfword column in the load itself,
// which leaves 1.7 instructions per weight (AND-OR, subtract, scale, a shift for every second
// nibble), 270 issue slots per stage and scheduler.  One CTA per SM, persistent over its tiles:
// conversion of the next tile runs while the epilogue drains the last one.
//
// Warp roles (736 threads, mbarrier rings between them):
//   0 - 15  conversion   warp (q, team): TMEM lane quarter q, stages u = team (mod 4)
//                        raw_full -> a_full, raw_empty
//   16 - 19 epilogue     TMEM -> registers -> output                              d_full -> d_empty
//   20      MMA issue    leader CTA only: one converged warp, elected lane
//                        x_full, a_full, d_empty -> mma_done, d_full
//   21      TMA          packed words of this CTA's 128 columns                   raw_empty -> raw_full
//   22      TMA          this CTA's half of the tokens, completing on the leader  x_empty -> x_full
//
// Work: tiles of 256 columns x `nt` tokens.  Strided: pair p takes the whole tiles p, p + P, ...
// Chunked: one contiguous range of the (tile, stage) list per pair, shared tiles handed over
// (handover.cuh).  The sum is taken in pair order: results do not depend on timing.
// SPLIT: tiles few enough for one wave of clusters.  The 2 to 8 pairs of a cluster share a tile, or three pairs two
// tiles, by even ranges of units; each pair sums some of the tile's eights of tokens, and the others store their parts of
// those into its shared memory (st.async, counted by an mbarrier).  A tile handed over through scratch cost 12 500 cycles
// from the MMAs' end at 112 tokens (helper: 4700 until its flag is up, finisher: 7000 for collection, sum and stores),
// this 4600: 1400 to send, 700 under way, 2000 for the sum and the stores of a pair's share, 500 to the exit.  More warps do not
// shorten it (the stores' path does not), nor does a rehearsal of the cold code.  us, ranges -> clusters (pairs):
//   8192 x 1280 M 48 10.1 -> 6.1 (5), M 300 17.2 -> 12.4 (3); 8192 x 5120 M 100 19.1 -> 14.4 (3); 4096 x 4096 M 77
//   groups of 64 12.1 -> 8.9 (2); 8192 x 8192 M 100 20.2 -> 16.9 (2), M 150 24.2 -> 21.1 (2); 8192 x 10240 M 100 23.4 ->
//   21.8 (3 for two tiles); 16384 x 2048 M 64 16.6 -> 12.6 (5).
// Prologue: tensor memory is asked for first, the warp of the packed words waits for nobody, a conversion warp's first
// scales are on their way before anything is waited for, and the cluster barrier is awaited only where a CTA first reaches
// into the other.  In a kernel that starts when the one before it has left the GPU the first MMAs wait for the first
// conversion, 7400 cycles from the start before, some 1000 less now: 1024 x 8192 M 40 4.85 -> 4.5 us, router + experts of
// 128 x 2048 x 768, top-8, 600 tokens 134.6 -> 123.0.
// The cut of a call (tokens of a tile, units of a range) is the one of the least estimated time
// (wt_cost).  Against tiles of up to 256 tokens that were always split, and partial tiles read with plain
// loads: 8192 x 1280 at M 250 38.5 -> 14.4 us, 8192 x 7424 at M 250 50 -> 28, at M 100 26.5 -> 20.6,
// 1024 x 8192 at M 24 8.1 -> 4.6, 1792 x 1984 at M 100 17.9 -> 6.4.
//
// MODE 0 is the dense linear.  MODE 1 / 2 are the grouped expert GEMMs of a fused-MoE layer over the
// tile table that moe_gather_kernel wrote: entry (expert, first row, rows) of the permuted list.
//   MODE 1  gate_up: each CTA holds 64 gate columns (lane quarters 0, 1) and the matching 64 up columns
//           (quarters 2, 3); epilogue act[pos, c] = silu(gate) * up.
//   MODE 2  down: epilogue y[pos, c] = routed weight * D, in permuted order, so that a row is rounded once
//           and what is rounded is the weighted row: D alone may lie outside the range of fp16.
//
// WIDE is the kernel of tiles with one accumulator, more than 128 tokens, that no pair shares: its epilogue goes
// through shared memory (wt_epilogue_wide).  That is the faster way also where a pair has one tile and no next tile hides
// its stores, though the ring of packed words is down from 12 stages to 4 at 256 tokens; from registers with 12 stages:
// 8192 x 8192 at M 264 31.4 us against 31.2, 4096 x 11040 at M 150 18.3 / 18.0, 1024 x 8192 at M 264 9.4 / 9.1, M 394 on
// 1024 x 5120 9.15 / 8.8; 25 shapes, none the other way round by more than its runs differ.
//
// TMEM columns: accumulators first, then A[slots][8 steps][8], 64 columns a slot.  With as many slots as teams a team waits
// for the MMAs of its own last unit; two more take that wait out of its loop.  Up to 64 tokens there are two accumulators and
// six slots.  Up to 128, two accumulators leave four slots; one accumulator and six slots gain on every unit, and lose at
// every tile that a CTA ends before another one, whose MMAs wait for the epilogue (wt_one_accumulator).  They are taken in
// clusters with one tile (4096 x 4096 M 77 7.8 -> 7.3 us) and in ranges with enough units between two ends of tiles.  Whole
// tiles in turn, the grouped ones too, keep two.
// Lane 32 q + 8 i + g holds column 8 (4 q + g / 2) + 2 i + g % 2 of the CTA's 128.
// All mbarrier and flag waits are bounded (tc_ptx.cuh).
//
// Measured (B200, K x N, against one CTA per tile with two A stages and 64 / 128 fixed tokens):
//   8192 x 59136   M 100: 123.6 -> 94.9 us (cool; 115 in a long loop); 29568 x 8192   M 100: 70 -> 54 us; the four linears
//   of a layer (8192 x 10240, 8192 x 8192, 8192 x 59136, 29568 x 8192) against weights dequantised into shared memory:
//   M 1000 1694 -> 1448 us, M 4096 6522 -> 5749 (1.25 PFLOP/s in a long loop, where the 1 kW limit holds the
//   clock near 1.2 GHz); router + experts, 128 experts of 2048 x 768, top-8, 2500 tokens: 507 -> 282 us.
// What bounds it: at M >= 256 the tensor pipe under the power limit; below, the conversion and, on the long layers,
// the power limit.  A unit took 630 cycles at M = 24 and at M = 100, now ~510.  The arithmetic is 270 of them (sub and mul
// of f16x2 take two cycles a warp and scheduler; a loop of the conversion alone runs at 300), but a conversion warp
// spent 2500 cycles on one of its own: half of that it waited for an instruction, a slot to issue, a branch or the
// store port.  What helps is less of each: fragments of 32 rows at a time, one index for zero points and scales, so
// that no register spills into the loop, and stores of the cheaper shape took 8192 x 59136 from 87.8 to 84.5 us at
// M = 24 and 122.4 to 118.5 at M = 100; one wait per unit instead of two, arrivals without a branch and load warps
// that stay converged to 80.7 and 114.8; router + experts of 128 x 2048 x 768, top-8, 1024 tokens 173 to 163.
// Units of twice the K, more load warps, a shorter loop (two halves in turn: 10 % slower) and longer suspended waits
// changed nothing or lost.
#include "common.cuh"
#include "cut_cache.h"
#include "handover.cuh"
#include "tc_ptx.cuh"

namespace awq {

namespace {

using namespace tc;
using handover::Work;

constexpr int kWtBN = 256;                    // weight columns of a pair
constexpr int kWtCols = 128;                  // of one CTA
constexpr int kWtBK = 128;                    // K rows of a stage
constexpr int kWtRawBytes = kWtBK * kWtCols / 2;
constexpr int kWtTeams = 4;
constexpr int kWtCvWarps = 16, kWtEpiWarps = 4;
constexpr int kWtEpiWarp0 = kWtCvWarps;
constexpr int kWtIssueWarp = kWtEpiWarp0 + kWtEpiWarps;
constexpr int kWtRawWarp = kWtIssueWarp + 1, kWtXWarp = kWtRawWarp + 1;
constexpr int kWtThreads = 32 * (kWtXWarp + 1);  // 736
constexpr int kWtTmemCols = 512;
constexpr int kWtMaxRaw = 16, kWtMaxX = 8;    // ring depths the barrier block has room for
constexpr int kWtPartRing = 8, kWtPartBytes = 32 * 32 * 4;  // per epilogue warp: 32 tokens x 32 columns
constexpr int kWtBarBytes = 1024;
static_assert(8 * (2 * kWtMaxRaw + 2 * kWtMaxX + 4 + kWtEpiWarps * kWtPartRing) <= kWtBarBytes, "barriers");
constexpr int kWtExFloats = 2 * 32 * 20;      // MODE 1: gate / up exchange of two epilogue warps
constexpr int kWtExBytes = 2 * 2 * kWtExFloats * 4;
constexpr int kWtSmemLimit = 232448 - 1024;   // dynamic shared memory less the static part
constexpr int kWtMaxPairs = 128;

// SPLIT: the tiles of a cluster and how its pairs share them.  A pair has at most two tiles, neighbours.
constexpr int kWtMaxShare = 8, kWtMaxTiles = 2;
struct WtShare {
  int pairs, tiles;                      // of a cluster; pairs 0: no SPLIT
  int recv;                              // bytes of partial sums that a CTA takes in for a tile
  short bound[kWtMaxShare + 1];          // pair i has the units [bound[i], bound[i + 1]) of the cluster's list
  signed char first[kWtMaxTiles], count[kWtMaxTiles];  // pairs that share a tile
  int recip[kWtMaxTiles];                // ceil(2^16 / count)
};

struct WtParams {
  const __half* scales;
  const uint32_t* qzeros;
  const __half* bias;
  __half* out;
  int M, N, K;
  int KT;                      // stages of a tile
  int nt;                      // tokens of a full tile, a multiple of 16
  int slabs, mtiles;           // dense: tiles = slabs * mtiles
  int chunk;                   // > 0: every pair takes this many (tile, stage) units in a row; 0: whole
                               // tiles strided
  int nraw, nx;                // ring depths; nx is 4 or 8
  int nbuf, dcols;             // accumulators in TMEM and the columns of one
  int slots, acol;             // A slots behind them (64 columns each) and the first one's column
  int xstage;                  // bytes of an x stage
  int stage_bytes;             // WIDE: of a tile's way out through shared memory
  WtShare share;               // SPLIT
  float* partial;              // [CTA][4][nt][32] partial tiles handed over
  handover::Flags flags;       // of the hand-over
  // grouped modes
  const int4* tiles;           // (expert, first row, rows, -)
  const int32_t* n_tiles;
  const float* row_weights;    // MODE 2: routed weight of every permuted row
  int half_cols;               // MODE 1: I (gate columns [0, I), up columns [I, 2 I))
};

// Tensor maps of the activations.  Grouped modes: boxes of 16, 32 .. 128 rows; dense: the boxes of a
// full tile and of the last one of a slab (a kernel's parameters are copied on every launch).
template <int MODE>
struct WtXMaps {
  static constexpr int kMaps = MODE == 0 ? 2 : 8;
  CUtensorMap map[kMaps];
};

struct WtTile {
  int slab, m0, rows, n;       // column slab, first token row, valid rows, MMA N
  int wrow0, grp0;             // first weight row / group row of the expert
};

template <int MODE, int GROUP>
__device__ __forceinline__ WtTile wt_tile(const WtParams& p, int id) {
  WtTile t;
  if (MODE == 0) {
    t.slab = id / p.mtiles;
    t.m0 = (id - t.slab * p.mtiles) * p.nt;
    t.rows = min(p.nt, p.M - t.m0);
    t.wrow0 = 0;
    t.grp0 = 0;
  } else {
    const int tt = id / p.slabs;
    t.slab = id - tt * p.slabs;
    const int4 e = __ldcg(p.tiles + tt);
    t.m0 = e.y;
    t.rows = e.z;
    t.wrow0 = e.x * p.K;
    t.grp0 = e.x * (p.K / GROUP);
  }
  t.n = (t.rows + 15) & ~15;
  return t;
}

// SPLIT: of a tile's `eights` of tokens, those that sharer i of n sums are [first(i), first(i + 1)).
__device__ __forceinline__ int wt_own_first(int eights, int n, int i) { return (i * eights + n - 1) / n; }

template <int MODE, bool WIDE, bool SPLIT>
__device__ __forceinline__ Work wt_work(const WtParams& p) {
  if constexpr (SPLIT) {
    const int cluster = blockIdx.x / (2 * p.share.pairs), pair = blockIdx.x % (2 * p.share.pairs) / 2;
    const int base = cluster * p.share.tiles * p.KT;
    return Work::range(base + p.share.bound[pair], base + p.share.bound[pair + 1], p.KT);
  }
  const int tiles = MODE == 0 ? p.slabs * p.mtiles : __ldcg(p.n_tiles) * p.slabs;
  return Work(blockIdx.x >> 1, gridDim.x >> 1, tiles, p.KT, MODE == 0 && !WIDE ? p.chunk : 0);
}

template <int ID, int COUNT>
__device__ __forceinline__ void named_barrier(int off = 0) {
  asm volatile("bar.sync %0, %1;" ::"r"(ID + off), "n"(COUNT) : "memory");
}

// Rounds eight tokens of a quarter's 32 columns, k-th of the chunk: v[h][4 k + 2 e + j] is token 8 k + 2 t + j of the
// column in TMEM lane 16 h + 8 e + g.  The four 8 x 8 matrices, transposed, leave thread (g, t) columns 8 t ..
// 8 t + 7 of token g: one 16-byte store.  (Columns on lanes, neighbours paired by shuffles and stored four bytes
// at a time, took twice the instructions: 1024 x 59136 at M 1024 144 -> 132 us, router + experts of 128 x 2048 x
// 768, top-8, at 1000 tokens 171 -> 149.)
template <int LEN>
__device__ __forceinline__ uint4 wt_round(const float (&v)[2][LEN], int k) {
  uint4 w;
  w.x = movmatrix_trans(as_u32(__floats2half2_rn(v[0][4 * k], v[0][4 * k + 1])));
  w.y = movmatrix_trans(as_u32(__floats2half2_rn(v[0][4 * k + 2], v[0][4 * k + 3])));
  w.z = movmatrix_trans(as_u32(__floats2half2_rn(v[1][4 * k], v[1][4 * k + 1])));
  w.w = movmatrix_trans(as_u32(__floats2half2_rn(v[1][4 * k + 2], v[1][4 * k + 3])));
  return w;
}
template <int K8, int LEN>
__device__ __forceinline__ void wt_store(const float (&v)[2][LEN], __half* dst, size_t pitch, int rows) {
#pragma unroll
  for (int k = 0; k < K8; ++k) {
    const uint4 w = wt_round(v, k);
    if (8 * k < rows) *reinterpret_cast<uint4*>(dst + (size_t)(8 * k) * pitch) = w;
  }
}
// Chunk of 32 tokens of a quarter of the accumulator.
__device__ __forceinline__ void wt_load_chunk(uint32_t dcol, float (&d)[2][16]) {
  tmem_ld_16x256b_x4(dcol, d[0]);
  tmem_ld_16x256b_x4(dcol + (16u << 16), d[1]);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Where an epilogue warp's part of a tile goes: this lane stores rows 0, 8, .. below `rows`.
template <int MODE>
struct WtOut {
  __half* dst;
  size_t pitch;
  int rows;
  bool inside;  // columns the output has
  // columns: dense / down 32 q of the CTA's 128; gate_up 32 (q % 2) of its 64
  __device__ __forceinline__ static int first_column(const WtTile& t, int rank, int q) {
    return MODE == 1 ? t.slab * 128 + rank * 64 + 32 * (q & 1) : t.slab * kWtBN + rank * kWtCols + 32 * q;
  }
  __device__ __forceinline__ WtOut(const WtParams& p, const WtTile& t, int rank, int q, int lane) {
    const int c = first_column(t, rank, q), width = MODE == 1 ? p.half_cols : p.N, g = lane >> 2;
    inside = c < width;
    rows = inside ? t.rows - g : 0;
    pitch = (size_t)width;
    dst = p.out + (size_t)(t.m0 + g) * width + c + 8 * (lane & 3);
  }
};
// MODE 0: the columns in TMEM lanes 8 i + g of a quarter.
__device__ __forceinline__ void wt_load_bias(const WtParams& p, int first_column, int g, float (&bias)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    bias[i] = p.bias != nullptr && first_column < p.N
                  ? load_bias(p.bias + first_column + 8 * (g >> 1) + 2 * i + (g & 1))
                  : 0.f;
}
__device__ __forceinline__ void wt_add_bias(float (&d)[2][16], const float (&bias)[4]) {
#pragma unroll
  for (int i = 0; i < 32; ++i) d[i >> 4][i & 15] += bias[2 * (i >> 4) + ((i >> 1) & 1)];
}
// MODE 1: the gate warps (q 0, 1) finish the first 16 tokens of the chunk, the up warps (q 2, 3) the other 16; each
// hands its partner through `box` the half it does not finish.
__device__ __forceinline__ void wt_glu(const float (&d)[2][16], int q, int lane, float* box, float (&o)[2][8]) {
  const bool up = q >= 2;
  float4* give = reinterpret_cast<float4*>(box + (up ? 0 : kWtExFloats / 2) + lane * 20);
  const float4* take = reinterpret_cast<const float4*>(box + (up ? kWtExFloats / 2 : 0) + lane * 20);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float* lo = &d[i >> 1][4 * (i & 1)];
    give[i] = make_float4(up ? lo[0] : lo[8], up ? lo[1] : lo[9], up ? lo[2] : lo[10], up ? lo[3] : lo[11]);
  }
  named_barrier<2, 64>(q & 1);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 v = take[i];
    const float got[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int at = 4 * (i & 1) + j;
      const float mine = up ? d[i >> 1][8 + at] : d[i >> 1][at];
      const float gt = up ? got[j] : mine, uv = up ? mine : got[j];
      o[i >> 1][at] = __fdividef(gt, 1.f + __expf(-gt)) * uv;
    }
  }
}
// MODE 2: lane l has the routed weight of token l of the chunk.
__device__ __forceinline__ void wt_weigh(float (&d)[2][16], float weight, int t4) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {  // token 8 (i / 2) + 2 t4 + i % 2
    const float w = __shfl_sync(0xffffffffu, weight, 8 * (i >> 1) + 2 * t4 + (i & 1));
    const int at = 4 * (i >> 1) + (i & 1);
    d[0][at] *= w;
    d[0][at + 2] *= w;
    d[1][at] *= w;
    d[1][at + 2] *= w;
  }
}
__device__ __forceinline__ void sts_uint4(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
__device__ __forceinline__ uint4 lds_uint4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr));
  return v;
}

// Epilogue warp q of the WIDE kernel (one accumulator, whole tiles).  The next tile's MMAs wait for the accumulator,
// so the warp first takes all of it, rounded, into shared memory and stores from there under those MMAs; a lane
// reads back what it wrote.  What made this wait long were the stores: all CTAs finish their tiles at about the same
// time, and 64 KB a CTA leave at 13 to 21 bytes a cycle and SM (256 tokens: 4900 cycles, 1900 without them).
// 768 x 2048 at M 20480 77.0 -> 64.9 us, 8192 x 8192 at M 4096 454 -> 442, 8192 x 59136 at M 1000 807 -> 776; router +
// experts of 128 x 2048 x 768, top-8, 2500 tokens 295 -> 282.  Through TMA stores, a proxy
// fence and a store for each chunk, it was slower than without shared memory (82 us for the first); and with the
// next chunk's load ahead of this one's rounding the kernel spilt registers (router + experts, 2500 tokens: 274 ->
// 311 us).
template <int MODE, int GROUP>
__device__ __forceinline__ void wt_epilogue_wide(const WtParams& p, const Work& work, uint32_t tmem, int rank, int q,
                                                 int lane, uint32_t d_full, uint32_t d_empty, float* ex,
                                                 uint32_t stage, volatile int* abort_flag) {
  const uint32_t dcol = tmem + ((uint32_t)(q * 32) << 16);
  const int g = lane >> 2, t4 = lane & 3;
  constexpr int K8 = MODE == 1 ? 2 : 4;  // eights of tokens that the warp finishes of a chunk
  d_empty = map_rank(d_empty, 0);
  stage += lane * 16;
  pdl_wait();  // orders this thread's writes after the kernel before this one
  // After a wait that gave up the loop still runs to its end, without waiting and without storing:
  // every warp then passes the same named barriers.
  bool ok = true;
  int flip = 0;
  for (int seg = 0; seg < work.segs; ++seg) {
    const WtTile t = wt_tile<MODE, GROUP>(p, work.tile_id(seg));
    float rw[MODE == 2 ? 8 : 1];  // lane l: routed weights of tokens 32 i + l
    if (MODE == 2) {
#pragma unroll
      for (int i = 0; i < 8; ++i) rw[i] = 32 * i < t.n ? __ldcg(p.row_weights + t.m0 + 32 * i + lane) : 0.f;
    }
    float bias[4];
    if (MODE == 0) wt_load_bias(p, WtOut<MODE>::first_column(t, rank, q), g, bias);
    const WtOut<MODE> out(p, t, rank, q, lane);
    if (ok) ok = mbar_wait(d_full, (uint32_t)seg & 1u, abort_flag, 38);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    uint32_t to = stage;
    for (int c0 = 0; c0 < t.n; c0 += 32) {
      float d[2][16];
      wt_load_chunk(dcol + c0, d);
      if (c0 + 32 >= t.n) {  // the accumulator is in registers: the next tile may start
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && seg + 1 < work.segs) mbar_arrive_cluster(d_empty);
      }
      if constexpr (MODE == 1) {
        float o[2][8];
        wt_glu(d, q, lane, ex + ((q & 1) * 2 + flip) * kWtExFloats, o);
        flip ^= 1;
#pragma unroll
        for (int k = 0; k < K8; ++k) sts_uint4(to + k * 512, wt_round(o, k));
      } else {
        if (MODE == 0) wt_add_bias(d, bias);
        if constexpr (MODE == 2) {
          wt_weigh(d, rw[0], t4);
#pragma unroll
          for (int i = 0; i < 7; ++i) rw[i] = rw[i + 1];
        }
#pragma unroll
        for (int k = 0; k < K8; ++k) sts_uint4(to + k * 512, wt_round(d, k));
      }
      to += K8 * 512;
    }
    const int rows = ok ? out.rows : 0, pieces = (t.n + 31) / 32 * K8;
#pragma unroll 4
    for (int i = 0; i < pieces; ++i) {
      const int m = MODE == 1 ? 32 * (i >> 1) + 16 * (q >> 1) + 8 * (i & 1) : 8 * i;
      const uint4 v = lds_uint4(stage + i * 512);
      if (m < rows) *reinterpret_cast<uint4*>(out.dst + (size_t)m * out.pitch) = v;
    }
  }
}

// Epilogue warp q of the SPLIT kernel: pairs of a cluster share a tile, and each sums some of its eights of tokens.  First
// the parts that others sum are stored into their shared memory (the CTA of the same rank), for all segments; then the
// own ones are added up in the pairs' order.  Every index is settled, and the bias fetched, while the MMAs run: the warp
// has nothing else to do then, and afterwards each division costs 200 cycles.
struct WtSplitSegment {
  uint32_t dcol;               // its accumulator
  uint32_t base;               // partial sums that this warp takes in, or puts into another CTA at the same place:
  int step;                    // [eights of the CTA that sums][other sharers], bytes of the inner dimension
  uint32_t d_full, full;       // barriers
  int first, n, me;            // sharers: the first pair, their number, this one
  int eights, recip;
  int column;                  // first one of the warp
  float bias[4];               // loaded after pdl_wait
  __half* dst;
  int rows;
  __device__ __forceinline__ int own_first(int i) const { return ((i * eights + n - 1) * recip) >> 16; }
};
template <int GROUP>
__device__ __forceinline__ WtSplitSegment wt_split_segment(const WtParams& p, const Work& work, int seg, uint32_t tmem,
                                                           int rank, int q, int lane, uint32_t d_full0, uint32_t recv,
                                                           uint32_t recv_full) {
  WtSplitSegment f;
  const int cluster = blockIdx.x / (2 * p.share.pairs), pair = blockIdx.x % (2 * p.share.pairs) / 2;
  const int tile = work.tile_id(seg), lt = tile - cluster * p.share.tiles, buf = seg & (p.nbuf - 1);
  const WtTile t = wt_tile<0, GROUP>(p, tile);
  f.eights = t.n / 8;
  f.first = p.share.first[lt];
  f.n = p.share.count[lt];
  f.recip = p.share.recip[lt];
  f.me = pair - f.first;
  f.step = (f.n - 1) * 1024;
  f.base = recv + (lt & 1) * p.share.recv + q * f.own_first(1) * f.step + lane * 16;
  f.full = recv_full + 8 * (lt & 1);
  f.d_full = d_full0 + 8 * buf;
  f.dcol = tmem + ((uint32_t)(q * 32) << 16) + buf * p.dcols;
  f.column = WtOut<0>::first_column(t, rank, q);
  const WtOut<0> out(p, t, rank, q, lane);
  f.dst = out.dst;
  f.rows = out.rows;
  return f;
}
template <int GROUP>
__device__ __forceinline__ void wt_epilogue_split(const WtParams& p, const Work& work, uint32_t tmem, int rank, int q,
                                                  int lane, uint32_t d_full0, uint32_t recv, uint32_t recv_full,
                                                  volatile int* abort_flag) {
  WtSplitSegment s0 = wt_split_segment<GROUP>(p, work, 0, tmem, rank, q, lane, d_full0, recv, recv_full);
  WtSplitSegment s1 = s0;
  if (work.segs > 1) s1 = wt_split_segment<GROUP>(p, work, 1, tmem, rank, q, lane, d_full0, recv, recv_full);
  const size_t pitch = (size_t)p.N;
  pdl_wait();  // orders this thread's writes after the kernel before this one, which may have written the bias
  wt_load_bias(p, s0.column, lane >> 2, s0.bias);
  wt_load_bias(p, s1.column, lane >> 2, s1.bias);
  bool ok = true;
#pragma unroll 1
  for (int seg = 0; seg < work.segs; ++seg) {
    const WtSplitSegment f = seg == 0 ? s0 : s1;
    if (ok) ok = mbar_wait(f.d_full, 0, abort_flag, 38);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    int e = 0;
    // a CTA that gave up sends nothing: who sums waits in vain, and stores nothing
#pragma unroll 1
    for (int to = ok ? 0 : f.n; to < f.n; ++to) {
      const int end = f.own_first(to + 1);
      if (to != f.me) {
        const uint32_t cta = 2 * (f.first + to) + rank, bar = map_rank(f.full, cta);
        uint32_t dst = map_rank(f.base + (f.me - (f.me > to)) * 1024, cta);
#pragma unroll 1
        for (; e < end; e += 2) {
          float d[2][8];
          tmem_ld_16x256b_x2(f.dcol + 8 * e, d[0]);
          tmem_ld_16x256b_x2(f.dcol + (16u << 16) + 8 * e, d[1]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          st_async_v4(dst, &d[0][0], bar);
          st_async_v4(dst + 512, &d[1][0], bar);
          dst += f.step;
          if (e + 1 < end) {
            st_async_v4(dst, &d[0][4], bar);
            st_async_v4(dst + 512, &d[1][4], bar);
            dst += f.step;
          }
        }
      }
      e = end;
    }
  }
#pragma unroll 1
  for (int seg = 0; seg < work.segs; ++seg) {
    const WtSplitSegment f = seg == 0 ? s0 : s1;
    const int own0 = f.own_first(f.me), own1 = f.own_first(f.me + 1);
    if (ok && f.n > 1 && own1 > own0) ok = mbar_wait_cluster(f.full, 0, abort_flag, 40);
    ok = __all_sync(0xffffffffu, ok);
    const int rows = ok ? f.rows : 0;
    uint32_t src = f.base;
    __half* dst = f.dst + (size_t)(8 * own0) * pitch;
#pragma unroll 1
    for (int e = own0; e < own1; e += 2) {
      float d[2][8];
      tmem_ld_16x256b_x2(f.dcol + 8 * e, d[0]);
      tmem_ld_16x256b_x2(f.dcol + (16u << 16) + 8 * e, d[1]);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (e + k >= own1) break;
        float y[2][4] = {};
#pragma unroll 1
        for (int from = 0; from < f.n; ++from) {
          float4 lo = make_float4(d[0][4 * k], d[0][4 * k + 1], d[0][4 * k + 2], d[0][4 * k + 3]);
          float4 hi = make_float4(d[1][4 * k], d[1][4 * k + 1], d[1][4 * k + 2], d[1][4 * k + 3]);
          if (from != f.me) {
            lo = lds_float4(src);
            hi = lds_float4(src + 512);
            src += 1024;
          }
          y[0][0] += lo.x;
          y[0][1] += lo.y;
          y[0][2] += lo.z;
          y[0][3] += lo.w;
          y[1][0] += hi.x;
          y[1][1] += hi.y;
          y[1][2] += hi.z;
          y[1][3] += hi.w;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) y[j >> 2][j & 3] += f.bias[2 * (j >> 2) + ((j >> 1) & 1)];
        const uint4 w = wt_round(y, 0);
        if (8 * (e + k) < rows) *reinterpret_cast<uint4*>(dst) = w;
        dst += 8 * pitch;
      }
    }
  }
}

// Epilogue warp q: TMEM lane quarter q of every segment of the pair's work.
template <int MODE, int GROUP>
__device__ __forceinline__ void wt_epilogue(const WtParams& p, const Work& work, uint32_t tmem,
                                            int rank, int q, int lane, uint32_t d_full0,
                                            uint32_t d_empty0, float* ex, uint32_t part_ring,
                                            uint32_t part_full, volatile int* abort_flag) {
  const uint32_t lane_q = (uint32_t)(q * 32) << 16;
  const int t4 = lane & 3;
  const uint32_t d_empty_leader = map_rank(d_empty0, 0);
  pdl_wait();  // orders this thread's writes after the kernel before this one
  // After a wait that gave up the loop still runs to its end, without waiting and without storing:
  // every warp then passes the same named barriers.
  bool ok = true;
  int flip = 0;
  for (int seg = 0; seg < work.segs; ++seg) {
    const WtTile t = wt_tile<MODE, GROUP>(p, work.tile_id(seg));
    const int buf = seg & (p.nbuf - 1);
    const bool handover = MODE == 0 && work.k_end(seg) < p.KT;  // another pair holds the tile's last stage
    // MODE 2: lane l has the routed weights of tokens 32 i + l of the tile (128 at most), all fetched ahead of the
    // MMAs' end
    float rw[MODE == 2 ? 4 : 1];
    if (MODE == 2) {
#pragma unroll
      for (int i = 0; i < 4; ++i) rw[i] = 32 * i < t.n ? __ldcg(p.row_weights + t.m0 + 32 * i + lane) : 0.f;
    }
    // where the output goes: settled ahead of the MMAs' end as well
    const WtOut<MODE> out(p, t, rank, q, lane);
    float bias[4];
    if (MODE == 0) wt_load_bias(p, WtOut<MODE>::first_column(t, rank, q), lane >> 2, bias);
    // CTAs whose partial tiles are added: blockIdx.x - 2 gather .. blockIdx.x - 2
    const int gather = MODE == 0 ? work.helpers(seg) : 0;
    if (ok) ok = mbar_wait(d_full0 + 8 * buf, (uint32_t)(p.nbuf == 2 ? seg >> 1 : seg) & 1u, abort_flag,
                          38);
    if (MODE == 0 && ok)
      for (int c = 1 + lane; c <= gather; c += 32) {
        uint32_t polls = 0;
        while (!p.flags.raised(blockIdx.x - 2 * c, q)) {
          if (++polls >= kSpinLimit || *abort_flag) {
            *abort_flag = 1;
            atomicCAS(&g_tc_status, 0, 39);
            ok = false;
            break;
          }
        }
        p.flags.lower(blockIdx.x - 2 * c, q);
      }
    ok = __all_sync(0xffffffffu, ok);
    __syncwarp();  // what a lane acquired holds for the warp's reads of the partial tiles
    tc_fence_after();
    const uint32_t dcol = tmem + lane_q + buf * p.dcols;
    const int rows = ok ? out.rows : 0;
    // Partial tiles handed over come through a ring in the packed words' and tokens' stages, which the
    // pair is done with (the tile it finishes for others is its last), 32 tokens of a CTA at a time: a
    // load that waits for L2 once per 32 tokens and CTA took 3.2 us per CTA at 128 tokens.
    const int pieces = gather * ((t.n + 31) / 32);
    int piece = 0;
    auto load_part = [&](int i) {
      const int c = i / gather, from = blockIdx.x - 2 * (gather - (i - c * gather));
      const uint32_t bytes = (uint32_t)min(32, t.n - 32 * c) * 128;
      const uint32_t bar = part_full + 8 * (i & (kWtPartRing - 1));
      mbar_arrive_expect_tx(bar, bytes);
      bulk_load(part_ring + (i & (kWtPartRing - 1)) * kWtPartBytes,
                p.partial + ((size_t)(from * kWtEpiWarps + q) * p.nt + 32 * c) * 32, bytes, bar);
    };
    if (MODE == 0 && ok && gather > 0 && lane == 0) {
      fence_proxy_async_all();  // the partial tiles were written with plain stores
      for (int i = 0; i < kWtPartRing && i < pieces; ++i) load_part(i);
    }
    for (int c0 = 0; c0 < t.n; c0 += 32) {
      float d[2][16];
      wt_load_chunk(dcol + c0, d);
      if (c0 + 32 >= t.n) {  // the accumulator is in registers: the next tile may start
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && seg + p.nbuf < work.segs) mbar_arrive_cluster(d_empty_leader + 8 * buf);
      }
      if (MODE == 1) {
        float o[2][8];
        wt_glu(d, q, lane, ex + ((q & 1) * 2 + flip) * kWtExFloats, o);
        flip ^= 1;
        const int m = c0 + 16 * (q >> 1);
        wt_store<2>(o, out.dst + (size_t)m * out.pitch, out.pitch, rows - m);
        continue;
      }
      if (MODE == 0 && handover) {
        float4* part = reinterpret_cast<float4*>(
            p.partial + ((size_t)(blockIdx.x * kWtEpiWarps + q) * p.nt + c0) * 32) + lane;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (c0 + 8 * (i >> 1) < t.n)
            part[i * 32] = *reinterpret_cast<const float4*>(&d[i & 1][4 * (i >> 1)]);
        continue;
      }
      if (MODE == 0) {
        wt_add_bias(d, bias);
        for (int s = gather; s > 0; --s, ++piece) {
          const int slot = piece & (kWtPartRing - 1);
          if (ok) ok = mbar_wait(part_full + 8 * slot, (uint32_t)(piece / kWtPartRing) & 1u, abort_flag, 40);
          ok = __all_sync(0xffffffffu, ok);
          const uint32_t part = part_ring + slot * kWtPartBytes + lane * 16;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 w = lds_float4(part + i * 512);
            float* v = &d[i & 1][4 * (i >> 1)];
            v[0] += w.x;
            v[1] += w.y;
            v[2] += w.z;
            v[3] += w.w;
          }
          __syncwarp();
          if (lane == 0 && ok && piece + kWtPartRing < pieces) load_part(piece + kWtPartRing);
        }
      }
      if (MODE == 2) {
        wt_weigh(d, rw[0], t4);
#pragma unroll
        for (int i = 0; i < 3; ++i) rw[i] = rw[i + 1];
      }
      wt_store<4>(d, out.dst + (size_t)c0 * out.pitch, out.pitch, ok ? rows - c0 : 0);
    }
    if (MODE == 0 && handover) {
      fence_proxy_async_all();
      __syncwarp();
      if (lane == 0 && ok && !*abort_flag) p.flags.raise(blockIdx.x, q);
    }
  }
}

// Zero words and scales of a conversion warp's units, fetched one unit ahead; the warp's position in the work.
template <int MODE, int GROUP>
struct WtScales {
  static constexpr int kGroups = kWtBK / GROUP;  // quantisation groups of a stage
  const WtParams& p;
  const Work& work;
  const int rank, q, team, g, words;
  int seg, k, k_end;
  uint32_t zs;                 // index of this lane's zero word and eight scales of the next unit
  uint32_t zw[kGroups];
  uint4 sv[kGroups];
  __device__ __forceinline__ WtScales(const WtParams& p_, const Work& work_, int rank_, int warp, int lane)
      : p(p_), work(work_), rank(rank_), q(warp & 3), team(warp >> 2), g(lane >> 2), words(p_.N / kPack) {}
  __device__ __forceinline__ void settle() {  // k past the end of its segment: into the next ones
    while (k >= k_end && seg + 1 < work.segs) {
      k -= k_end;
      ++seg;
      k += work.k_begin(seg);
      k_end = work.k_end(seg);
    }
  }
  __device__ __forceinline__ uint32_t locate() const {
    const WtTile t = wt_tile<MODE, GROUP>(p, work.tile_id(seg));
    int w;
    if (MODE == 1)
      w = (q >> 1) * (p.half_cols / kPack) + t.slab * 16 + rank * 8 + 4 * (q & 1) + (g >> 1);
    else
      w = t.slab * (kWtBN / kPack) + rank * (kWtCols / kPack) + 4 * q + (g >> 1);
    w = min(w, words - 1);  // columns past the edge: any value, nothing of them is stored
    return (uint32_t)(t.grp0 + k * kGroups) * words + w;
  }
  __device__ __forceinline__ void fetch() {
#pragma unroll
    for (int i = 0; i < kGroups; ++i) {
      zw[i] = __ldg(p.qzeros + zs + i * words);
      sv[i] = __ldg(reinterpret_cast<const uint4*>(p.scales) + zs + i * words);
    }
  }
  __device__ __forceinline__ void start() {
    seg = 0;
    k = work.k_begin(0) + team;
    k_end = work.k_end(0);
    settle();
    if (team < work.count) {
      zs = locate();
      fetch();
    }
  }
  __device__ __forceinline__ void next() {
    k += kWtTeams;
    zs += (uint32_t)(kWtTeams * kGroups * words);
    if (k >= k_end) {
      settle();
      zs = locate();
    }
    fetch();
  }
};

template <int MODE, int GROUP, bool WIDE, bool SPLIT>
__global__ void __launch_bounds__(kWtThreads, 1)
gemm_wt_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ WtXMaps<MODE> map_x,
               const WtParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ volatile int s_abort;
  __shared__ uint32_t s_tmem_base;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x & 1;  // of the pair: rank 0 is the leader
  const int leader = SPLIT ? blockIdx.x % (2 * p.share.pairs) & ~1 : 0;  // its rank in the cluster
  const uint16_t pair_mask = SPLIT ? (uint16_t)(3u << leader) : (uint16_t)3;
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t x_base = smem_base;
  const uint32_t raw_base = x_base + p.nx * p.xstage;
  const uint32_t bar_base = raw_base + p.nraw * kWtRawBytes;
  auto raw_full = [&](int s) { return bar_base + 8 * s; };
  auto raw_empty = [&](int s) { return bar_base + 8 * (kWtMaxRaw + s); };
  // unit u of the pair is complete in the leader: both halves of its tokens have landed and the
  // conversion warps of both CTAs have written its A slot
  auto unit_full = [&](int u) { return bar_base + 8 * (2 * kWtMaxRaw + (u & (kWtMaxX - 1))); };
  // completion of the MMAs of unit u, in both CTAs: frees its x stage and its A slot
  auto mma_done = [&](int u) {
    return bar_base + 8 * (2 * kWtMaxRaw + kWtMaxX + (u & (kWtMaxX - 1)));
  };
  auto unit_phase = [&](int u) { return (uint32_t)((u / kWtMaxX) & 1); };
  auto d_full = [&](int b) { return bar_base + 8 * (2 * kWtMaxRaw + 2 * kWtMaxX + b); };
  auto d_empty = [&](int b) { return bar_base + 8 * (2 * kWtMaxRaw + 2 * kWtMaxX + 2 + b); };
  auto part_full = [&](int q) {
    return bar_base + 8 * (2 * kWtMaxRaw + 2 * kWtMaxX + 4 + q * kWtPartRing);
  };

  // MODE 1 waits for the kernel before it, which writes the tile table.  MODE 2 reads the same table ahead of its own wait:
  // it may start once every CTA of MODE 1 has seen that kernel complete, and its first words and scales are then under way
  // while the last CTAs of MODE 1 run.  Experts 64 x 4096 x 1536, top-4, 1024 tokens: 274 -> 253 us; 128 x 2048 x 768,
  // top-8, 1024 tokens 150 -> 144, 2500 266 -> 261; 4 x 2048 x 1024, top-1, 512 tokens 26.2 -> 23.4.
  if (MODE != 1) pdl_launch_dependents();
  if (warp == kWtIssueWarp) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s_tmem_base)),
                 "r"((uint32_t)kWtTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (MODE == 1) {
    pdl_wait();
    pdl_launch_dependents();
  }
  const Work work = wt_work<MODE, WIDE, SPLIT>(p);

  // Packed words, unit by unit: 128 rows x 16 words (MODE 1: 8 gate words and the matching 8 up
  // words).  State of the raw producer's warp.
  int raw_u = 0, raw_seg = 0, raw_k = 0, raw_end = 0, raw_s = 0, raw_w0 = 0, raw_row0 = 0;
  uint32_t raw_phase = 0;
  auto load_raw = [&]() {  // returns whether the stage after this one is known to be empty
    if (raw_k == raw_end) {
      const WtTile t = wt_tile<MODE, GROUP>(p, work.tile_id(raw_seg));
      raw_k = work.k_begin(raw_seg);
      raw_end = work.k_end(raw_seg++);
      raw_row0 = t.wrow0;
      raw_w0 = MODE == 1 ? t.slab * 16 + rank * 8
                         : t.slab * (kWtBN / kPack) + rank * (kWtCols / kPack);
    }
    const uint32_t dst = raw_base + raw_s * kWtRawBytes, bar = raw_full(raw_s);
    const int row = raw_row0 + raw_k * kWtBK;
    ++raw_u;
    ++raw_k;
    if (++raw_s == p.nraw) {
      raw_s = 0;
      raw_phase ^= 1u;
    }
    bool r = false;
    if (elect_one()) {
      r = mbar_test(raw_empty(raw_s), raw_phase ^ 1u);
      mbar_arrive_expect_tx(bar, kWtRawBytes);
      tma_load_2d(dst, &map_w, raw_w0, row, bar);
      if (MODE == 1) tma_load_2d(dst + kWtRawBytes / 2, &map_w, p.half_cols / kPack + raw_w0, row, bar);
    }
    return __any_sync(0xffffffffu, r);
  };

  if (warp == kWtRawWarp) {
    if (lane == 0) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
    if (lane == 0) s_abort = 0;
    if (lane < p.nraw) {
      mbar_init(raw_full(lane), 1);
      mbar_init(raw_empty(lane), kWtCvWarps / kWtTeams);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      fence_proxy_async();
    }
    __syncwarp();
    asm volatile("bar.arrive 1, %0;" ::"n"(kWtThreads) : "memory");
    cluster_arrive();
    // the first packed words are on their way before anyone else is through the prologue; no
    // kernel writes weights, so they need not wait for the kernel before this one
    for (int i = 0; i < kWtTeams && raw_u < work.count; ++i) load_raw();
  }
  if (warp == kWtXWarp && lane == 0) {
    for (int u = 0; u < kWtMaxX; ++u) {
      // four conversion warps of each CTA, and the leader's announcement of the tokens' bytes
      mbar_init(unit_full(u), 2 * (kWtCvWarps / kWtTeams) + 1);
      mbar_init(mma_done(u), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(d_full(b), 1);
      mbar_init(d_empty(b), 2 * kWtEpiWarps);             // the epilogue warps of both CTAs
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (MODE == 0 && !WIDE && !SPLIT && warp >= kWtEpiWarp0 && warp < kWtEpiWarp0 + kWtEpiWarps && lane < kWtPartRing) {
    mbar_init(part_full(warp - kWtEpiWarp0) + 8 * lane, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (SPLIT && warp >= kWtEpiWarp0 && warp < kWtEpiWarp0 + kWtEpiWarps && lane < work.segs) {
    // lane: segment.  What the tile's other pairs store into this CTA for this warp
    const int tile = work.tile_id(lane), eights = wt_tile<MODE, GROUP>(p, tile).n / 8;
    const int lt = tile % p.share.tiles, n = p.share.count[lt];
    const int me = blockIdx.x % (2 * p.share.pairs) / 2 - p.share.first[lt];
    const uint32_t bar = part_full(warp - kWtEpiWarp0) + 8 * (lt & 1);
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_arrive_expect_tx(bar, (wt_own_first(eights, n, me + 1) - wt_own_first(eights, n, me)) * (n - 1) * 1024);
  }
  // What a conversion warp needs for its first unit, on its way during the rest of the prologue: no kernel writes it.
  WtScales<MODE, GROUP> scales(p, work, rank, warp, lane);
  if (warp < kWtCvWarps) scales.start();
  __syncwarp();
  // Everyone but the warp of the packed words, which only tells that its barriers are set up, waits for the others'; the
  // two CTAs' set-up is awaited where something first goes from one to the other.
  tc_fence_before();
  if (warp != kWtRawWarp) named_barrier<1, kWtThreads>();
  tc_fence_after();
  if (warp != kWtRawWarp) cluster_arrive();
  const uint32_t tmem = s_tmem_base;

  if (warp == kWtRawWarp) {
    // ------------------------------------------------------------------ packed words
    // Converged, an elected lane issues, and the next stage's barrier is probed ahead of this one's load: a lane
    // that looped alone and waited for every stage took 444 cycles a unit whatever the rest of the kernel did.
    // The same for the tokens.
    bool ok = true, ready = false;
    while (raw_u < work.count) {
      if (raw_u >= p.nraw && !ready) {  // the first trip round the ring finds it empty
        ok = mbar_wait(raw_empty(raw_s), raw_phase ^ 1u, &s_abort, 31);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
      ready = load_raw();
    }
    cluster_wait();
  } else if (warp == kWtXWarp) {
    // ------------------------------------------------------------------ tokens
    pdl_wait();  // the activations may be the output of the kernel before this one
    cluster_wait();
    bool ok = true, ready = false;
    int seg = 0, k = 0, k_end = 0, s = 0;
    const CUtensorMap* map = nullptr;
    uint32_t bytes = 0;
    int row = 0;
    const uint32_t full0 = map_rank(unit_full(0), leader);
    for (int u = 0; u < work.count; ++u) {
      if (k == k_end) {
        const WtTile t = wt_tile<MODE, GROUP>(p, work.tile_id(seg));
        k = work.k_begin(seg);
        k_end = work.k_end(seg++);
        const int boxes = (t.n / 2 + 15) / 16;
        map = &map_x.map[MODE == 0 ? (t.rows < p.nt ? 1 : 0) : boxes - 1];
        bytes = (uint32_t)boxes * 16 * 256;
        row = t.m0 + rank * (t.n / 2);
      }
      if (u >= p.nx && !ready) {
        ok = mbar_wait(mma_done(u - p.nx), unit_phase(u - p.nx), &s_abort, 32);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
      bool r = false;
      if (elect_one()) {
        r = u + 1 >= p.nx && mbar_test(mma_done(u + 1 - p.nx), unit_phase(u + 1 - p.nx));
        if (rank == 0) mbar_arrive_expect_tx(unit_full(u), 2 * bytes);
        tma_load_3d_pair(x_base + s * p.xstage, map, 0, row, 2 * k, full0 + 8 * (u & (kWtMaxX - 1)));
      }
      ready = __any_sync(0xffffffffu, r);
      ++k;
      if (++s == p.nx) s = 0;
    }
    // The commits of the last units arrive asynchronously and nobody else waits for all of
    // them: see them land before the CTA may exit.  One lane: with all 32 in these waits a call took 0.05 us longer.
    if (lane == 0)
      for (int u = work.count > kWtMaxX ? work.count - kWtMaxX : 0; u < work.count && ok; ++u)
        ok = mbar_wait(mma_done(u), unit_phase(u), &s_abort, 32);
  } else if (warp == kWtIssueWarp) {
    // ------------------------------------------------------------------ MMA issue (leader)
    cluster_wait();
    if (rank == 0) {
      // What bounds this warp is its own serial chain: a barrier wait costs ~150 cycles even when
      // the phase is complete, an MMA ~25, every other instruction of the loop its full latency
      // (first version: two waits, three commits and an index division per unit, 860 cycles a
      // unit, more than anything else in the kernel).  So a unit has one barrier, probed for unit
      // u + 1 ahead of the MMAs of unit u, and one commit.
      const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
      const uint64_t desc0 = make_desc(__shfl_sync(0xffffffffu, x_base, 0), 16, 1024);
      const uint32_t stage16 = (uint32_t)p.xstage / 16, xmask = (uint32_t)p.nx - 1;
      const uint32_t full0 = unit_full(0), done0 = mma_done(0);
      bool ok = true, ready = false;
      int u = 0, slot = 0;
      for (int seg = 0; seg < work.segs && ok; ++seg) {
        // D fp32, A / B fp16, both K-major, N tokens, M = 256 weight columns
        const WtTile t = wt_tile<MODE, GROUP>(p, work.tile_id(seg));
        const int n = __shfl_sync(0xffffffffu, t.n, 0);
        const uint32_t idesc = (1u << 4) | ((uint32_t)(n >> 3) << 17) | (16u << 24);
        const uint32_t half16 = (uint32_t)((n / 2 + 15) / 16) * (16 * 128 / 16);
        const int buf = WIDE ? 0 : seg & (p.nbuf - 1), use = !WIDE && p.nbuf == 2 ? seg >> 1 : seg;
        const uint32_t dcol = tmem_u + buf * p.dcols;
        const int u_end = u + work.k_end(seg) - work.k_begin(seg);
        // the accumulator's previous tile must have been read by both epilogues
        if (use > 0) ok = mbar_wait(d_empty(buf), (uint32_t)((use - 1) & 1), &s_abort, 33);
        uint32_t acc = 0;
        for (; u < u_end; ++u) {
          if (!ready) {
            if (ok) ok = mbar_wait(full0 + 8 * (u & 7), (uint32_t)(u >> 3) & 1u, &s_abort, 34);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
          }
          tc_fence_after();
          const uint64_t dx = desc0 + (((uint32_t)u & xmask) * stage16);
          const uint32_t acol = tmem_u + p.acol + slot * 64;
          if (++slot == p.slots) slot = 0;
          bool r = false;
          if (elect_one()) {
            r = umma_unit_pair(dcol, acol, dx, half16, idesc, acc, done0 + 8 * (u & 7),
                               full0 + 8 * ((u + 1) & 7), (uint32_t)((u + 1) >> 3) & 1u, pair_mask);
            if (u == u_end - 1) umma_commit_pair(d_full(buf), pair_mask);
          }
          acc = 1;
          ready = __any_sync(0xffffffffu, r);
        }
      }
    }
  } else if (warp < kWtCvWarps) {
    // ------------------------------------------------------------------ conversion warps
    const int g = lane >> 2;
    const int q = warp & 3, team = warp >> 2;
    const uint32_t lane_q = (uint32_t)(q * 32) << 16;
    // ldmatrix: matrix m = lane / 8 of the four holds rows 8 m .. 8 m + 7 of 32; after the transposed load
    // thread (g, t) has rows 2 t and 2 t + 1 of halfword column g in a register of each.
    const uint32_t ld_off =
        MODE == 1
            // two boxes of [128 rows x 32 B], 32-byte swizzle
            ? (uint32_t)((q >> 1) * (kWtRawBytes / 2) + lane * 32 + (((q & 1) ^ ((lane >> 2) & 1)) << 4))
            // one box of [128 rows x 64 B], 64-byte swizzle
            : (uint32_t)(lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4));
    constexpr uint32_t kPairBytes = 32 * (MODE == 1 ? 32 : 64);  // 32 rows further on
    const uint32_t half_sel = (g & 1) ? 0x3232u : 0x1010u;      // this lane's halfword, duplicated
    constexpr int kGroups = kWtBK / GROUP;                        // quantisation groups of a stage
    const uint32_t full_leader = map_rank(unit_full(0), leader);

    bool ok = true, joined = false;
    int s = team, slot = team;  // nraw, slots >= kWtTeams
    uint32_t phase = 0;
    for (int u = team; u < work.count; u += kWtTeams) {
      uint32_t zw[kGroups];
      uint4 sv[kGroups];
#pragma unroll
      for (int i = 0; i < kGroups; ++i) {
        zw[i] = scales.zw[i];
        sv[i] = scales.sv[i];
      }
      if (u + kWtTeams < work.count) scales.next();

      // the unit's words, and the MMAs that read its A slot last; probed together, a wait of its own each took
      // 100 to 150 cycles with nothing to wait for
      const bool first = u < p.slots;
      const uint32_t slot_bar = first ? raw_full(s) : mma_done(u - p.slots);
      const uint32_t slot_phase = first ? phase : unit_phase(u - p.slots);
      if (!__all_sync(0xffffffffu, mbar_try_wait2(raw_full(s), phase, slot_bar, slot_phase))) {
        ok = mbar_wait(raw_full(s), phase, &s_abort, 36) && mbar_wait(slot_bar, slot_phase, &s_abort, 37);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
      }
      tc_fence_after();
      const uint32_t raw = raw_base + s * kWtRawBytes + ld_off;
      uint32_t w[4][4];
#pragma unroll
      for (int pr = 0; pr < 4; ++pr) ldmatrix_x4_trans(raw + pr * kPairBytes, w[pr]);
      const uint32_t a_slot = tmem + lane_q + p.acol + slot * 64;
      // column 2 i + g % 2 of this lane's word: zero and scale, duplicated over (k, k + 1).  Odd i
      // keep the nibble in place (1024 + 16 q): their zero is 1024 + 16 z, their scale s / 16.
      __half2 z[4], sc[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {  // 32 rows each
        if (h * 32 % GROUP == 0) {
          const int gi = h * 32 / GROUP;
          const uint32_t zz = prmt(zw[gi], zw[gi], half_sel), zh = zz >> 8;
          z[0] = as_half2(lop3_and_or(zz, 0x000F000Fu, 0x64006400u));
          z[1] = as_half2(lop3_and_or(zz, 0x00F000F0u, 0x64006400u));
          z[2] = as_half2(lop3_and_or(zh, 0x000F000Fu, 0x64006400u));
          z[3] = as_half2(lop3_and_or(zh, 0x00F000F0u, 0x64006400u));
          const __half2 r16 = __float2half2_rn(0.0625f);
          sc[0] = as_half2(prmt(sv[gi].x, sv[gi].x, half_sel));
          sc[1] = __hmul2(as_half2(prmt(sv[gi].y, sv[gi].y, half_sel)), r16);
          sc[2] = as_half2(prmt(sv[gi].z, sv[gi].z, half_sel));
          sc[3] = __hmul2(as_half2(prmt(sv[gi].w, sv[gi].w, half_sel)), r16);
        }
        uint32_t frag[2][8];  // [lane half of the quarter][2 * eight rows + i odd]
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t r = w[h][c], rh = r >> 8;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            frag[i >> 1][2 * c + (i & 1)] = as_u32(__hmul2(
                __hsub2(as_half2(lop3_and_or((i & 2) ? rh : r, (i & 1) ? 0x00F000F0u : 0x000F000Fu,
                                             0x64006400u)),
                        z[i]),
                sc[i]));
        }
        tmem_st_16x128b(a_slot + h * 16, frag[0]);
        tmem_st_16x128b(a_slot + (16u << 16) + h * 16, frag[1]);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (!joined) cluster_wait();  // the leader's barriers are set up
      joined = true;
      mbar_arrive_both(full_leader + 8 * (u & (kWtMaxX - 1)), raw_empty(s), lane == 0);
      slot += kWtTeams;
      if (slot >= p.slots) slot -= p.slots;
      s += kWtTeams;
      if (s >= p.nraw) {
        s -= p.nraw;
        phase ^= 1u;
      }
    }
    if (!joined) cluster_wait();
  } else {
    // ------------------------------------------------------------------ epilogue
    cluster_wait();
    const int e = warp - kWtEpiWarp0;
    const uint32_t ex_base = bar_base + kWtBarBytes;
    float* ex = reinterpret_cast<float*>(smem_raw + (ex_base - smem_u32(smem_raw)));
    if constexpr (WIDE) {
      const uint32_t stage = ex_base + (MODE == 1 ? kWtExBytes : 0) + e * (p.stage_bytes / kWtEpiWarps);
      wt_epilogue_wide<MODE, GROUP>(p, work, tmem, rank, e, lane, d_full(0), d_empty(0), ex, stage, &s_abort);
    } else if constexpr (SPLIT) {
      wt_epilogue_split<GROUP>(p, work, tmem, rank, e, lane, d_full(0), ex_base, part_full(e), &s_abort);
    } else {
      wt_epilogue<MODE, GROUP>(p, work, tmem, rank, e, lane, d_full(0), d_empty(0), ex,
                               x_base + e * (kWtPartRing * kWtPartBytes), part_full(e), &s_abort);
    }
  }

  // ---- teardown ----
  __syncwarp();
  if (s_abort) {
    // a wait gave up: copies and MMAs may still be in flight towards this pair's shared and
    // tensor memory.  Let them land before both are given back.
    linger();
    // flags raised meanwhile: a replay of this launch must not find them
    if (MODE == 0 && !WIDE && !SPLIT && warp >= kWtEpiWarp0 && warp < kWtEpiWarp0 + kWtEpiWarps && work.segs > 0)
      for (int c = 1 + lane; c <= work.helpers(work.segs - 1); c += 32)
        p.flags.lower(blockIdx.x - 2 * c, warp - kWtEpiWarp0);
  }
  tc_fence_before();
  __syncthreads();
  // Nothing of another CTA is on its way to this one any more: whatever one sent another has been waited for there, but
  // after a wait that gave up.  So the barrier orders no memory: a release waits for this CTA's stores of the output, 1000
  // cycles.  1024 x 8192 at M 40 5.00 -> 4.85 us, 3712 x 8192 at M 200 15.0 -> 14.4, 2048 x 5120 at M 300 10.9 -> 10.3.
  cluster_arrive_relaxed();
  cluster_wait();
  if (warp == kWtIssueWarp) {
    if (s_abort) linger();  // what was sent until the barrier lands
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"((uint32_t)kWtTmemCols)
                 : "memory");
  }
}

// ---- host side -------------------------------------------------------------------------------

// Pairs of CTAs the GPU holds at once (one CTA per SM): how wide the work is spread, every GPU has room for one.
template <int MODE, int GROUP, bool WIDE, bool SPLIT = false>
int wt_pairs(int smem) {
  static std::atomic<int> cached[64][9];  // zero-initialised: not asked yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
  const int got = resident_clusters(gemm_wt_kernel<MODE, GROUP, WIDE, SPLIT>, 2, kWtThreads, smem, cached[dev]);
  const int most = sm_count() / 2 < kWtMaxPairs ? sm_count() / 2 : kWtMaxPairs;
  return got > 0 && got < most ? got : most;
}

template <int MODE, int GROUP, bool WIDE, bool SPLIT = false>
int wt_prepare() {
  static std::atomic<bool> attr_done[64];  // zero-initialised; setting the attribute twice is harmless
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return AWQ_B200_ERR_DEVICE;
  if (!attr_done[dev]) {
    if (cudaFuncSetAttribute(gemm_wt_kernel<MODE, GROUP, WIDE, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kWtSmemLimit) != cudaSuccess)
      return AWQ_B200_ERR_LAUNCH;
    if (SPLIT && cudaFuncSetAttribute(gemm_wt_kernel<MODE, GROUP, WIDE, SPLIT>,
                                      cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
      return AWQ_B200_ERR_LAUNCH;
    attr_done[dev] = true;
  }
  return AWQ_B200_OK;
}

// How `pairs` pairs of a cluster share its `tiles` tiles of up to `nt` tokens: even ranges.
WtShare wt_share(int pairs, int tiles, int KT, int nt) {
  WtShare s = {};
  s.pairs = pairs;
  s.tiles = tiles;
  for (int i = 0; i <= pairs; ++i) s.bound[i] = (short)((long)i * tiles * KT / pairs);
  for (int t = 0; t < tiles; ++t) {
    int a = 0, b = pairs - 1;
    while (s.bound[a + 1] <= t * KT) ++a;
    while (s.bound[b] >= (t + 1) * KT) --b;
    const int n = b - a + 1, bytes = kWtEpiWarps * ((nt / 8 + n - 1) / n) * (n - 1) * 1024;
    s.first[t] = (signed char)a;
    s.count[t] = (signed char)n;
    s.recip[t] = (65536 + n - 1) / n;
    if (bytes > s.recv) s.recv = bytes;
  }
  return s;
}

// Ranges of `chunk` units, tiles of KT units and 65 to 128 tokens: whether one accumulator and six A slots are faster than
// two and four.  The epilogue that nothing hides is paid for once a tile of KT units, unless the range is shorter than a
// tile and ends one at most.  At 128 tokens the MMAs take as long as the conversion, and a unit gains less, but in groups
// of 64, whose conversion is longer.  Two -> one, us: 29568 x 8192 M 100 54.8 -> 53.7, groups of 64 56.4 -> 55.0; 14336 x
// 28672 M 100 87.3 -> 85.6; 7168 x 22016 M 100 36.2 -> 36.0, M 128 42.3 -> 43.1; 8192 x 28672 M 128 58.3 -> 59.2, groups
// of 64 62.3 -> 61.8; 11008 x 57344 M 128 98.3 -> 98.0, x 28672 no difference; 14336 x 28672 M 128 105.1 -> 104.3; 8192
// x 12288 M 112 34.9 -> 33.9 and 10240 x 11008 M 128 34.5 -> 33.8 (less than a tile a range); 4096 x 22016 M 100 22.7 ->
// 22.9.
constexpr int kWtOneStages = 56, kWtOneStagesFull = 80;
bool wt_one_accumulator(int nt, int chunk, int KT, int group) {
  if (chunk == 0 || KT < kWtOneStages) return false;
  return nt < 128 || group == 64 || chunk < KT || KT >= kWtOneStagesFull;
}

// Ring depths for a tile of `nt` tokens; the rest of shared memory goes to the packed words, which
// come from HBM (8 KB a stage).  `group`: of a dense call.
int wt_rings(WtParams* p, int mode, int group) {
  const int rows = (p->nt / 2 + 15) / 16 * 16;
  p->xstage = rows * 256;
  p->nx = p->xstage <= (16 << 10) ? 8 : 4;
  // Two accumulators, so that the next tile's MMAs run under the epilogue, while they fit beside six A slots, or beside four
  // where a CTA has many tiles; what TMEM is left over goes to A slots.
  const bool one =
      p->nt > 128 || (p->nt > 64 && (p->share.tiles == 1 || wt_one_accumulator(p->nt, p->chunk, p->KT, group)));
  p->nbuf = one ? 1 : 2;
  // One accumulator and whole tiles: the WIDE kernel.
  p->stage_bytes = p->nbuf == 2 || p->chunk > 0 || p->share.pairs > 0 ? 0 : (p->nt + 31) / 32 * 32 * kWtCols * (mode == 1 ? 1 : 2);
  const int recv = p->share.pairs > 0 ? p->share.recv * (p->share.tiles > 1 ? 2 : 1) : 0;
  const int fixed = 1024 + kWtBarBytes + (mode == 1 ? kWtExBytes : 0) + p->stage_bytes + recv;
  p->dcols = p->nt <= 64 ? 64 : 128;
  p->acol = p->nbuf == 2 ? 2 * p->dcols : (p->nt + 63) / 64 * 64;
  p->slots = (kWtTmemCols - p->acol) / 64;
  p->nraw = (kWtSmemLimit - fixed - p->nx * p->xstage) / kWtRawBytes;
  if (recv > 0 && p->nx == 8 && p->nraw < 2 * kWtTeams) {
    p->nx = 4;
    p->nraw = (kWtSmemLimit - fixed - p->nx * p->xstage) / kWtRawBytes;
  }
  if (p->nraw > kWtMaxRaw) p->nraw = kWtMaxRaw;
  // A team waits for unit u in the stage that unit u - nraw had.  Either it read that one itself, or it has seen
  // the MMAs of a later unit complete (u - 4 - slots, when it wrote unit u - 4); between the two, the parity of
  // the filling before could pass for the one it waits for.  Fewer slots rather than fewer x stages: with four of those 8192 x
  // 8192 at M 100 took 17.3 us, with eight 17.0.
  if (p->nraw < 2 * kWtTeams) p->nraw = kWtTeams;
  else if (p->slots > p->nraw - kWtTeams) p->slots = p->nraw - kWtTeams;
  return fixed + p->nx * p->xstage + p->nraw * kWtRawBytes;
}

template <int MODE, int GROUP, bool WIDE, bool SPLIT = false>
int launch_wt_kernel(const CUtensorMap& map_w, const WtXMaps<MODE>& map_x, const WtParams& p, int pairs,
                     int smem, cudaStream_t stream) {
  if (int rc = wt_prepare<MODE, GROUP, WIDE, SPLIT>()) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(kWtThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = SPLIT ? 2 * p.share.pairs : 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = add_pdl_attribute(attr, 1);
  if (cudaLaunchKernelEx(&cfg, gemm_wt_kernel<MODE, GROUP, WIDE, SPLIT>, map_w, map_x, p) != cudaSuccess) {
    cudaGetLastError();
    return AWQ_B200_ERR_LAUNCH;
  }
  return AWQ_B200_OK;
}

// packed weights [rows][N / 8 words], box [128 rows x 16 words] (gate_up: 8), swizzle = box width
int make_wt_map(CUtensorMap* map_w, const uint32_t* qweight, int64_t wrows, int N, int box_words) {
  return encode_map_2d(map_w, CU_TENSOR_MAP_DATA_TYPE_INT32, qweight, (uint64_t)(N / kPack),
                       (uint64_t)wrows, (uint64_t)(N / kPack) * 4, (uint32_t)box_words, kWtBK,
                       box_words == 16 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

// Scratch of the chunked split: one partial tile per CTA, and the flags.
size_t wt_partial_bytes(int nt, int pairs) { return (size_t)2 * pairs * nt * kWtCols * sizeof(float); }
size_t wt_scratch_bytes(int nt, int pairs) { return wt_partial_bytes(nt, pairs) + handover::kFlagBytes; }

// How a dense call is cut: tokens of a tile, and units of a pair's range (0: whole tiles, strided) or the pairs and
// tiles of a cluster (SPLIT).
struct WtPlan {
  int nt, chunk, pairs;
  int share, share_tiles;
  long cost;  // estimated time in ns
};

// Estimated time in ns of `tiles` tiles of `nt` tokens and KT units on `pairs` pairs (chunk as above).
// Fitted to 7 shapes between 1024 x 8192 and 4096 x 11040 at 14 batch sizes from 17 to 1000, 1500 cuts in all, when a
// unit took 630 cycles and the epilogue of one accumulator 6600.  On the present kernel the cut it picks is 0.9 % from
// the best one on average, 15 % at worst (1735 cuts of 174 batches, 12 shapes up to 8192 x 59136, 17 to 1000 tokens; 1024 x
// 8192 at 160 tokens takes tiles of 80, 8.3 us, where 160 take 7.3).
//   2400 + 18 nt            start, and the epilogue that nothing hides
//   units x max(...)        315: the conversion arithmetic; 2.5 nt: the tensor pipe; 4.9 pairs: the words'
//                           way from HBM through L2
//   1300                    more than half of the GPU: the next kernel's start is not hidden
//   2000 + 11 nt            a tile handed over, and 40 + 8 nt for each CTA the last one collects from
//   17 nt / 6 nt            a further tile of the pair (one accumulator / two, hidden in part)
long wt_cost(int nt, int tiles, int KT, int chunk, int most, int pairs) {
  int units, segs, gather = 0;
  if (chunk == 0) {
    segs = (tiles + pairs - 1) / pairs;
    units = segs * KT;
  } else {
    units = chunk;
    segs = (chunk + KT - 1) / KT;
    if (KT % chunk == 0) {
      gather = KT / chunk - 1;
    } else if (chunk % KT != 0) {
      gather = chunk > KT ? 1 : (KT - 2) / chunk + 1;
      ++segs;
    }
  }
  long unit = 315;
  if (unit < nt * 5 / 2) unit = nt * 5 / 2;
  if (unit < pairs * 49 / 10) unit = pairs * 49 / 10;
  long t = 2400 + 18 * nt + units * unit + (long)(segs - 1) * nt * (nt > 128 ? 17 : 6);
  if (pairs > most / 2) t += 1300;
  if (gather > 0) t += 2000 + 11 * nt + gather * (40 + 8 * nt);
  return t;
}

// The cheapest cut.  Small tiles and split ones cost conversion twice or a hand-over, and pay where
// whole ones leave pairs idle; `split` false: whole tiles only (no scratch).  Where tiles of 256 tokens
// fill the GPU the tiles stay whole and large, since the power limit then counts as well, and the waves of
// tiles shall carry the fewest token columns in sequence.
WtPlan wt_search(int M, int slabs, int KT, int most, bool split) {
  WtPlan best = {0, 0, 1, 0, 0, -1};
  const bool full = M > 256 && (long)slabs * ((M + 255) / 256) >= most;
  if (full) {
    for (int nt = 256; nt >= 128; nt -= 16) {
      const long tiles = (long)slabs * ((M + nt - 1) / nt), cost = (tiles + most - 1) / most * nt;
      if (best.cost < 0 || cost < best.cost) best = {nt, 0, most, 0, 0, cost};
    }
    return best;
  }
  const int least = M > 512 ? 96 : 32;  // the smallest tiles never won beyond 512 tokens
  for (int top = 256, last = 0; top >= least || last == 0; top -= 16) {
    const int mtiles = (M + top - 1) / top, nt = ((M + mtiles - 1) / mtiles + 15) / 16 * 16;
    if (nt == last) continue;
    last = nt;
    const int tiles = slabs * ((M + nt - 1) / nt);
    const long units = (long)tiles * KT;
    const int even = (int)((units + most - 1) / most);
    for (int parts = 1; parts <= (split && units < (1 << 30) ? 6 : 1); ++parts) {
      WtPlan plan = {nt, 0, tiles < most ? tiles : most, 0, 0, 0};
      if (parts > 1) {
        const int floor = (KT + parts - 1) / parts;
        plan.chunk = even > floor ? even : floor;
        plan.pairs = (int)((units + plan.chunk - 1) / plan.chunk);
      }
      plan.cost = wt_cost(nt, tiles, KT, plan.chunk, most, plan.pairs);
      if (best.cost < 0 || plan.cost < best.cost) best = plan;
      if (plan.chunk == even) break;  // more parts: the same cut
    }
  }
  return best;
}

// Clusters of `pairs` pairs that share `tiles` tiles each, all in one wave: estimated time in ns; `resident` clusters
// of that size fit the GPU.  Fitted to 550 cuts, 17 shapes from 1024 x 2048 to 14848 x 8192 at 11 batches from 33 to
// 400 tokens, 4 % off on average.
//   1170 + 25 nt + 144 pairs        start, the parts' way to the CTA that sums them, the sum
//   units x max(...)                274: the conversion arithmetic; 2.3 nt: the tensor pipe; 5.1 pairs of the call: words
//   1240 + 1510 x (...)             no room for the next kernel's clusters beside these: its start is not hidden
//   18 nt - 600                     two tiles for three pairs: the middle pair sums parts of both
long wt_cluster_cost(int nt, int pairs, int tiles, int clusters, int KT, int resident) {
  long unit = 274;
  if (unit < nt * 23 / 10) unit = nt * 23 / 10;
  if (unit < (long)clusters * pairs * 51 / 10) unit = (long)clusters * pairs * 51 / 10;
  long t = 1170 + 25 * nt + 144 * pairs + (tiles * KT + pairs - 1) / pairs * unit;
  if (2 * clusters > resident) t += 1240 + 1510L * (2 * clusters - resident) / resident;
  if (tiles > 1) t += 18 * nt - 600;
  return t;
}
// The cheapest cut into clusters, if it is cheaper than the ranges by more than the estimates are apart: wt_cost was fitted
// to a kernel whose start took longer, and says too little of whole tiles on more than half of the GPU, beside which the next
// kernel's do not start.  Fitted to 1540 calls of 33 to 700 tokens, near the line most of them, timed as clusters and as
// ranges; `most` pairs fit the GPU.  With a margin of 400 ns 271 were slower in clusters than in ranges by more than 1 %, most
// of them with K up to 1024 (896 x 3232 at M 109 4.3 -> 5.3 us); now 40, 8 % at worst, and 0.2 % from the better of the two
// on average, which was 1.3 %.
long wt_cluster_margin(bool two_tiles, const WtPlan& ranges, int KT, int most) {
  const bool over_half = ranges.chunk == 0 && 2 * ranges.pairs > most;
  return 1200 + (two_tiles ? 200 : 0) - (over_half ? 30 * (KT < 30 ? KT : 30) : 0);
}
constexpr int kWtShares[][2] = {{2, 1}, {3, 1}, {4, 1}, {5, 1}, {6, 1}, {8, 1}, {3, 2}};  // pairs, tiles of a cluster
template <typename Resident>
WtPlan wt_cluster_search(WtPlan best, int M, int slabs, int KT, int most, Resident resident) {
  const WtPlan ranges = best;
  best.cost = -1;
  int room[kMaxCluster + 1] = {};
  for (const auto& s : kWtShares) room[s[0]] = resident(s[0]);
  for (int top = 256, last = 0; top >= 32; top -= 16) {
    const int mtiles = (M + top - 1) / top, nt = ((M + mtiles - 1) / mtiles + 15) / 16 * 16;
    if (nt == last) continue;
    last = nt;
    const int tiles = slabs * ((M + nt - 1) / nt);
    for (const auto& s : kWtShares) {
      const int pairs = s[0], per = s[1], clusters = tiles / per;
      // two tiles in turn need two accumulators; every pair has a unit; WtShare counts in 16 bits
      if (tiles % per != 0 || (long)per * KT > 32767 || (per > 1 && nt > 128) || KT < pairs || clusters > room[pairs]) continue;
      const long cost = wt_cluster_cost(nt, pairs, per, clusters, KT, room[pairs]);
      if (best.cost >= 0 && cost >= best.cost) continue;
      WtParams p = {};
      p.nt = nt;
      p.share = wt_share(pairs, per, KT, nt);
      const int smem = wt_rings(&p, 0, kWtBK);
      if (p.nraw >= kWtTeams && smem <= kWtSmemLimit) best = {nt, 0, clusters * pairs, pairs, per, cost};
    }
  }
  if (best.cost < 0) return ranges;
  return best.cost + wt_cluster_margin(best.share_tiles > 1, ranges, KT, most) < ranges.cost ? best : ranges;
}

template <typename Resident>
WtPlan wt_find(int M, int slabs, int KT, int most, bool split, bool clusters, Resident resident) {
  const WtPlan plan = wt_search(M, slabs, KT, most, split);
  // whole tiles that fill the GPU stay as they are
  const bool full = M > 256 && (long)slabs * ((M + 255) / 256) >= most;
  return clusters && !full ? wt_cluster_search(plan, M, slabs, KT, most, resident) : plan;
}

int current_device() {
  int dev = -1;
  return cudaGetDevice(&dev) == cudaSuccess ? dev : -1;
}

// `resident`: nullptr for no clusters.  A call asks for the ranges (how much scratch) and for the clusters of one shape.
WtPlan wt_plan(int M, int slabs, int KT, int most, bool split, int group, int (*resident)(int pairs) = nullptr) {
  static thread_local CutCache<WtPlan> cuts;
  const CutKey key = {M, slabs, KT, most, current_device(), group, (split ? 1 : 0) + (resident != nullptr ? 2 : 0)};
  return cuts.get(key, [&] { return wt_find(M, slabs, KT, most, split, resident != nullptr, resident); });
}

// Clusters of that many pairs that the GPU holds at once.
template <int GROUP>
int wt_resident(int pairs) {
  static std::atomic<int> cached[64][kMaxCluster + 1];  // zero-initialised: not asked yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  return resident_clusters(gemm_wt_kernel<0, GROUP, false, true>, 2 * pairs, kWtThreads, kWtSmemLimit, cached[dev]);
}

template <int GROUP>
int launch_wt_dense(const __half* x, const uint32_t* qweight, WtParams p, void* workspace,
                    size_t workspace_bytes, bool clusters, cudaStream_t stream) {
  if (int rc = wt_prepare<0, GROUP, false>()) return rc;
  if (int rc = wt_prepare<0, GROUP, false, true>()) return rc;
  p.slabs = (p.N + kWtBN - 1) / kWtBN;
  p.KT = p.K / kWtBK;
  const int most = wt_pairs<0, GROUP, false>(kWtSmemLimit);
  const auto resident = clusters ? wt_resident<GROUP> : nullptr;
  WtPlan plan = wt_plan(p.M, p.slabs, p.KT, most, true, GROUP, resident);
  if (plan.chunk > 0) {
    if (workspace != nullptr && workspace_bytes >= wt_scratch_bytes(plan.nt, plan.pairs)) {
      p.partial = static_cast<float*>(workspace);
      p.flags = handover::make_flags(workspace, wt_partial_bytes(plan.nt, plan.pairs));
    } else {
      plan = wt_plan(p.M, p.slabs, p.KT, most, false, GROUP, resident);
    }
  }
  p.nt = plan.nt;
  p.chunk = plan.chunk;
  p.mtiles = (p.M + p.nt - 1) / p.nt;
  if (plan.share > 0) p.share = wt_share(plan.share, plan.share_tiles, p.KT, p.nt);
  const int smem = wt_rings(&p, 0, GROUP);
  CUtensorMap map_w;
  WtXMaps<0> map_x;
  if (int rc = make_wt_map(&map_w, qweight, p.K, p.N, 16)) return rc;
  const int rows[2] = {p.nt, p.M - (p.mtiles - 1) * p.nt};  // of a full tile, of the last one
  for (int i = 0; i < 2; ++i) {
    const int boxes = ((rows[i] + 15) / 16 * 8 + 15) / 16;
    if (int rc = encode_map_x(&map_x.map[i], x, p.M, p.K, boxes * 16)) return rc;
  }
  if (plan.share > 0) return launch_wt_kernel<0, GROUP, false, true>(map_w, map_x, p, plan.pairs, smem, stream);
  return p.stage_bytes > 0 ? launch_wt_kernel<0, GROUP, true>(map_w, map_x, p, plan.pairs, smem, stream)
                           : launch_wt_kernel<0, GROUP, false>(map_w, map_x, p, plan.pairs, smem, stream);
}

}  // namespace

bool gemm_wt_supported(int M, int N, int K, int group) {
  // N % 32: 16-byte TMA row pitch of the packed weights; K % 128: whole stages
  return M >= 1 && N % 32 == 0 && K % kWtBK == 0 && (group == 128 || group == 64);
}

size_t gemm_wt_workspace_bytes(int M, int N, int K, int group) {
  if (!gemm_wt_supported(M, N, K, group)) return 0;
  const WtPlan plan = wt_plan(M, (N + kWtBN - 1) / kWtBN, K / kWtBK, sm_count() / 2, true, group);
  return plan.chunk > 0 ? wt_scratch_bytes(plan.nt, plan.pairs) : 0;
}

int gemm_wt_cut(int M, int N, int K, int group, int cta_pairs, int* tokens, int* chunk, int* wide) {
  if (!gemm_wt_supported(M, N, K, group)) return AWQ_B200_ERR_SHAPE;
  if (cta_pairs == 0) {
    if (int rc = group == 128 ? wt_prepare<0, 128, false>() : wt_prepare<0, 64, false>()) return rc;
    cta_pairs = group == 128 ? wt_pairs<0, 128, false>(kWtSmemLimit) : wt_pairs<0, 64, false>(kWtSmemLimit);
  }
  const WtPlan plan = wt_plan(M, (N + kWtBN - 1) / kWtBN, K / kWtBK, cta_pairs, true, group);
  WtParams p = {};
  p.nt = plan.nt;
  p.chunk = plan.chunk;
  p.KT = K / kWtBK;
  wt_rings(&p, 0, group);
  *tokens = plan.nt;
  *chunk = plan.chunk;
  *wide = p.stage_bytes > 0 ? 1 : 0;
  return AWQ_B200_OK;
}

int gemm_wt_cut(int M, int N, int K, int group, bool clusters, const int* room, GemmCut* out) {
  if (!gemm_wt_supported(M, N, K, group)) return AWQ_B200_ERR_SHAPE;
  const int slabs = (N + kWtBN - 1) / kWtBN, KT = K / kWtBK;
  WtPlan plan;
  if (room == nullptr) {
    int rc = group == 128 ? wt_prepare<0, 128, false>() : wt_prepare<0, 64, false>();
    if (rc == AWQ_B200_OK) rc = group == 128 ? wt_prepare<0, 128, false, true>() : wt_prepare<0, 64, false, true>();
    if (rc) return rc;
    const int most = group == 128 ? wt_pairs<0, 128, false>(kWtSmemLimit) : wt_pairs<0, 64, false>(kWtSmemLimit);
    plan = wt_plan(M, slabs, KT, most, true, group, !clusters ? nullptr : group == 128 ? wt_resident<128> : wt_resident<64>);
  } else {
    plan = wt_find(M, slabs, KT, room[2], true, clusters, [room](int pairs) { return room[2 * pairs]; });
  }
  WtParams p = {};
  p.nt = plan.nt;
  p.chunk = plan.chunk;
  p.KT = KT;
  if (plan.share > 0) p.share = wt_share(plan.share, plan.share_tiles, KT, plan.nt);
  wt_rings(&p, 0, group);
  *out = {plan.nt, plan.chunk, 2 * plan.share, plan.share_tiles, p.nbuf};
  return AWQ_B200_OK;
}

int launch_gemm_wt(const __half* x, const uint32_t* qweight, const __half* scales,
                   const uint32_t* qzeros, const __half* bias, __half* out, int M, int N, int K,
                   int group, void* workspace, size_t workspace_bytes, bool clusters, cudaStream_t stream) {
  if (!gemm_wt_supported(M, N, K, group)) return AWQ_B200_ERR_SHAPE;
  WtParams p = {};
  p.scales = scales;
  p.qzeros = qzeros;
  p.bias = bias;
  p.out = out;
  p.M = M;
  p.N = N;
  p.K = K;
  return group == 128 ? launch_wt_dense<128>(x, qweight, p, workspace, workspace_bytes, clusters, stream)
                      : launch_wt_dense<64>(x, qweight, p, workspace, workspace_bytes, clusters, stream);
}

namespace {
template <int MODE, int GROUP>
int launch_wt_moe(const __half* a, int64_t a_rows, const uint32_t* w, int experts, int tile_rows,
                  WtParams p, cudaStream_t stream) {
  if (int rc = wt_prepare<MODE, GROUP, false>()) return rc;
  p.KT = p.K / kWtBK;
  p.slabs = MODE == 1 ? p.half_cols / 128 : p.N / kWtBN;
  p.nt = tile_rows;
  const int smem = wt_rings(&p, MODE, GROUP);
  CUtensorMap map_w;
  WtXMaps<MODE> map_x;
  if (int rc = make_wt_map(&map_w, w, (int64_t)experts * p.K, p.N, MODE == 1 ? 8 : 16)) return rc;
  for (int boxes = 1; boxes <= 8; ++boxes)
    if (int rc = encode_map_x(&map_x.map[boxes - 1], a, a_rows, p.K, boxes * 16)) return rc;
  const int pairs = wt_pairs<MODE, GROUP, false>(kWtSmemLimit);
  return p.stage_bytes > 0 ? launch_wt_kernel<MODE, GROUP, true>(map_w, map_x, p, pairs, smem, stream)
                           : launch_wt_kernel<MODE, GROUP, false>(map_w, map_x, p, pairs, smem, stream);
}
}  // namespace

// Grouped expert GEMM of a fused-MoE layer (MODE 1 / 2 of the kernel) over the tile table of
// moe_gather_kernel, of at most tile_rows rows each.  a: activations in permuted row order [a_rows, K];
// w: packed expert weights stacked along the rows [experts * K, N / 8].  row_weights (mode 2): a routed
// weight per row of a, readable up to 32 rows past the last tile.
int launch_wt_grouped(int mode, int tile_rows, const __half* a, int64_t a_rows, const uint32_t* w, int experts,
                      const __half* scales, const uint32_t* qzeros, const int4* tiles,
                      const int32_t* n_tiles, const float* row_weights, __half* out, int K, int N, int group,
                      int half_cols, cudaStream_t stream) {
  if ((group != 128 && group != 64) || K % kWtBK != 0 || N % 32 != 0) return AWQ_B200_ERR_SHAPE;
  WtParams p = {};
  p.scales = scales;
  p.qzeros = qzeros;
  p.out = out;
  p.M = (int)a_rows;
  p.N = N;
  p.K = K;
  p.tiles = tiles;
  p.n_tiles = n_tiles;
  p.row_weights = row_weights;
  p.half_cols = half_cols;
  if (mode == 1)
    return group == 128 ? launch_wt_moe<1, 128>(a, a_rows, w, experts, tile_rows, p, stream)
                        : launch_wt_moe<1, 64>(a, a_rows, w, experts, tile_rows, p, stream);
  return group == 128 ? launch_wt_moe<2, 128>(a, a_rows, w, experts, tile_rows, p, stream)
                      : launch_wt_moe<2, 64>(a, a_rows, w, experts, tile_rows, p, stream);
}

int wt_device_status(int* out, int clear) { return read_tc_status(out, clear); }

}  // namespace awq
