// Decode-size AWQ GEMM (M <= 32) on tcgen05 with the weights going registers -> TMEM.
//
//   D[n, m] = sum_k W[k, n] * x[m, k]          (the transposed product, as in stream_core.cuh)
//
// The int4 weights are unpacked in registers (ldmatrix.trans pairs the rows k, k + 1 of a halfword
// column in the load; one AND per pair, nibbles used as fp16 subnormals q * 2^-24, exact), written to
// tensor memory with tcgen05.st.16x128b and are the A operand (128 weight columns x 16 k) of
// tcgen05.mma.kind::f16; the activations are the small B operand as TMA delivers them.  No arithmetic
// is spent on a weight: zero point and scale are applied per quantisation group to the fp32
// accumulators,  tot += scale * (acc - zero * sum_k x).
// SUB forms subtract the zero point in the conversion (q - z is exact in the subnormals too) and need no token sums:
// tot += scale * acc.  That costs the conversion 128 instructions a unit and scheduler, on the FMA pipe, and saves the
// warp that sums tokens, whose chain of loads and mma.sync took 700 to 1200 cycles a unit and was the slowest role from
// 16 tokens on, and half of the fold.  M 32 on 8192 x 59136: with token sums 74 us, with SUB and its second issuing warp
// 56; M 16, groups of 64: 56.0 -> 50.5.  At M <= 16 and groups of 128 long layers keep the sums (SUB: 41.4 -> 43.6 us at
// M 1, 47.4 -> 48.2 at 16), short ones go to clusters (below), which gain from a shorter chain: 2048 x 5120 at M 1 5.24 ->
// 4.73 us from SUB alone.
//
// One CTA per SM; slab of 256 output columns = two A tiles of 128 lanes; unit = 128 weight rows = one
// quantisation group (groups of 64: two, with accumulators and sums of their own): 16 KB of packed words,
// 512 B of scales and 128 B of zero points per group, all by TMA.  The
// (slab, unit) list is cut into one range per CTA and shared slabs are handed over (handover.cuh).
// SPLIT is the form of short layers: a cluster of 2 to 16 CTAs shares each slab, and its sums go from CTA to CTA through
// shared memory.  A CTA sums its share of the (32 columns, half of the tokens) pieces: every other CTA stores its
// part of one there with st.async, counted by an mbarrier, and all warps that have nothing left to do add them up in the
// CTAs' order.  A partial slab through global scratch costs its stores, a release, an acquire and the loads, 1.5 us at one
// token and 4 to 8 at 32; this 0.8 us.  The barrier at the end is a relaxed one: as a release it waited 1000 cycles
// for the stores of the output.  (Bulk copies between shared memories instead of st.async: 0.1 us slower.)
//   us, ranges -> clusters (CTAs)   M 1                   M 16                  M 24 (ranges: gemm_wt)
//   1024 x 8192                      4.6 -> 3.4 (2)        5.1 -> 3.8            4.6 -> 4.5
//   2048 x 5120                      5.2 -> 4.1 (3)        6.6 -> 4.5            6.9 -> 5.2
//   8192 x 1280                      6.2 -> 4.8 (16)       9.1 -> 5.3            9.9 -> 5.9
//   8192 x 7424                     10.1 -> 10.1 (4)      12.0 -> 10.6          15.8 -> 11.1
//   3712 x 8192                      6.9 -> 7.2 (3)        8.4 -> 7.8 (3)       11.0 -> 8.0 (4)
// The last two stay in ranges at one token (ts_cut).
// What is left of 1024 x 8192 at M 1, in cycles from the end of the kernel before: 860 the tokens' way through L2, 1400
// the MMAs of four units (22 each), 350 the last fold, 900 the cluster's sum, 450 the exit.
//
// Warp roles (768 threads), joined by mbarrier rings:
//   12      conversion   warp (q, team): chunk of 32 columns q of both tiles, units u = team (mod 3);
//                        A slot = team                             raw_full -> unit_full, raw_empty
//   8       fold         warp (q, tile): tcgen05.ld of the unit's sums, fold into registers; the
//                        epilogue at the end of a segment          mma_done -> unit_full
//   1       MMA issue    converged warp, elected lane (SUB: two, units in turn)
//                                                                  unit_full -> mma_done
//   1       sums         sum_k x of every token with mma.sync against a constant operand (not SUB)
//                                                                  unit_full -> mma_done
//   1       TMA          tokens; zero points but in MODE 1 and SUB mma_done -> unit_full
//   1       TMA          packed words, scales; zero points in MODE 1 and SUB
//                                                                  raw_empty -> raw_full
// MODE 0 is the dense linear.  The other modes are the expert GEMMs of a fused-MoE layer with few rows
// per expert; a tile is (row block, slab) and a block's rows belong to one expert:
//   MODE 1  gate_up: a tile's units are those of 256 gate columns, then those of the matching up
//           columns.  The gate sums wait in shared memory; epilogue act[row] = silu(gate) * up.  Rows of
//           x by index (TMA gather) from the permuted list.  Direct form (no permutation): block b is
//           pair b alone.  (128 gate and 128 up columns side by side in a unit, as two boxes of 64-byte
//           rows, took 2 to 7 us longer at every batch size: the words arrive slower.)
//   MODE 2  down: rows of act; epilogue pair_out[pair] = routed weight * D, rounded as in the other expert
//           kernels, for a sum over the slots afterwards.  Direct form: a pair without an expert here
//           (negative id) gets a row of zeros.
// SPLIT, direct form: MODE 1 as a dense layer, every CTA with the same units of gate and up.  MODE 2: the CTAs of a
// cluster have the slots of a token, each the whole matrix, and add the rounded rows in slot order, so that no kernel for
// the sum follows.  Each where the estimates say so.  Experts without the router, ranges and a kernel for the sum -> now:
// 128 of 2048 x 768, one token, top-8 16.8 -> 14.5 us (gate_up in ranges, on clusters 15.3); 64 of 2048 x 1024, top-4 14.8
// -> 13.2; 64 of 2048 x 768, two tokens, top-4 16.2 -> 14.1.  (With zero points subtracted in the conversion 0.1 us slower,
// and other roundings than through the permutation.)
//
// unit_full counts the conversion warps, the announcement of the tokens and the fold warps of the unit
// NDB before, whose accumulators the MMAs overwrite.  mma_done counts the MMA warp's commit and the
// sums warp: it frees the x stage and the A slot and hands accumulators and sums to the fold warps.
//
// Shared-memory rings without a barrier of their own: scales / zero points and token sums have 16
// slots.  A slot is overwritten by unit u + 16 at the earliest after conversion of unit u + 16 - 9
// (the raw ring), which needs the MMAs of three units before, which need the folds of up to four before
// that: unit u has long been folded.
//
// TMEM columns: D[buffers][2 tiles][16 or 32 tokens] at 0 .. 127, A[3 slots][2 tiles][8 steps][8] at 128 .. 511.
// Lane 32 q + 8 i + g of tile t holds column
// 128 t + 32 q + 8 (g / 2) + 2 i + g % 2 of the slab.  Every wait is bounded (tc_ptx.cuh).
//
// Measured (B200, K x N, first replays of a cool GPU; a second later, at the power limit, 8192 x 59136 takes 45.6 us at M 4
// and 49.8 at M 16; before: mma.sync streaming kernel up to M = 8, its decode-layout copy in
// brackets, an earlier form of this kernel above; K-major copy in brackets):
//   8192 x 59136   M 4: 56.2 (50.6) -> 41.6 us, 5.8 TB/s of int4    M 16: 82.1 (64.1) -> 45.3 us
//   29568 x 8192   M 4: 35.0 (30.2) -> 24.7 us                        M 16: 40.0 (43.7) -> 27.3 us
//   8192 x 10240   M 4: 17.2 (16.0) -> 11.9 us                        M 16: 20.0 (22.9) -> 13.3 us
//   1024 x 8192    M 1: 7.6 -> 4.6 us
//   M 24 and 32 (before: gemm_wt): 8192 x 59136 76 -> 53 and 76 -> 56 us; 29568 x 8192 M 32 41 -> 36
//   groups of 64 (before: mma.sync streaming kernel; M 24: two calls of 16 rows)
//   8192 x 59136   M 4: 69.2 -> 43.2 us, M 16: 106.8 -> 50.5, M 24: 113 -> 78;  4096 x 11040  M 20: 19.6 -> 13.2
// The instructions of the some 36 waits a unit takes are a fifth of all, so a wait for a complete phase is one probe,
// one vote and one branch (mbar_wait_warp): 8192 x 59136 at M 8 55.4 -> 53.3 us, 8192 x 10240 groups of 64 at M 8 13.27
// -> 13.07, experts of 128 x 2048 x 768 at 64 tokens 83.2 -> 80.6 (that step alone; the fold warps differ, see there).
// Tried and taken back: 16 fold warps of 16 tokens each for M 32 (64 registers a thread: 56 -> 64 us); two warps for the
// token sums, or sums in four chains (nothing, or 1 % slower on short layers); a team per half unit, with two
// halves of A slots each (the conversion warps then get in each other's way, 55 -> 59 us at M 16); all MMAs of a unit in
// one asm block, predicated arrivals (no difference); the sum over a token's slots by the warp that stores the last
// of its rows (fences and counters at the end of every tile: 80 -> 99 us at 64 tokens, 16.4 -> 17.0 at one).
// Bound by HBM on the long layers (6.45 TB/s allow 712 cycles a unit; some 810 at M = 16, 46 300 of a CTA with 50 units,
// ncu), by start-up and hand-over (~5 us) on the short ones.
// Experts without the router, 128 of 2048 x 768, 8 per token (before: mma.sync kernels on the decode copies;
// replayed graph, cool): T 1: 22.9 -> 16.2 us, T 16: 71.0 -> 53.8, T 64: 101.9 -> 72.2, T 128: 110.7 -> 92.1.  At T = 64 all
// 302 MB of int4 words are read, 48 us at the HBM rate; a block of 8 rows costs the conversion of a
// whole matrix, which is what bounds it.
#include <cmath>

#include "common.cuh"
#include "handover.cuh"
#include "tc_ptx.cuh"

namespace awq {

namespace {

using namespace tc;
using handover::Work;

constexpr int kTsBN = 256, kTsBK = 128;
constexpr int kTsRawBytes = kTsBK * kTsBN / 2;         // 16384
constexpr int kTsScaleBytes = kTsBN * 2, kTsZeroBytes = kTsBN / 2;  // of one group
constexpr int kTsSzRing = 16;
constexpr int kTsUnits = 8;                            // x stages, unit barriers
constexpr int kTsTmemCols = 512;

// MT: tokens (4, 8, 16, 32).
constexpr int kTsTeams = 3;                            // sets of four conversion warps = A slots
constexpr int kTsColD = 128;                           // TMEM columns of the accumulators
constexpr int kTsCvWarps = 4 * kTsTeams;
static_assert(kTsColD + kTsTeams * 128 <= kTsTmemCols, "TMEM columns");
// What depends on the quantisation group (128 or 64: one or two of a unit) and on the tokens.
template <int MT, int MODE, int GROUP, bool SPLIT = false>
struct TsCfg {
  static constexpr int G = kTsBK / GROUP;              // groups of a unit
  static constexpr int NT = MT <= 16 ? 16 : 32;        // tokens of the B operand
  static constexpr int kFoldWarps = 8;
  static constexpr int kFold0 = kTsCvWarps, kIssue = kFold0 + kFoldWarps;
  // the conversion subtracts the zero points: no token sums
  static constexpr bool SUB = (SPLIT && MODE == 0) || MT > 16 || (MT == 16 && GROUP == 64);
  // Scales and zero points by plain bulk copies (TsRow).  Groups of 64 need twice as many: up to 16 tokens 4096 x 11040 at
  // M 16 took 10.4 -> 10.7 us with them, at M 24 12.4 -> 11.5.
  static constexpr bool BULK = SPLIT && MODE == 0 && (GROUP == 128 || MT > 16);
  static constexpr int kIssueWarps = SUB ? 2 : 1;
  static constexpr int kSum = kIssue + kIssueWarps, kXWarp = kSum + (SUB ? 0 : 1), kRaw = kXWarp + 1;
  static constexpr int kThreads = 32 * (kRaw + 1);     // 768
  static constexpr int kX = NT * kTsBK * 2;            // bytes of an x stage
  // Stages of packed words.  A team must know that a stage's last filling has landed when it waits for the next one,
  // or the parity of the filling before that could pass for it: it read the last one itself (a multiple of the teams), or
  // has seen the MMAs of unit u - 6 complete, which had to wait for the folds up to unit u - 6 - NDB.
  static constexpr int NRAW = SPLIT && MT > 16 ? 6 : G == 1 ? 9 : MT <= 16 ? 8 : 7;
  static constexpr int NDB = kTsColD / (2 * G * NT);   // units with accumulators of their own
  static constexpr int kScales = G * kTsScaleBytes, kZeros = G * kTsZeroBytes;
  static constexpr int kSz = kScales + kZeros;         // scales, zero words
  static constexpr int kSums = SUB ? 0 : G * NT * 4;
  // SPLIT: a fold warp's sums leave in pieces of up to half of the tokens, each summed by one CTA of the cluster
  static constexpr int kHalves = MT >= 8 ? 2 : 1, kPieceTokens = MT / kHalves, kPieces = 8 * kHalves;
  static constexpr int kPieceBytes = kPieceTokens * 32 * 4;
  static constexpr int kRecvPieces = 20;  // (pieces that a CTA sums) x (CTAs of the cluster), at most
  static constexpr int kRecv = SPLIT ? kRecvPieces * kPieceBytes : 0;
  static constexpr int kSmem = 1024 + NRAW * kTsRawBytes + kTsUnits * kX + kTsSzRing * (kSz + kSums) + 512 + kRecv;
  // MODE 1 parks the gate sums of 16 tokens at most in static shared memory
  static_assert(kSmem + (MT <= 16 ? kFoldWarps * 16 * 32 * 4 : 0) <= 232448 - 512, "shared memory");
  static_assert(8 * (2 * NRAW + 2 * kTsUnits + kPieces / 2) <= 512, "barriers");
  static_assert(NRAW % kTsTeams == 0 || NRAW >= 2 * kTsTeams + NDB, "a stage's parity");
  static_assert(kTsSzRing >= NRAW + kTsTeams + NDB, "scale / sum ring too short");
};

struct TsParams {
  const __half* bias;
  __half* out;
  int M, N, K, KT, slabs;  // KT: units of one matrix (K / 128)
  int chunk;               // dense: units per CTA, 0: whole slabs strided
  // grouped modes
  union {
    const int32_t* sorted_ids;  // permuted flat pair ids, padding = numel; nullptr: direct form
    const __half* scales;       // BULK: [groups][N]
  };
  union {
    const int32_t* expert_ids;  // expert of every row block (direct: of every pair)
    const uint32_t* qzeros;     // BULK: [groups][N / 8]
  };
  const int32_t* num_post;     // permuted rows in use
  const float* topk_weights;
  int numel, topk, half_cols;
  int split;                   // SPLIT: CTAs of a cluster
  int max_split;               // CTAs a tile is split over at most, about
  float* partial;          // [CTA][MT][256] partial tiles handed over (MODE 1: gate and up, [CTA][2])
  handover::Flags flags;
};

// Pairs of fp32 values in 64-bit registers: one instruction for two FMAs.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ uint64_t pack2(uint32_t a, uint32_t b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ void lds_2x64(uint32_t addr, uint64_t& a, uint64_t& b) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void sts_float4(uint32_t addr, const float* v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
               : "memory");
}
template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[N]);
template <>
__device__ __forceinline__ void tmem_ld<4>(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr)
               : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld<8>(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// Routing tables are read through L2: MODE 2 reads them ahead of pdl_wait.
__device__ __forceinline__ int ts_expert(const TsParams& p, int tile) {
  return __ldcg(p.expert_ids + tile / p.slabs);
}
template <int MT, int MODE>
__device__ __forceinline__ Work ts_work(const TsParams& p) {
  if (MODE == 0) return Work(blockIdx.x, gridDim.x, p.slabs, p.KT, p.chunk);
  const int blocks = p.sorted_ids ? __ldcg(p.num_post) / MT : p.numel;
  const int KT = MODE == 1 ? 2 * p.KT : p.KT, tiles = blocks * p.slabs;
  const int even = (tiles * KT + (int)gridDim.x - 1) / (int)gridDim.x;
  const int least = (KT + p.max_split - 1) / p.max_split;
  return Work(blockIdx.x, gridDim.x, tiles, KT, max(1, max(even, least)));
}

// SPLIT: a cluster's tile.  MODE 2: the CTAs of a cluster have the slots of a token, whole.
template <int MODE>
__device__ __forceinline__ Work ts_split_work(const TsParams& p, int rank, int kt) {
  const int cluster = blockIdx.x / p.split;
  if (MODE == 0)
    return Work::range(cluster * p.KT + rank * p.KT / p.split, cluster * p.KT + (rank + 1) * p.KT / p.split, p.KT);
  if (MODE == 1) return Work::range(cluster * 2 * kt, (cluster + 1) * 2 * kt, 2 * kt);
  const int token = cluster / p.slabs, tile = (token * p.split + rank) * p.slabs + cluster - token * p.slabs;
  return Work::range(tile * p.KT, (tile + 1) * p.KT, p.KT);
}

// BULK: scales and zero words of 256 columns of a group, of which `cols` exist, for plain bulk copies: they are contiguous.
// What a copy leaves as it is belongs to columns that are not stored.  Maps -> copies: the host needs two tensor maps less, 0.1
// us of a call (eager, 2048 x 5120 at M 1 4.78 -> 4.72 us, which is less than runs differ by; replayed, clusters in groups of
// 128 are 0.2 to 0.9 % slower, 4.21 -> 4.23); groups of 64 at M 24, 4096 x 11040 12.4 -> 11.7 (with maps some runs take
// 11.5), eight other shapes of 17 to 32 tokens +- 0.9 %.  Long layers keep their maps: 8192 x 59136 at M 32 55 -> 58.
struct TsRow {
  const __half* scales;
  const uint32_t* zeros;
  uint32_t cols;
  __device__ __forceinline__ TsRow(const TsParams& p, int column, int group)
      : scales(p.scales + (size_t)group * p.N + column),
        zeros(p.qzeros + (size_t)group * (p.N / kPack) + column / kPack),
        cols((uint32_t)min(kTsBN, p.N - column)) {}
};

// A load stream's walk over the CTA's units: the weight rows / group row of every unit, and the column
// slab.  The expert of the next matrix is fetched while the current one is loaded.
template <int MODE>
struct TsWalk {
  const TsParams& p;
  const Work& work;
  const int kt, unit0;  // units of a matrix that the walk has, and the first
  int u = 0, seg = 0, k = 0, k_end = 0, tile = 0, slab = 0;
  int expert = 0, expert_next = 0;
  bool fetched = false;
  __device__ __forceinline__ TsWalk(const TsParams& p_, const Work& w_, int kt_, int unit0_)
      : p(p_), work(w_), kt(kt_), unit0(unit0_) {}
  // Positions on unit u; returns whether a new tile begins.  MODE 1: k counts gate units, then up.
  __device__ __forceinline__ bool settle() {
    if (k != k_end) return false;
    tile = work.tile_id(seg);
    k = work.k_begin(seg);
    k_end = work.k_end(seg++);
    slab = MODE == 0 ? tile : tile - tile / p.slabs * p.slabs;
    if (MODE != 0) {
      if (!fetched) {
        expert_next = ts_expert(p, tile);
        fetched = true;
      }
      expert = max(expert_next, 0);  // absent (negative): any matrix, nothing of it is used
      if (seg < work.segs) expert_next = ts_expert(p, work.tile_id(seg));
    }
    return true;
  }
  __device__ __forceinline__ void next() {
    ++u;
    ++k;
  }
  __device__ __forceinline__ bool up() const { return MODE == 1 && k >= kt; }
  __device__ __forceinline__ int unit() const { return unit0 + (up() ? k - kt : k); }  // inside the matrix
  __device__ __forceinline__ int column() const { return slab * kTsBN + (up() ? p.half_cols : 0); }
};

// MARKS: partial tiles are handed over with a token beside every two sums, without flags (ts_marks).
template <int MT, int MODE, int GROUP, bool SPLIT, bool MARKS = false>
__global__ void __launch_bounds__((TsCfg<MT, MODE, GROUP, SPLIT>::kThreads), 1)
// map_s, map_z: not read where BULK
gemm_ts_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_s,
               const __grid_constant__ CUtensorMap map_z, const __grid_constant__ CUtensorMap map_x,
               const TsParams p) {
  using Cfg = TsCfg<MT, MODE, GROUP, SPLIT>;
  constexpr int NT = Cfg::NT, G = Cfg::G, NDB = Cfg::NDB, NRAW = Cfg::NRAW, kSz = Cfg::kSz, kTsXBytes = Cfg::kX;
  constexpr int kTsFoldWarps = Cfg::kFoldWarps, kTsFold0 = Cfg::kFold0, kTsIssue = Cfg::kIssue, kIssueWarps = Cfg::kIssueWarps;
  constexpr bool SUB = Cfg::SUB, kRawZeros = MODE == 1 || SUB;  // zero points with the packed words
  constexpr int kTsSum = Cfg::kSum, kTsX = Cfg::kXWarp, kTsRaw = Cfg::kRaw;
  constexpr int kScales = Cfg::kScales, kZeros = Cfg::kZeros, kSums = Cfg::kSums;
  extern __shared__ uint8_t smem_raw[];
  __shared__ volatile int s_abort;
  __shared__ uint32_t s_tmem_base;
  __shared__ float s_gate[MODE == 1 ? kTsFoldWarps * MT * 32 : 1];  // gate sums during the up units

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t raw_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t x_base = raw_base + NRAW * kTsRawBytes;
  const uint32_t sz_base = x_base + kTsUnits * kTsXBytes;
  const uint32_t sx_base = sz_base + kTsSzRing * kSz;
  const uint32_t bar_base = sx_base + kTsSzRing * kSums;
  auto raw_full = [&](int s) { return bar_base + 8 * s; };
  auto raw_empty = [&](int s) { return bar_base + 8 * (NRAW + s); };
  // unit u may be multiplied: converted, tokens and zero points landed, and its accumulators free (the
  // fold warps have read unit u - NDB)
  auto unit_full = [&](int u) { return bar_base + 8 * (2 * NRAW + (u & (kTsUnits - 1))); };
  auto mma_done = [&](int u) { return bar_base + 8 * (2 * NRAW + kTsUnits + (u & (kTsUnits - 1))); };
  auto unit_phase = [&](int u) { return (uint32_t)((u / kTsUnits) & 1); };

  // With 32 tokens tensor memory is asked for first and the warp of the packed words, which only tells that its barriers
  // are set up, waits for nobody: M 24 on 8192 x 7424 11.3 -> 11.0 us, 3712 x 8192 8.3 -> 8.0, M 32 on 8192 x 10240 13.95 -> 13.7.  The smaller forms
  // compiled 1 to 3 % worse that way (experts of 128 x 2048 x 768, top-8, 64 tokens 72.4 -> 74.0).
  constexpr bool kFree = MT > 16;
  auto alloc = [&]() {
    if (warp == kTsIssue) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(&s_tmem_base)),
                   "r"((uint32_t)kTsTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  };
  if (kFree) alloc();
  // The dependents of MODE 1 read the routing tables before their own pdl_wait: they may start once
  // every CTA here knows that the kernels that wrote the tables are complete.
  if (MODE == 1) pdl_wait();
  pdl_launch_dependents();
  const int rank = SPLIT ? blockIdx.x % p.split : 0;
  // MODE 1, SPLIT: this CTA's units of gate, then the same of up
  const int unit0 = SPLIT && MODE == 1 ? rank * p.KT / p.split : 0;
  const int kt = SPLIT && MODE == 1 ? (rank + 1) * p.KT / p.split - unit0 : p.KT;
  const Work work = SPLIT ? ts_split_work<MODE>(p, rank, kt) : ts_work<MT, MODE>(p);
  // SPLIT: barrier and shared memory of the n-th piece that this CTA sums, partial sums of CTA `from`
  auto recv_full = [&](int n) { return bar_base + 8 * (2 * NRAW + 2 * kTsUnits + n); };
  auto recv_at = [&](int n, int from) { return bar_base + 512 + (n * p.split + from) * Cfg::kPieceBytes; };
  // quads of tokens of a piece that the call has
  auto piece_quads = [&](int half) {
    return min(Cfg::kPieceTokens / 4, max(0, (p.M - half * Cfg::kPieceTokens + 3) / 4));
  };

  // packed words, scales, MODE 1 also zero points (raw warp, converged: an elected lane issues; TMAs
  // of a lane that loops alone take it longer)
  TsWalk<MODE> raw(p, work, kt, unit0);
  int raw_s = 0;
  uint32_t raw_phase = 0;
  auto load_raw = [&]() {
    raw.settle();
    const uint32_t bar = raw_full(raw_s), dst = raw_base + raw_s * kTsRawBytes;
    const uint32_t sz = sz_base + (raw.u & (kTsSzRing - 1)) * kSz;
    const int column = raw.column(), row = raw.expert * p.K + raw.unit() * kTsBK;
    const int grp = (raw.expert * p.KT + raw.unit()) * G;
    if constexpr (Cfg::BULK) {
      const TsRow of(p, column, grp);
      if (elect_one()) {
        mbar_arrive_expect_tx(bar, kTsRawBytes + G * (of.cols * 2 + (kRawZeros ? of.cols / 2 : 0)));
        tma_load_2d(dst, &map_w, column / kPack, row, bar);
#pragma unroll
        for (int h = 0; h < G; ++h) {
          bulk_load(sz + h * kTsScaleBytes, of.scales + (size_t)h * p.N, of.cols * 2, bar);
          if (kRawZeros)
            bulk_load(sz + kScales + h * kTsZeroBytes, of.zeros + (size_t)h * (p.N / kPack), of.cols / 2, bar);
        }
      }
    } else if (elect_one()) {
      mbar_arrive_expect_tx(bar, kTsRawBytes + kScales + (kRawZeros ? kZeros : 0));
      tma_load_2d(dst, &map_w, column / kPack, row, bar);
      tma_load_2d(sz, &map_s, column, grp, bar);
      if (kRawZeros) tma_load_2d(sz + kScales, &map_z, column / kPack, grp, bar);
    }
    raw.next();
    if (++raw_s == NRAW) {
      raw_s = 0;
      raw_phase ^= 1u;
    }
  };

  if (warp == kTsRaw) {
    if (kFree && lane == 0) s_abort = 0;
    if (lane < NRAW) {
      mbar_init(raw_full(lane), 1);
      mbar_init(raw_empty(lane), 4);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      fence_proxy_async();
    }
    __syncwarp();
    if (kFree) asm volatile("bar.arrive 1, %0;" ::"n"(Cfg::kThreads) : "memory");
    if (SPLIT && kFree) cluster_arrive();
    // the first packed words are on their way before anyone else is through the prologue; no
    // kernel writes weights, so they need not wait for the kernel before this one
    for (int i = 0; i < 3 && raw.u < work.count; ++i) load_raw();
  }
  if (warp == kTsX) {
    if (!kFree && lane == 0) s_abort = 0;
    if (lane < kTsUnits) {
      // conversion warps, announcement of the tokens, fold warps (none before unit NDB)
      mbar_init(unit_full(lane), 4 + 1 + kTsFoldWarps);
      mbar_init(mma_done(lane), SUB ? 1 : 2);  // commit, sums warp
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (SPLIT && lane * p.split + rank < Cfg::kPieces) {  // piece lane * split + rank is this CTA's
      const int quads = piece_quads((lane * p.split + rank) / 8);
      mbar_init(recv_full(lane), 2);  // the bytes of the other CTAs, the warp here that has the piece
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      mbar_arrive_expect_tx(recv_full(lane), (p.split - 1) * (MODE == 0 ? quads * 512 : 256));
    }
  }
  __syncwarp();
  if (!kFree) alloc();
  tc_fence_before();
  if (!kFree) __syncthreads();
  else if (warp != kTsRaw) asm volatile("bar.sync 1, %0;" ::"n"(Cfg::kThreads) : "memory");
  tc_fence_after();
  if (SPLIT && (!kFree || warp != kTsRaw)) cluster_arrive();  // awaited ahead of the first store into another CTA
  const uint32_t tmem = s_tmem_base;

  if (warp == kTsRaw) {
    // ------------------------------------------------------------------ packed words, scales
    bool ok = true;
    while (raw.u < work.count) {
      // the first trip round the ring finds it empty
      if (raw.u >= NRAW) ok = mbar_wait_warp(raw_empty(raw_s), raw_phase ^ 1u, &s_abort, 21);
      if (!ok) break;
      load_raw();
    }
  } else if (warp == kTsX) {
    // ------------------------------------------------------------------ tokens (zero points)
    pdl_wait();  // the activations may be the output of the kernel before this one
    TsWalk<MODE> x(p, work, kt, unit0);
    bool ok = true;
    int row = 0, fid_next = -1, quads = MT / 4;
    int rows[MODE == 1 ? MT : 1];  // MODE 1: the block's rows of x
    auto block_fid = [&](int seg) {  // lane m: pair in row m of a segment's block
      const int block = work.tile_id(seg) / p.slabs;
      return lane < MT ? __ldcg(p.sorted_ids + block * MT + lane) : p.numel;
    };
    while (x.u < work.count && ok) {
      if (x.settle() && MODE != 0) {
        const int block = x.tile / p.slabs;
        if (MODE == 2) row = p.sorted_ids != nullptr ? block * MT : block;  // of act
        if (MODE == 1 && p.sorted_ids == nullptr) row = block / p.topk;  // the pair's token
        if (MODE == 1 && p.sorted_ids != nullptr) {
          const int fid = fid_next >= 0 ? fid_next : block_fid(x.seg - 1);
          if (x.seg < work.segs) fid_next = block_fid(x.seg);
          const int token = fid < p.numel ? fid / p.topk : 0;  // padding: any row
#pragma unroll
          for (int m = 0; m < MT; ++m) rows[m] = __shfl_sync(0xffffffffu, token, m);
          // valid rows come first; the tile's other rows keep what they hold, nothing of them is used
          quads = max(1, (__popc(__ballot_sync(0xffffffffu, fid < p.numel)) + 3) / 4);
        }
      }
      if (x.u >= kTsUnits)
        ok = mbar_wait_warp(mma_done(x.u - kTsUnits), unit_phase(x.u - kTsUnits), &s_abort, 22);
      if (!ok) break;
      const uint32_t bar = unit_full(x.u), dst = x_base + (x.u & (kTsUnits - 1)) * kTsXBytes;
      const uint32_t zdst = sz_base + (x.u & (kTsSzRing - 1)) * kSz + kScales;
      const int unit = x.unit(), zcol = x.column() / kPack, zrow = (x.expert * p.KT + unit) * G;
      if (elect_one()) {
        if (MODE == 1 && p.sorted_ids != nullptr) {
          mbar_arrive_expect_tx(bar, quads * (4 * kTsBK * 2));
#pragma unroll
          for (int m = 0; m < MT; m += 4)
            if (m < 4 * quads)
#pragma unroll
              for (int h = 0; h < 2; ++h)
                tma_gather4(dst + h * (kTsXBytes / 2) + m * 128, &map_x, unit * kTsBK + h * 64, rows[m],
                            rows[m + 1], rows[m + 2], rows[m + 3], bar);
        } else {
          mbar_arrive_expect_tx(bar, (kRawZeros ? 0 : kZeros) + kTsXBytes);
          tma_load_3d(dst, &map_x, 0, row, 2 * unit, bar);
          if (!kRawZeros) tma_load_2d(zdst, &map_z, zcol, zrow, bar);
        }
      }
      __syncwarp();
      x.next();
    }
    // The commits of the last units arrive asynchronously and nobody else waits for all of them: see
    // them land before the CTA may exit.
    for (int u = work.count > kTsUnits ? work.count - kTsUnits : 0; u < work.count && ok; ++u)
      ok = mbar_wait(mma_done(u), unit_phase(u), &s_abort, 22);
  } else if (!SUB && warp == kTsSum) {
    // ------------------------------------------------------------------ token sums
    // x tile as the A operand of mma.sync (16 tokens x 16 k), every B element 2^-24: each column of
    // the result is 2^-24 * sum_k x, in the scaling of the weight tiles' accumulators
    const int row = (lane & 7) + 8 * ((lane >> 3) & 1), kc = lane >> 4;
    bool ok = true;
    for (int u = 0; u < work.count && ok; ++u) {
      ok = mbar_wait_warp(unit_full(u), unit_phase(u), &s_abort, 23);
      if (!ok) break;
      const uint32_t xt = x_base + (u & (kTsUnits - 1)) * kTsXBytes;
#pragma unroll
      for (int h = 0; h < G; ++h) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks = h * (8 / G); ks < (h + 1) * (8 / G); ++ks) {
          uint32_t a[4];
          const int c = 2 * (ks & 3) + kc;
          ldmatrix_x4(xt + (ks >> 2) * (NT * 128) + row * 128 + ((c ^ (row & 7)) << 4), a);
          mma16816(acc, a, 0x00010001u, 0x00010001u, acc);
        }
        if ((lane & 3) == 0) {
          const uint32_t dst = sx_base + (u & (kTsSzRing - 1)) * kSums + (h * NT + (lane >> 2)) * 4;
          asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst), "f"(acc[0]) : "memory");
          asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst + 32), "f"(acc[2]) : "memory");
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(mma_done(u));
    }
  } else if (warp >= kTsIssue && warp < kTsIssue + kIssueWarps) {
    // ------------------------------------------------------------------ MMA issue
    // One barrier per unit, the next unit's probed under this one's MMAs.  SUB: two warps issue units in turn, so that
    // one's wait and loop run under the other's MMAs (M 32 on 8192 x 59136: 66.6 -> 64.4 us, with 16 fold warps then).  (A
    // second issuing warp, one per tile, made it slower: 54 against 50 us at M = 16.)  D fp32, A / B fp16,
    // both K-major, N = NT tokens, M = 128 columns.
    constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | (8u << 24);
    constexpr uint32_t half = NT * 128 / 16;
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
    const uint64_t desc0 = make_desc(__shfl_sync(0xffffffffu, x_base, 0), 16, 1024);
    bool ok = true, ready = false;
    int slot = warp - kTsIssue;
    for (int u = slot; u < work.count; u += kIssueWarps) {
      if (!ready) {
        ok = mbar_wait_warp(unit_full(u), unit_phase(u), &s_abort, 24);
        if (!ok) break;
      }
      tc_fence_after();
      const uint64_t dx = desc0 + (uint32_t)(u & (kTsUnits - 1)) * (kTsXBytes / 16);
      const uint32_t dcol = tmem_u + (uint32_t)(u & (NDB - 1)) * (G * 2 * NT);
      const uint32_t acol = tmem_u + kTsColD + slot * 128;
      bool r = false;
      if (elect_one()) {
        r = mbar_test(unit_full(u + kIssueWarps), unit_phase(u + kIssueWarps));
#pragma unroll
        for (int step = 0; step < 8; ++step) {
          const uint64_t db = dx + (step >> 2) * half + (step & 3) * 2;
          const uint32_t d = dcol + step / (8 / G) * (2 * NT), more = step % (8 / G) ? 1u : 0u;
          umma_f16_ts(d, acol + step * 8, db, idesc, more);
          umma_f16_ts(d + NT, acol + 64 + step * 8, db, idesc, more);
        }
        umma_commit(mma_done(u));
      }
      slot += kIssueWarps;
      if (slot >= kTsTeams) slot -= kTsTeams;
      ready = __any_sync(0xffffffffu, r);
    }
  } else if (warp < kTsCvWarps) {
    // ------------------------------------------------------------------ conversion warps
    const int q = warp & 3, team = warp >> 2;
    {
      const uint32_t lane_q = (uint32_t)(q * 32) << 16;
      // ldmatrix: matrix m = lane / 8 of the four holds rows 8 m .. 8 m + 7 of 32; after the transposed load
      // thread (g, t) has rows 2 t and 2 t + 1 of halfword column g in a register of each.  Rows of 128 B,
      // 16-byte chunk c at position c ^ (row % 8).
      const uint32_t off0 = (uint32_t)(lane * 128 + ((q ^ (lane & 7)) << 4));
      const uint32_t z_addr = sz_base + kScales + (uint32_t)(4 * q + (lane >> 3)) * 4;
      const uint32_t off1 = (uint32_t)(lane * 128 + (((q + 4) ^ (lane & 7)) << 4));
      bool ok = true;
      int s = team;
      uint32_t phase = 0;
      for (int u = team; u < work.count; u += kTsTeams) {
        ok = mbar_wait_warp(raw_full(s), phase, &s_abort, 26);
        if (!ok) break;
        const uint32_t raw = raw_base + s * kTsRawBytes;
        const uint32_t a_slot = tmem + lane_q + kTsColD + team * 128;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          uint32_t w[4][4];
#pragma unroll
          for (int pr = 0; pr < 4; ++pr) ldmatrix_x4_trans(raw + (t ? off1 : off0) + pr * 4096, w[pr]);
          if (t == 0) {
            // the MMAs that read this A slot last must be complete
            if (u >= kTsTeams)
              ok = mbar_wait_warp(mma_done(u - kTsTeams), unit_phase(u - kTsTeams), &s_abort, 27);
            if (!ok) break;
            tc_fence_after();
          }
          uint32_t zz[SUB ? G : 1][4];  // SUB: zero points of this lane's four columns, in place like the weights
          if constexpr (SUB) {
#pragma unroll
            for (int gi = 0; gi < G; ++gi) {
              const uint32_t zw = lds32(z_addr + (u & (kTsSzRing - 1)) * kSz + gi * kTsZeroBytes + t * (kTsZeroBytes / 2));
              const uint32_t z2 = prmt(zw, zw, (lane & 4) ? 0x3232u : 0x1010u), zh = z2 >> 8;
              zz[gi][0] = z2 & 0x000F000Fu;
              zz[gi][1] = z2 & 0x00F000F0u;
              zz[gi][2] = zh & 0x000F000Fu;
              zz[gi][3] = zh & 0x00F000F0u;
            }
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {  // 64 rows each, eight by eight
            // Logic and shifts take two cycles a warp and scheduler: 320 of them a unit are what
            // bounds the kernel beside HBM.  (The shift as a multiplication on the FMA pipe, which is
            // idle here, measured 7 % slower: mul.hi takes four cycles.)
            uint32_t frag[2][16];  // [lane half of the quarter][2 * eight rows + i odd]
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const uint32_t r = w[2 * h + (c >> 2)][c & 3], rh = r >> 8;
#pragma unroll
              for (int i = 0; i < 4; ++i)
              {
                uint32_t v = ((i & 2) ? rh : r) & ((i & 1) ? 0x00F000F0u : 0x000F000Fu);
                if constexpr (SUB) v = as_u32(__hsub2(as_half2(v), as_half2(zz[h * G / 2][i])));
                frag[i >> 1][2 * c + (i & 1)] = v;
              }
            }
            tmem_st_16x128b(a_slot + t * 64 + h * 32, frag[0]);
            tmem_st_16x128b(a_slot + (16u << 16) + t * 64 + h * 32, frag[1]);
          }
        }
        if (!ok) break;
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(unit_full(u));
          mbar_arrive(raw_empty(s));
        }
        s += kTsTeams;
        if (s >= NRAW) {
          s -= NRAW;
          phase ^= 1u;
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ fold + epilogue
    const int fold = warp - kTsFold0, q = warp & 3, tile = fold >> 2;
    const uint32_t lane_q = (uint32_t)(q * 32) << 16;
    const int g = lane & 7, i = lane >> 3;
    const bool odd = (g & 1) != 0;
    const int chunk_col = tile * 128 + 32 * q;                     // first column of this warp's 32
    const int col = chunk_col + 8 * (g >> 1) + 2 * i + (g & 1);    // this lane's column of the slab
    const uint32_t s_addr = sz_base + (uint32_t)col * 2;
    const uint32_t z_addr = sz_base + kScales + (uint32_t)(col >> 3) * 4;
    const int z_shift = 16 * (g & 1) + 4 * i;
    // odd i hold nibbles kept in place (16 q), so their zero point is 16 z.  -zf * z from the nibble as
    // the low bits of 2^23 + z (exact), without an integer conversion.
    const float zf = (i & 1) ? -16.f : -1.f, zc = zf * -8388608.f;
    const float unscale = (i & 1) ? 1048576.f : 16777216.f;        // undo 2^-20 / 2^-24
    const uint32_t d_addr = tmem + lane_q + (uint32_t)(tile * NT);
    float* gate = s_gate + (MODE == 1 ? fold * (MT * 32) + lane : 0);
    // the first units find their accumulators free
    if (lane == 0)
      for (int u = 0; u < NDB; ++u) mbar_arrive(unit_full(u));
    pdl_wait();  // orders this thread's writes after the kernel before this one
    const unsigned long long token = p.flags.token;
    unsigned long long* flag = p.flags.at(blockIdx.x, fold);  // this warp's
    // After a wait that gave up nothing more is folded.  In which form the loop over the units says so decides how it
    // compiles.  The first figures are with one vote and going on.  Groups of 128 take one vote and leave (us): 8192 x
    // 59136 at M 8 51.5 -> 50.2, M 16 56.2 -> 53.7; 2304 x 8288 at M 16 7.30 -> 6.74; 1152 x 2048 at M 1 4.22 -> 4.14;
    // experts of 128 x 2048 x 768, top-8, 64 tokens 81.0 -> 79.3.  Groups of 64 differ by tokens: up to 4 a probe and a
    // vote, then they leave (8192 x 59136 at M 1 49.0 -> 48.4; one vote 50.4); up to 8 as groups of 128 (52.8 at M 8; two
    // 53.5); up to 16 a probe and a vote, and they go on (2304 x 8288 8.45 -> 7.99; leaving 8.20, with one vote 8.11).
    constexpr bool kOneVote = GROUP == 128 || MT == 8, kStay = GROUP == 64 && MT == 16;
    bool ok = true;
    int u = 0;
    // MODE 2: tiles are walked down one by one, so a segment's block and slab need no division, and pairs are fetched a
    // segment ahead: the address of their weights waits for them.  Experts of 128 x 2048 x 768, top-8, 128 tokens 94.5 ->
    // 93.1 us, 500 tokens 189 -> 184.
    int block_next = 0, slab_next = 0, fid_next = p.numel;
    auto pair_of = [&](int block) {  // lane m: pair in row m
      if (lane >= MT) return p.numel;
      return p.sorted_ids != nullptr ? __ldcg(p.sorted_ids + block * MT + lane) : (lane == 0 ? block : p.numel);
    };
    if (MODE == 2 && work.segs > 0) {
      block_next = work.tile_id(0) / p.slabs;
      slab_next = work.tile_id(0) - block_next * p.slabs;
      fid_next = pair_of(block_next);
    }
    for (int seg = 0; seg < work.segs; ++seg) {
      const int id = work.tile_id(seg), kb = work.k_begin(seg), ke = work.k_end(seg);
      const int block = MODE == 0 ? 0 : MODE == 2 ? block_next : id / p.slabs;
      const int slab = MODE == 0 ? id : MODE == 2 ? slab_next : id - block * p.slabs;
      // What the end of the segment needs, fetched ahead of its units.  MODE 2: lane m knows pair and
      // routed weight of row m.
      const int fid = fid_next;
      float fw = 0.f;
      int expert = 0;  // negative: an expert of another rank
      if (MODE == 1 || MODE == 2) expert = __ldcg(p.expert_ids + block);
      if (MODE == 2) {
        if (fid < p.numel) fw = __ldcg(p.topk_weights + fid);
        if (--slab_next < 0) {
          slab_next = p.slabs - 1;
          --block_next;
        }
        if (seg + 1 < work.segs) fid_next = pair_of(block_next);
      }
      uint64_t tot[MT / 2];
#pragma unroll
      for (int m = 0; m < MT / 2; ++m) tot[m] = 0ull;
      for (int k = ok || kStay ? kb : ke; k < ke; ++k, ++u) {
        if (MODE == 1 && k == kt && kb < kt) {  // gate complete: park its sums, start on up
#pragma unroll
          for (int m = 0; m < MT / 2; ++m) {
            const float2 v = unpack2(tot[m]);
            gate[(2 * m) * 32] = v.x;
            gate[(2 * m + 1) * 32] = v.y;
            tot[m] = 0ull;
          }
        }
        if constexpr (kOneVote) {
          ok = mbar_wait_warp(mma_done(u), unit_phase(u), &s_abort, 28);
        } else {
          if (ok || !kStay) ok = mbar_wait(mma_done(u), unit_phase(u), &s_abort, 28);
          ok = __all_sync(0xffffffffu, ok);
        }
        if (!ok) {
          if constexpr (kStay) continue;
          break;
        }
        tc_fence_after();
        const uint32_t dcol = d_addr + (uint32_t)(u & (NDB - 1)) * (G * 2 * NT);
        const uint32_t ring = (uint32_t)(u & (kTsSzRing - 1));
        // scale of this lane's column in a group
        auto scale = [&](int h) {
          uint16_t sh;
          asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sh) : "r"(s_addr + ring * kSz + h * kTsScaleBytes));
          const float sc = __half2float(__ushort_as_half(sh));
          return pack2(sc, sc);
        };
        auto release = [&]() {  // the accumulators are in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(unit_full(u + NDB));
        };
        if constexpr (SUB) {  // sixteen tokens of a group at a time
          constexpr int LD = MT <= 16 ? MT : 16;
#pragma unroll
          for (int h = 0; h < G; ++h) {
            const uint64_t sc2 = scale(h);
#pragma unroll
            for (int m0 = 0; m0 < MT; m0 += LD) {
              uint32_t d[LD];
              tmem_ld<LD>(dcol + h * 2 * NT + m0, d);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              if (h == G - 1 && m0 + LD == MT) release();
#pragma unroll
              for (int m = 0; m < LD; m += 2) tot[(m0 + m) / 2] = fma2(sc2, pack2(d[m], d[m + 1]), tot[(m0 + m) / 2]);
            }
          }
        } else {
          uint32_t d[G][MT];
          uint64_t sc2[G], nz2[G];
#pragma unroll
          for (int h = 0; h < G; ++h) {
            tmem_ld<MT>(dcol + h * 2 * NT, d[h]);
            sc2[h] = scale(h);
            const uint32_t zw = lds32(z_addr + ring * kSz + h * kTsZeroBytes);
            const float nz = fmaf(__uint_as_float(((zw >> z_shift) & 0xFu) | 0x4B000000u), zf, zc);
            nz2[h] = pack2(nz, nz);
          }
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          release();
#pragma unroll
          for (int h = 0; h < G; ++h) {
            const uint32_t sx = sx_base + ring * kSums + h * (NT * 4);
#pragma unroll
            for (int m = 0; m < MT; m += 4) {
              uint64_t x01, x23;
              lds_2x64(sx + m * 4, x01, x23);
              tot[m / 2] = fma2(sc2[h], fma2(nz2[h], x01, pack2(d[h][m], d[h][m + 1])), tot[m / 2]);
              tot[m / 2 + 1] =
                  fma2(sc2[h], fma2(nz2[h], x23, pack2(d[h][m + 2], d[h][m + 3])), tot[m / 2 + 1]);
            }
          }
        }
      }
      // ---- end of the segment ----
      const bool valid = expert >= 0;
      float v[MT];
#pragma unroll
      for (int m = 0; m < MT / 2; ++m) {
        const float2 t = unpack2(tot[m]);
        v[2 * m] = t.x;
        v[2 * m + 1] = t.y;
      }
      if constexpr (SPLIT && MODE != 0) {
        // direct form: one row.  MODE 1: gate and up; MODE 2: the pair's weighted row, rounded as ever
        float a = gate[0], b = v[0];
        if (MODE == 2) {
          a = valid ? __half2float(__float2half_rn(v[0] * unscale * __shfl_sync(0xffffffffu, fw, 0))) : 0.f;
          b = 0.f;
        }
        cluster_wait();
        if (!ok) continue;  // a CTA that gave up sends nothing: who sums waits in vain, and stores nothing
        const int owner = fold % p.split, n = fold / p.split;
        const uint32_t dst = recv_at(n, rank) + lane * 8;
        if (owner == rank) {
          asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(dst), "f"(a), "f"(b) : "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(recv_full(n));
        } else {
          st_async_v2(map_rank(dst, owner), a, b, map_rank(recv_full(n), owner));
        }
        continue;
      }
      if constexpr (SPLIT) {
        constexpr int T = Cfg::kPieceTokens, Q = T / 4;
        cluster_wait();  // every CTA's barriers are set up
        if (!ok) continue;  // as above
#pragma unroll
        for (int half = 0; half < Cfg::kHalves; ++half) {
          const int piece = half * 8 + fold, owner = piece % p.split, n = piece / p.split, quads = piece_quads(half);
          if (owner == rank) {
#pragma unroll
            for (int m = 0; m < Q; ++m)
              if (m < quads) sts_float4(recv_at(n, rank) + lane * 16 + m * 512, &v[half * T + 4 * m]);
            __syncwarp();
            if (lane == 0) mbar_arrive(recv_full(n));
            continue;
          }
          const uint32_t dst = map_rank(recv_at(n, rank) + lane * 16, owner), bar = map_rank(recv_full(n), owner);
#pragma unroll
          for (int m = 0; m < Q; ++m)
            if (m < quads) st_async_v4(dst + m * 512, &v[half * T + 4 * m], bar);
        }
        continue;
      }
      // partial tile of CTA c: [MT][256], MODE 1: gate, then up
      constexpr int kTile = MT * kTsBN, kTiles = MODE == 1 ? 2 : 1;
      float* part = p.partial + (size_t)blockIdx.x * (kTiles * kTile) + chunk_col + lane;
      // MARKS: [MT / 2][256] pairs of sums with the launch's token beside each.  Whoever adds them reads until it sees the
      // token.
      constexpr int P = MT / 2, kMarked = P * kTsBN;
      uint4* marked = reinterpret_cast<uint4*>(p.partial) + (size_t)blockIdx.x * (kTiles * kMarked) + chunk_col + lane;
      if (MARKS && ke < work.KT) {
        uint4* dst = marked + (MODE == 1 && ke > p.KT ? kMarked : 0);
        const unsigned long long mark = ok && !s_abort ? token : 0ull;
#pragma unroll
        for (int m = 0; m < P; ++m) handover::store_marked(dst + m * kTsBN, pack2(v[2 * m], v[2 * m + 1]), mark);
        if (MODE == 1 && ke > p.KT && kb < p.KT) {
#pragma unroll
          for (int m = 0; m < P; ++m)
            handover::store_marked(marked + m * kTsBN, pack2(gate[2 * m * 32], gate[(2 * m + 1) * 32]), mark);
        }
        continue;
      }
      if (!MARKS && ke < work.KT) {  // another CTA holds the tile's last unit
        float* dst = part + (MODE == 1 && ke > p.KT ? kTile : 0);
#pragma unroll
        for (int m = 0; m < MT; ++m)
          if (MODE != 0 || m < p.M) dst[m * kTsBN] = v[m];
        if (MODE == 1 && ke > p.KT && kb < p.KT) {
#pragma unroll
          for (int m = 0; m < MT; ++m) part[m * kTsBN] = gate[m * 32];
        }
        __syncwarp();
        if (lane == 0 && ok && !s_abort) handover::raise_flag(flag, token);
        continue;
      }
      int gather = 0;  // CTAs before this one that share the tile
      if (kb > 0) {
        gather = blockIdx.x - id * work.KT / work.chunk;
        for (int c = 1 + lane; !MARKS && c <= gather; c += 32) {
          unsigned long long* theirs = flag - c * handover::kMaxWarps;
          uint32_t polls = 0;
          while (handover::read_flag(theirs) != token) {
            if (++polls >= kSpinLimit || s_abort) {
              s_abort = 1;
              atomicCAS(&g_tc_status, 0, 29);
              ok = false;
              linger();  // no replay must find what is raised meanwhile
              break;
            }
          }
          *theirs = 0;
        }
        ok = __all_sync(0xffffffffu, ok);
        __syncwarp();  // what a lane acquired holds for the warp's reads of the partial tiles
      }
      // sum of the partial tiles of CTAs [first, last] before this one, in CTA order, several in flight
      constexpr int AHEAD = MT > 16 ? 1 : 32 / MT;
      auto add_parts = [&](float (&sum)[MT], const float* src, int first, int last) {
        for (int c = first; c >= last; c -= AHEAD) {
          float w[AHEAD][MT];
#pragma unroll
          for (int a = 0; a < AHEAD; ++a)
#pragma unroll
            for (int m = 0; m < MT; ++m)
              w[a][m] = c - a >= last && (MODE != 0 || m < p.M)
                            ? __ldcg(src - (size_t)(c - a) * (kTiles * kTile) + m * kTsBN)
                            : 0.f;
#pragma unroll
          for (int a = 0; a < AHEAD; ++a)
#pragma unroll
            for (int m = 0; m < MT; ++m) sum[m] += w[a][m];
        }
      };
      // MARKS: the same
      constexpr int M_AHEAD = 8 / P > 0 ? 8 / P : 1;
      auto add_marked = [&](float (&sum)[MT], uint4* src, int first, int last) {
        for (int c = first; c >= last; c -= M_AHEAD) {
          uint64_t w[M_AHEAD][P];
          const auto at = [&](int a, int m) { return src - (size_t)(c - a) * (kTiles * kMarked) + m * kTsBN; };
          for (uint32_t polls = 0;;) {
            bool got = true;
#pragma unroll
            for (int a = 0; a < M_AHEAD; ++a)
#pragma unroll
              for (int m = 0; m < P; ++m) {
                w[a][m] = 0ull;
                if (c - a >= last) got &= handover::load_marked(at(a, m), w[a][m]) == token;
              }
            if (__all_sync(0xffffffffu, got)) break;
            if (!ok || ++polls >= kSpinLimit || s_abort) {
              s_abort = 1;
              atomicCAS(&g_tc_status, 0, 29);
              ok = false;
              linger();  // no replay must find what arrives meanwhile
              break;
            }
          }
          ok = __all_sync(0xffffffffu, ok);
#pragma unroll
          for (int a = 0; a < M_AHEAD; ++a)
#pragma unroll
            for (int m = 0; m < P; ++m) {
              if (c - a >= last) handover::take_mark(at(a, m));
              const float2 x = unpack2(w[a][m]);
              sum[2 * m] += x.x;
              sum[2 * m + 1] += x.y;
            }
        }
      };
      // MODE 1: CTA blockIdx.x - c has units of up if its range ends past unit KT of the tile, of gate
      // if it begins before
      int up_first = gather, gate_last = 1;
      if (MODE == 1 && gather > 0) {
        const int split = id * work.KT + p.KT;  // first unit of up
        while (up_first > 0 && ((int)blockIdx.x - up_first + 1) * work.chunk <= split) --up_first;
        while (gate_last <= gather && ((int)blockIdx.x - gate_last) * work.chunk >= split) ++gate_last;
      }
      if constexpr (MARKS) add_marked(v, marked + (MODE == 1 ? kMarked : 0), up_first, 1);
      else add_parts(v, part + (MODE == 1 ? kTile : 0), up_first, 1);
#pragma unroll
      for (int m = 0; m < MT; ++m) v[m] *= unscale;
      const int first = odd ? 1 : 0;
      const int n0 = slab * kTsBN + (col & ~1);
      if (MODE == 0) {
        const float bias = p.bias != nullptr && n0 < p.N ? load_bias(p.bias + n0 + first) : 0.f;
#pragma unroll
        for (int m = 0; m < MT; ++m) v[m] += bias;
        handover::store_rows<MT>(v, p.out + (size_t)first * p.N + n0, (size_t)p.N, first,
                                 ok && n0 < p.N ? p.M : 0, odd);
      } else if (MODE == 1) {
        float gt[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) gt[m] = kb < p.KT ? gate[m * 32] : 0.f;
        if constexpr (MARKS) add_marked(gt, marked, gather, gate_last);
        else add_parts(gt, part, gather, gate_last);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const float x = gt[m] * unscale;
          v[m] *= __fdividef(x, 1.f + __expf(-x));
        }
        // direct form: the block is one row of act
        const int row0 = p.sorted_ids != nullptr ? block * MT : block;
        handover::store_rows<MT>(v, p.out + (size_t)(row0 + first) * p.half_cols + n0,
                                 (size_t)p.half_cols, first,
                                 ok && valid && n0 < p.half_cols ? (p.sorted_ids != nullptr ? MT : 1) : 0,
                                 odd);
      } else {
        const uint32_t sel = odd ? 0x3276u : 0x5410u;
#pragma unroll
        for (int m = 0; m < MT; m += 2) {
          const float w0 = __shfl_sync(0xffffffffu, fw, m), w1 = __shfl_sync(0xffffffffu, fw, m + 1);
          const int f = __shfl_sync(0xffffffffu, fid, m + first);
          const uint32_t own = valid ? as_u32(__floats2half2_rn(v[m] * w0, v[m + 1] * w1)) : 0u;
          const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 1);
          if (ok && n0 < p.N && f < p.numel)
            *reinterpret_cast<uint32_t*>(p.out + (size_t)f * p.N + n0) = prmt(own, other, sel);
        }
      }
    }
  }

  if constexpr (SPLIT && MODE != 0) {
    const int fold = warp - kTsFold0, piece = fold * p.split + rank;
    if (fold >= 0 && piece < Cfg::kPieces) {
      __syncwarp();
      const int cluster = blockIdx.x / p.split, row = cluster / p.slabs, slab = cluster - row * p.slabs;
      const int g = lane & 7, i = lane >> 3, width = MODE == 1 ? p.half_cols : p.N;
      const int n0 = slab * kTsBN + 32 * piece + 8 * (g >> 1) + 2 * i;
      const bool valid = MODE == 2 || __ldcg(p.expert_ids + row) >= 0;
      const bool ok = __all_sync(0xffffffffu, mbar_wait_cluster(recv_full(fold), 0, &s_abort, 25));
      float a = 0.f, b = 0.f;
      for (int r = 0; r < p.split; ++r) {
        float x, y;
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(recv_at(fold, r) + lane * 8));
        a += x;
        b += y;
      }
      if (MODE == 1) {
        const float unscale = (i & 1) ? 1048576.f : 16777216.f;
        a *= unscale;
        a = b * unscale * __fdividef(a, 1.f + __expf(-a));
      }
      const float other = __shfl_xor_sync(0xffffffffu, a, 1);
      if (ok && !s_abort && valid && n0 < width && (lane & 1) == 0)
        *reinterpret_cast<__half2*>(p.out + (size_t)row * width + n0) = __floats2half2_rn(a, other);
    }
  } else if constexpr (SPLIT) {
    // ------------------------------------------------------------------ sums over the cluster
    // The quads of this CTA's pieces, shared out over the warps that convert and fold, are summed in the CTAs' order.
    // Rolled loops: the code is cold.
    constexpr int Q = Cfg::kPieceTokens / 4;
    constexpr bool kAll = MT > 8;  // up to 8 tokens the fold warps have a quad each
    constexpr int kWarps = kTsFoldWarps + (kAll ? kTsCvWarps : 0);
    if (warp >= (kAll ? 0 : kTsFold0) && warp < kTsFold0 + kTsFoldWarps) {
      __syncwarp();
      if (kAll) pdl_wait();  // orders this thread's writes after the kernel before this one
      const int own = (Cfg::kPieces - rank + p.split - 1) / p.split, g = lane & 7, i = lane >> 3;
      const bool odd = (lane & 1) != 0;
      const int first = odd ? 1 : 0, slab = blockIdx.x / p.split;
      const float unscale = (i & 1) ? 1048576.f : 16777216.f;
#pragma unroll 1
      for (int task = warp >= kTsFold0 ? warp - kTsFold0 : warp + kTsFoldWarps; task < own * Q; task += kWarps) {
        const int n = task / Q, piece = n * p.split + rank, token = (piece >> 3) * Cfg::kPieceTokens + 4 * (task % Q);
        if (token >= p.M) continue;
        const int n0 = slab * kTsBN + 32 * (piece & 7) + 8 * (g >> 1) + 2 * i;
        const float bias = p.bias != nullptr && n0 < p.N ? load_bias(p.bias + n0 + first) : 0.f;
        const bool ok = __all_sync(0xffffffffu, mbar_wait_cluster(recv_full(n), 0, &s_abort, 25));
        const uint32_t src = recv_at(n, 0) + (task % Q) * 512 + lane * 16;
        float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int r = 0; r < p.split; ++r) {
          const float4 w = lds_float4(src + r * Cfg::kPieceBytes);
          y[0] += w.x;
          y[1] += w.y;
          y[2] += w.z;
          y[3] += w.w;
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) y[m] = y[m] * unscale + bias;
        handover::store_rows<4>(y, p.out + (size_t)(token + first) * p.N + n0, (size_t)p.N, token + first,
                                ok && !s_abort && n0 < p.N ? p.M : 0, odd);
      }
    }
  }

  // ---- teardown ----
  // After a wait that gave up: copies, MMAs and, until the barrier below, what other CTAs of the cluster store may still be
  // in flight towards this CTA's shared and tensor memory.  Let them land before both are given back.  In ranges every warp
  // asks (one warp at the end: 6656 x 2464 in groups of 64 at M 1 6.2 -> 6.5 us), in clusters the last one (every warp: 2304
  // x 3168 at M 2 3.7 -> 4.3).
  __syncwarp();
  if (!SPLIT && s_abort) linger();
  tc_fence_before();
  if (SPLIT) {
    // a CTA may go when nobody stores into it any more
    __syncwarp();
    if (warp < kTsFold0 || warp >= kTsFold0 + kTsFoldWarps || work.segs == 0) cluster_wait();
    cluster_arrive_relaxed();
    cluster_wait();
  }
  __syncthreads();
  if (warp == kTsIssue) {
    if (SPLIT && s_abort) linger();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"((uint32_t)kTsTmemCols)
                 : "memory");
  }
}

// ---- host side -------------------------------------------------------------------------------

// How a dense call is cut: `split` CTAs of a cluster share a slab, or (0) `chunk` units of a CTA's range, 0: whole slabs.
struct TsCut {
  int split, chunk;
  long cost;  // estimated time in ns
};

// Ranges: the cut of the least estimated time.  Fitted to 12 shapes between 1024 x 1024 and 29568 x 8192 at 1, 4, 8 and
// 16 tokens, cut in up to 32 parts; the cut it picks is 0.6 % from the best one on average, 6 % at worst.  (Always an
// eighth of a slab, or an even share: 5.4 %.  1536 x 28672, M 4: 9.2 -> 7.8 us whole; 16384 x 1024, M 4: 9.9 -> 7.8 in
// 16 parts.)
//   1700 + 47 tokens                start and end
//   units x max(...)                352 + 3 tokens: conversion; 2.7 CTAs: the words' way from HBM
//   1440 + 16 tokens (1 + CTAs)     a slab handed over, CTAs the last one collects from
//   530                             a further slab
//   580                             more than half of the GPU (of `most` SMs): the next kernel's start is not hidden
TsCut ts_ranges(int slabs, int KT, int tokens, int most) {
  const long units = (long)slabs * KT;
  const int even = (int)((units + most - 1) / most);
  TsCut best = {0, 0, -1};
  for (const int parts : {1, 2, 3, 4, 6, 8, 12, 16}) {
    const int floor = (KT + parts - 1) / parts, chunk = parts == 1 ? 0 : (even > floor ? even : floor);
    int ctas, run, segs, gather = 0;
    if (chunk == 0) {
      ctas = slabs < most ? slabs : most;
      segs = (slabs + ctas - 1) / ctas;
      run = segs * KT;
    } else {
      ctas = (int)((units + chunk - 1) / chunk);
      segs = (chunk + KT - 1) / KT;
      run = chunk;
      if (KT % chunk == 0) {
        gather = KT / chunk - 1;
      } else if (chunk % KT != 0) {
        gather = chunk > KT ? 1 : (KT - 2) / chunk + 1;
        ++segs;
      }
    }
    const int arith = 352 + 3 * tokens, words = ctas * 27 / 10, unit = arith > words ? arith : words;
    long cost = 1700 + 47 * tokens + (long)run * unit + 530L * (segs - 1);
    if (gather > 0) cost += 1440 + 16 * tokens * (1 + gather);
    if (ctas > most / 2) cost += 580;
    if (best.cost < 0 || cost < best.cost) best = {0, chunk, cost};
    if (chunk == even) break;  // more parts: the same cut
  }
  return best;
}

// A slab to each cluster of `split` CTAs, in one wave: estimated time in ns, `resident` clusters of that size fit the
// GPU.  Fitted to 18 shapes from 1024 x 1024 to 14848 x 8192 at 1, 8, 16, 20 and 32 tokens, groups of 128 and 64, clusters
// of 2, 3, 4, 5, 6, 8 and 16.
//   1950 + 23 tokens                start and end
//   units x max(...)                355 + 2 tokens, groups of 64 15 + 2 tokens more: conversion, MMAs; 3.1 CTAs: words
//   12 split                        the sum over the cluster
//   780 + 1500 x (...)              no room for the next kernel's clusters beside these: its start is not hidden
long ts_split_cost(int slabs, int KT, int tokens, int group, int split, int resident) {
  const int arith = 355 + 2 * tokens + (group == 128 ? 0 : 15 + 2 * tokens), words = slabs * split * 31 / 10;
  long cost = 1950 + 23 * tokens + (long)((KT + split - 1) / split) * (arith > words ? arith : words) + 12 * split;
  if (2 * slabs > resident) cost += 780 + 1500L * (2 * slabs - resident) / resident;
  return cost;
}

// MODE 2, SPLIT: the CTAs of a cluster have a token's slots, whole, and add them up: estimated time, against ranges and
// a kernel for the sum.
constexpr long kTsSumKernel = 2200;
long ts_slots_cost(int slabs, int clusters, int KT, int topk) {
  const int arith = 363, words = clusters * topk * 31 / 10;
  return 2050 + (long)KT * (arith > words ? arith : words) + 12 * topk;
}

struct TsMaps {
  CUtensorMap w, s, z, x;
};

// Attributes of a SPLIT kernel, and how many of its clusters of every size the GPU holds at once.
template <int MT, int GROUP, int MODE = 0>
int ts_prepare_split() {
  static std::atomic<bool> attr_done[64];  // as in launch_ts
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return AWQ_B200_ERR_DEVICE;
  if (!attr_done[dev]) {
    auto kernel = gemm_ts_kernel<MT, MODE, GROUP, true>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TsCfg<MT, MODE, GROUP, true>::kSmem) !=
            cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
      return AWQ_B200_ERR_LAUNCH;
    attr_done[dev] = true;
  }
  return AWQ_B200_OK;
}
template <int MT, int GROUP, int MODE = 0>
int ts_resident(int split) {
  static std::atomic<int> cached[64][kMaxCluster + 1];  // zero-initialised: not asked yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  using Cfg = TsCfg<MT, MODE, GROUP, true>;
  return resident_clusters(gemm_ts_kernel<MT, MODE, GROUP, true>, split, Cfg::kThreads, Cfg::kSmem, cached[dev]);
}

// `room`: clusters of every size that the GPU holds at once, the first its SMs; nullptr: of this GPU.  `most`: CTAs of a
// cluster that the caller takes.
template <int MT, int GROUP, int MODE = 0>
TsCut ts_cut(int slabs, int KT, const int* room = nullptr, int most = kMaxCluster) {
  const TsCut ranges = ts_ranges(slabs, KT, MT, room != nullptr ? room[1] : sm_count());
  TsCut best = {0, 0, -1};
  bool hidden = true;  // the next kernel's start
  for (const int split : {2, 3, 4, 5, 6, 8, 16}) {
    if (split > KT || split > most) break;
    const int resident = room != nullptr ? room[split] : ts_resident<MT, GROUP, MODE>(split);
    if (slabs > resident) continue;
    long cost = ts_split_cost(slabs, KT, MT, GROUP, split, resident);
    // Every cluster taken: odd sizes leave SMs of a GPC idle until the last one is done, and with few tokens 112 CTAs load
    // the words more slowly than 148.
    if (MODE == 0 && slabs == resident) cost += split % 2 != 0 ? 1000 : (split == 16 && MT <= 4 ? 700 : 0);
    if (best.cost >= 0 && cost >= best.cost) continue;
    best = {split, 0, cost};
    hidden = 2 * slabs <= resident;
  }
  // The two estimates were fitted apart.  What brings them together up to 16 tokens was fitted to 95 shapes at 1, 4, 8 and 16
  // tokens, ranges and every cluster timed, and then, with the terms for all clusters taken, whole slabs and short K, to 2500
  // calls of 256 to 32768 rows that went to clusters, timed in ranges too: 113 of them were slower in clusters by more than
  // 1 % (15488 x 1696 at M 2 6.9 -> 7.5 us, 4864 x 11360 at M 15 11.2 -> 12.4, 384 x 576 at M 10 2.8 -> 3.0); now 32, 5 % at
  // most, and 5 gain more than 3 % less than they could.  In clusters instead of ranges a call takes 0.71 of the time on
  // average.  From 17 tokens whole slabs take less time than estimated: of 1000 calls that went to clusters 125 were slower
  // there (1152 x 9088 at M 32 5.8 -> 7.3 us, 256 x 5120 at M 24 2.9 -> 3.7), now 16.
  long margin = 0;
  if (MODE == 0 && MT > 16) {
    if (ranges.chunk == 0) margin = GROUP == 128 || KT <= 3 ? 1600 : 1000;
  } else if (MODE == 0) {
    const int run = ranges.chunk > 0 ? ranges.chunk : KT;
    margin = 600 + 25 * MT + (GROUP == 128 ? 0 : 200) - 45 * (run < 30 ? run : 30) + (hidden ? 0 : 300);
    if (ranges.chunk == 0) margin += 60;
    if (!hidden && GROUP == 128 && KT <= 32) margin += 100;
  }
  // gate_up of one or two tokens: of 85 calls on clusters 19 were slower there than in ranges by more than 1 %, most with
  // eight units a CTA or more (128 experts of 3712 x 256, top-4, 3 tokens 15.9 -> 17.7 us with the down GEMM).
  if (MODE == 1 && best.split > 0 && KT >= 8 * best.split) margin = 800;
  return best.cost >= 0 && best.cost + margin < ranges.cost ? best : ranges;
}

template <int MT, int GROUP, int MODE = 0>
int launch_ts_split(const TsMaps& maps, const TsParams& p, int clusters, cudaStream_t stream) {
  using Cfg = TsCfg<MT, MODE, GROUP, true>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * p.split, 1, 1);
  cfg.blockDim = dim3(Cfg::kThreads, 1, 1);
  cfg.dynamicSmemBytes = Cfg::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = add_pdl_attribute(attr, 1);
  if (cudaLaunchKernelEx(&cfg, gemm_ts_kernel<MT, MODE, GROUP, true>, maps.w, maps.s, maps.z, maps.x, p) != cudaSuccess) {
    cudaGetLastError();
    return AWQ_B200_ERR_LAUNCH;
  }
  return AWQ_B200_OK;
}

template <int MT, int MODE, int GROUP = 128, bool MARKS = false>
int launch_ts(const TsMaps& maps, const TsParams& p, int ctas, cudaStream_t stream) {
  static std::atomic<bool> attr_done[64];  // zero-initialised; setting the attribute twice is harmless
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return AWQ_B200_ERR_DEVICE;
  auto kernel = gemm_ts_kernel<MT, MODE, GROUP, false, MARKS>;
  constexpr int smem = TsCfg<MT, MODE, GROUP>::kSmem;
  if (!attr_done[dev]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
        cudaSuccess)
      return AWQ_B200_ERR_LAUNCH;
    attr_done[dev] = true;
  }
  if (launch_pdl(kernel, dim3(ctas), dim3(TsCfg<MT, MODE, GROUP>::kThreads), smem, stream, maps.w, maps.s, maps.z,
                 maps.x, p) != cudaSuccess) {
    cudaGetLastError();
    return AWQ_B200_ERR_LAUNCH;
  }
  return AWQ_B200_OK;
}

int ts_ctas() { return sm_count() < handover::kMaxCtas ? sm_count() : handover::kMaxCtas; }

// packed words [rows][words], box [128 rows x 32 words], 128-byte swizzle
int ts_word_map(TsMaps* m, const uint32_t* w, uint64_t rows, uint64_t N) {
  const uint64_t words = N / kPack;
  return encode_map_2d(&m->w, CU_TENSOR_MAP_DATA_TYPE_INT32, w, words, rows, words * 4, kTsBN / kPack, kTsBK,
                       CU_TENSOR_MAP_SWIZZLE_128B);
}
// The same, and scales and zero points, one row per group.
int ts_weight_maps(TsMaps* m, const uint32_t* w, const __half* scales, const uint32_t* qzeros,
                   uint64_t rows, uint64_t N, int group = kTsBK) {
  const uint64_t words = N / kPack, groups = rows / group;
  const uint32_t box = kTsBK / group;  // groups of a unit
  if (int rc = ts_word_map(m, w, rows, N)) return rc;
  if (int rc = encode_map_2d(&m->s, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, scales, N, groups, N * 2,
                             kTsBN, box, CU_TENSOR_MAP_SWIZZLE_NONE))
    return rc;
  return encode_map_2d(&m->z, CU_TENSOR_MAP_DATA_TYPE_INT32, qzeros, words, groups, words * 4,
                       kTsBN / kPack, box, CU_TENSOR_MAP_SWIZZLE_NONE);
}

// Partial tiles of all CTAs.
constexpr size_t ts_partial_bytes(int tokens) {
  return (size_t)handover::kMaxCtas * tokens * kTsBN * sizeof(float);
}

template <int MT, int GROUP>
int launch_ts_dense(const __half* x, const uint32_t* qweight, const __half* scales,
                    const uint32_t* qzeros, TsParams p, void* workspace, size_t workspace_bytes,
                    bool clusters, cudaStream_t stream) {
  p.KT = p.K / kTsBK;
  p.slabs = (p.N + kTsBN - 1) / kTsBN;
  if (int rc = ts_prepare_split<MT, GROUP>()) return rc;
  const TsCut cut = clusters ? ts_cut<MT, GROUP>(p.slabs, p.KT) : ts_ranges(p.slabs, p.KT, MT, sm_count());
  p.split = cut.split;
  int ctas = ts_ctas() < p.slabs ? ts_ctas() : p.slabs;
  if (cut.chunk > 0 && workspace != nullptr && workspace_bytes >= gemm_ts_workspace_bytes(p.M, p.N, p.K, GROUP)) {
    p.chunk = cut.chunk;
    p.partial = static_cast<float*>(workspace);
    p.flags = handover::make_flags(workspace, ts_partial_bytes(MT));
    ctas = (int)(((long)p.slabs * p.KT + p.chunk - 1) / p.chunk);
  }
  TsMaps maps;
  if (p.split > 1 && TsCfg<MT, 0, GROUP, true>::BULK) {
    p.scales = scales;
    p.qzeros = qzeros;
    if (int rc = ts_word_map(&maps, qweight, (uint64_t)p.K, (uint64_t)p.N)) return rc;
    maps.s = maps.z = maps.w;  // the kernel does not read them
  } else if (int rc = ts_weight_maps(&maps, qweight, scales, qzeros, (uint64_t)p.K, (uint64_t)p.N, GROUP)) {
    return rc;
  }
  if (int rc = encode_map_x(&maps.x, x, (uint64_t)p.M, (uint64_t)p.K, TsCfg<MT, 0, GROUP>::NT)) return rc;
  if (p.split > 1) return launch_ts_split<MT, GROUP>(maps, p, p.slabs, stream);
  return launch_ts<MT, 0, GROUP>(maps, p, ctas, stream);
}

// Expert GEMMs, blocks of up to 8 rows: whether partial tiles carry a token beside every two sums instead of a flag each.  A
// release takes a fold warp 2000 to 5000 cycles under the words' stream, also long after its stores, and the next tile's
// folds wait for it; but reading takes longer (16-byte strong loads, 2500 cycles for eight), and for every CTA that shares
// the tile.  So flags where many share it: in gate_up, which has twice the sums, more than about two, in down more than
// three, and in both more than six with one row.  `tiles` are expected ones.  Without the router, flags -> tokens, us: 128
// experts of 2048 x 768, top-8, 4 tokens 27.5 -> 25.6, 16 55.8 -> 53.6, 64 75.0 -> 73.4 (runs differ by 1.5); 16 of 2048 x
// 256, top-6, 2 tokens 19.9 -> 24.1 (gate_up 16 CTAs a tile; down alone 19.9); 16 of 896 x 128, top-2, 15 tokens 16.0 ->
// 17.2 (down alone 15.5).  Dense layers, where many CTAs share a slab, and blocks of 16 rows have flags: 29568 x 8192 at M
// 16 28 us, with tokens 37, 8192 x 59136 at M 1 41.4 and 43.3, 500 tokens 171 and 175.
template <int MT, int MODE>
bool ts_marks(double tiles, int KT, int max_split, int ctas) {
  const double even = tiles * KT / ctas, least = (double)KT / max_split, chunk = even > least ? even : least;
  return KT <= (MT == 4 ? 6.0 : MODE == 1 ? 1.25 : 3.0) * (chunk > 1.0 ? chunk : 1.0);
}
// Row blocks to expect: one for every expert that any pair has, and more if they do not hold the rows.
double ts_expected_blocks(const MoeArgs& a) {
  const double numel = (double)a.T * a.topk;
  if (a.direct) return numel;  // a block for a pair
  // a permutation's capacity tells over how many experts the pairs are spread, of which E are here
  const double all = a.expert_parallel ? (a.sorted_capacity - numel) / (a.block - 1) : 0.0;
  const double experts = all > a.E ? all : a.E, here = a.E / experts;
  const double hit = a.E * (1.0 - std::pow(1.0 - 1.0 / experts, numel)), full = numel * here / a.block;
  return hit > full ? hit : full;
}
template <int MT, int MODE>
int launch_ts_grouped(const TsMaps& maps, const TsParams& p, double blocks, int ctas, cudaStream_t stream) {
  if constexpr (MT <= 8)
    if (ts_marks<MT, MODE>(blocks * p.slabs, MODE == 1 ? 2 * p.KT : p.KT, p.max_split, ctas))
      return launch_ts<MT, MODE, 128, true>(maps, p, ctas, stream);
  return launch_ts<MT, MODE>(maps, p, ctas, stream);
}

// Expert GEMMs: gate_up, then down.
// *summed: whether the sum over a token's slots is done as well (MODE 2, SPLIT).
template <int MT>
int launch_ts_experts(const MoeArgs& a, __half* act, int64_t act_rows, __half* pair_out, TsParams p, bool* summed,
                      cudaStream_t stream) {
  const int ctas = ts_ctas();
  *summed = false;
  p.flags = handover::make_flags(p.partial, 2 * ts_partial_bytes(MT));
  p.sorted_ids = a.sorted_ids;
  p.expert_ids = a.expert_ids;
  p.num_post = a.num_post_pad;
  p.topk_weights = a.topk_weights;
  p.numel = a.T * a.topk;
  p.topk = a.topk;
  p.half_cols = a.I;
  p.max_split = 16;
  const double blocks = ts_expected_blocks(a);
  const uint64_t I = (uint64_t)a.I;
  {
    p.K = a.H;
    p.N = 2 * a.I;
    p.KT = a.H / kTsBK;
    p.slabs = (a.I + kTsBN - 1) / kTsBN;
    p.out = act;
    TsMaps maps;
    if (int rc = ts_weight_maps(&maps, a.w13_q, a.w13_s, a.w13_z, (uint64_t)a.E * a.H, 2 * I)) return rc;
    const int rc = a.sorted_ids != nullptr
                       ? encode_map_2d(&maps.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.x, (uint64_t)a.H,
                                       (uint64_t)a.T, (uint64_t)a.H * 2, 64, 1,
                                       CU_TENSOR_MAP_SWIZZLE_128B)
                       : encode_map_x(&maps.x, a.x, (uint64_t)a.T, (uint64_t)a.H, 16);
    if (rc) return rc;
    bool split = false;
    if constexpr (MT == 4) {
      // Direct form, the number of tiles is known: clusters as for a dense layer of that many slabs and twice the units
      if (int rc2 = ts_prepare_split<MT, 128, 1>()) return rc2;
      if (p.sorted_ids == nullptr)
        p.split = ts_cut<MT, 128, 1>(p.numel * p.slabs, 2 * p.KT, nullptr, p.KT < 8 ? p.KT : 8).split;
      split = p.split > 1;
      if (split)
        if (int rc2 = launch_ts_split<MT, 128, 1>(maps, p, p.numel * p.slabs, stream)) return rc2;
    }
    if (!split)
      if (int rc2 = launch_ts_grouped<MT, 1>(maps, p, blocks, ctas, stream)) return rc2;
  }
  p.K = a.I;
  p.N = a.H;
  p.KT = a.I / kTsBK;
  p.slabs = (a.H + kTsBN - 1) / kTsBN;
  p.out = pair_out;
  p.flags.token = handover::next_token();
  TsMaps maps;
  if (int rc = ts_weight_maps(&maps, a.w2_q, a.w2_s, a.w2_z, (uint64_t)a.E * a.I, (uint64_t)a.H))
    return rc;
  if (int rc = encode_map_x(&maps.x, act, (uint64_t)act_rows, I, 16)) return rc;
  if constexpr (MT == 4) {
    if (int rc = ts_prepare_split<MT, 128, 2>()) return rc;
    if (p.sorted_ids == nullptr && a.topk > 1 && a.topk <= 8) {
      const int clusters = a.T * p.slabs, resident = ts_resident<MT, 128, 2>(a.topk);
      if (clusters <= resident && ts_slots_cost(p.slabs, clusters, p.KT, a.topk) <
                                      ts_ranges(p.numel * p.slabs, p.KT, MT, sm_count()).cost + kTsSumKernel) {
        *summed = true;
        p.split = a.topk;
        p.out = a.out;
        return launch_ts_split<MT, 128, 2>(maps, p, clusters, stream);
      }
    }
  }
  return launch_ts_grouped<MT, 2>(maps, p, blocks, ctas, stream);
}

int ts_tokens(int M) { return M <= 4 ? 4 : (M <= 8 ? 8 : (M <= 16 ? 16 : 32)); }

}  // namespace

bool gemm_ts_supported(int M, int N, int K, int group) {
  // N % 32: 16-byte TMA row pitch of the packed weights; K % 128: whole stages
  return M >= 1 && M <= kTsMaxRows && N % 32 == 0 && K % kTsBK == 0 && (group == 128 || group == 64);
}

size_t gemm_ts_workspace_bytes(int M, int N, int K, int group) {
  if (!gemm_ts_supported(M, N, K, group)) return 0;
  return ts_partial_bytes(ts_tokens(M)) + handover::kFlagBytes;
}

int launch_gemm_ts(const __half* x, const uint32_t* qweight, const __half* scales,
                   const uint32_t* qzeros, const __half* bias, __half* out, int M, int N, int K,
                   int group, void* workspace, size_t workspace_bytes, bool clusters, cudaStream_t stream) {
  if (!gemm_ts_supported(M, N, K, group)) return AWQ_B200_ERR_SHAPE;
  TsParams p = {};
  p.bias = bias;
  p.out = out;
  p.M = M;
  p.N = N;
  p.K = K;
  auto launch = group == 128 ? launch_ts_dense<32, 128> : launch_ts_dense<32, 64>;
  if (M <= 4) launch = group == 128 ? launch_ts_dense<4, 128> : launch_ts_dense<4, 64>;
  else if (M <= 8) launch = group == 128 ? launch_ts_dense<8, 128> : launch_ts_dense<8, 64>;
  else if (M <= 16) launch = group == 128 ? launch_ts_dense<16, 128> : launch_ts_dense<16, 64>;
  return launch(x, qweight, scales, qzeros, p, workspace, workspace_bytes, clusters, stream);
}

namespace {
template <int MT, int GROUP>
int ts_tell_cut(int slabs, int KT, bool clusters, const int* room, TsCut* cut) {
  if (room == nullptr)
    if (int rc = ts_prepare_split<MT, GROUP>()) return rc;
  *cut = clusters ? ts_cut<MT, GROUP>(slabs, KT, room)
                  : ts_ranges(slabs, KT, MT, room != nullptr ? room[1] : sm_count());
  return AWQ_B200_OK;
}
}  // namespace

int gemm_ts_cut(int M, int N, int K, int group, bool clusters, const int* room, GemmCut* out) {
  if (!gemm_ts_supported(M, N, K, group)) return AWQ_B200_ERR_SHAPE;
  auto tell = group == 128 ? ts_tell_cut<32, 128> : ts_tell_cut<32, 64>;
  if (M <= 4) tell = group == 128 ? ts_tell_cut<4, 128> : ts_tell_cut<4, 64>;
  else if (M <= 8) tell = group == 128 ? ts_tell_cut<8, 128> : ts_tell_cut<8, 64>;
  else if (M <= 16) tell = group == 128 ? ts_tell_cut<16, 128> : ts_tell_cut<16, 64>;
  TsCut cut;
  if (int rc = tell((N + kTsBN - 1) / kTsBN, K / kTsBK, clusters, room, &cut)) return rc;
  *out = {ts_tokens(M), cut.chunk, cut.split, cut.split > 0 ? 1 : 0, 0};
  return AWQ_B200_OK;
}

bool moe_ts_supported(const MoeArgs& a) {
  // whole stages of K, 16-byte pitches and box starts
  return a.group == kTsBK && !a.decode_layout && a.H % kTsBK == 0 && a.I % kTsBK == 0;
}

// Partial tiles of gate and up, rows of the largest block, and the flags.
size_t moe_ts_partial_bytes(int block) {
  const size_t flagged = 2 * ts_partial_bytes(block) + handover::kFlagBytes;
  // blocks of 8 rows and the direct form may have a token beside every two sums
  const size_t marked = block <= 8 ? (size_t)2 * ts_ctas() * block * kTsBN * 8 : 0;
  return marked > flagged ? marked : flagged;
}

// Both expert GEMMs of a small batch, pair_out by pair.  Rows of act by position, direct (no
// permutation) by pair.
int launch_moe_ts(const MoeArgs& a, __half* act, int64_t act_rows, __half* pair_out, float* partial, bool* summed,
                  cudaStream_t stream) {
  TsParams p = {};
  p.partial = partial;
  if (a.direct) return launch_ts_experts<4>(a, act, act_rows, pair_out, p, summed, stream);
  return a.block == 8 ? launch_ts_experts<8>(a, act, act_rows, pair_out, p, summed, stream)
                      : launch_ts_experts<16>(a, act, act_rows, pair_out, p, summed, stream);
}

int ts_device_status(int* out, int clear) { return read_tc_status(out, clear); }

}  // namespace awq
