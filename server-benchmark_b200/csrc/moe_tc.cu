// Fused-MoE experts for prefill-sized token counts (many rows per expert), group 128 or 64.
//
// The (token, slot) pairs are already sorted by expert with every expert's run padded to whole
// row blocks (moe_align_kernel, 128 rows):
//
//   moe_gather_kernel   x_perm[pos] = x[token(pos)], the inverse permutation, the routed weight of every
//                       row, and the tile table of the grouped GEMMs: up to 256 rows of one expert per entry
//   gemm_wt_kernel<1>   gate_up with silu(gate) * up in the epilogue -> act[pos]
//   gemm_wt_kernel<2>   routed weight * down -> y[pos], over x_perm, which nobody reads any more
//   moe_combine_kernel  out[t] = sum over the slots of y[pos(t, slot)]
//
// Rows move in permuted order between the kernels, so the GEMM epilogues store whole row segments at
// a fixed pitch; what is scattered is the last kernel's reads, 4 KB at a time.
#include <cmath>

#include "common.cuh"

namespace awq {

namespace {

constexpr int kMBM = 128;      // rows of a block of the permutation
constexpr int kTileRows = 256;  // rows of a grouped GEMM's tile, at most

}  // namespace

// Rows of a tile (a multiple of 16): those of the least expected cost, for experts whose row counts scatter about
// the average by its root.  In SM cycles a (tile, slab) of n rows costs its units times max(460, 4 n), the conversion or
// the tensor pipe, and what its epilogue leaves uncovered: 400 with two accumulators (up to 128 rows), 800 + 10 n with one.
// A GEMM of `local` experts takes the average cost times the tiles of a pair, half way between their average and the
// next whole number: with few experts some pairs have a tile more than the others.  Fitted to all tiles from 128 to 256
// rows at 229 batches of 104 to 450 rows per expert, 15 shapes of 4 to 128 experts; the size it picks is 0.7 % from the
// best on average, 14 % at worst, and 0.6 and 6 % at 90 batches of 11 other shapes.  Without the tiles of a pair (and 500,
// 400 + 12 n) it was 1.8 %, 25 % at worst: 16 experts of 2048 x 1024, top-2, 960 tokens 128 rows, 49.9 us, 144 rows 46.3.
// Routing that the host cannot know, experts drawn with a bias, prefers 128 rows by 10 %.
// Against 128 rows up to 100 per expert and 256 beyond, whatever the batch (router excluded, top-8, us): 128 experts of
// 2048 x 768: 1800 tokens 233 -> 200, 4096 492 -> 408; 64 of 4096 x 1536, top-4: 4096 814 -> 708.
int moe_tile_rows(long long pairs, long long experts, int local, int H, int I, int cta_pairs) {
  const double mean = (double)pairs / experts, root = sqrt(mean);
  const int slabs[2] = {I / 128, H / 256};
  const double stages[2] = {H / 128., I / 128.};  // of a tile
  int best = kMBM;
  double best_cost = -1;
  for (int rows = kMBM; rows <= kTileRows; rows += 16) {
    double units = 0, epilogue = 0, tiles = 0;  // of one expert
    auto add = [&](double count, double n) {
      units += count * (4 * n > 460 ? 4 * n : 460.);
      epilogue += count * (rows <= 128 ? 400. : 800 + 10 * n);
      tiles += count;
    };
    for (int z = -4; z <= 4; ++z) {  // half deviations, weighted by the normal density
      constexpr double kWeight[5] = {0.2041, 0.1801, 0.1238, 0.0665, 0.0276};
      const double weight = kWeight[z < 0 ? -z : z];
      const double count = mean + 0.5 * z * root > 1 ? mean + 0.5 * z * root : 1;
      const double whole = floor(count / rows), rest = count - whole * rows;
      add(weight * whole, rows);
      if (rest > 0) add(weight, rest);
    }
    double cost = 0;
    for (int g = 0; g < 2; ++g) {
      const double per_pair = tiles * local * slabs[g] / cta_pairs;
      cost += (stages[g] * units + epilogue) / tiles * (per_pair + ceil(per_pair - 1e-3)) / 2;
    }
    if (best_cost < 0 || cost < best_cost) {
      best = rows;
      best_cost = cost;
    }
  }
  return best;
}

namespace {

// Experts that the permutation was built for: those of all ranks under expert parallelism, where `E` counts
// the local ones.  Read off the capacity of the permuted list, which has room for kMBM - 1 entries of padding
// per expert (awq_b200_moe_sorted_capacity; a batch of 36 rows per expert has more pairs than experts).
long long routed_experts(const MoeArgs& a) {
  const long long from_capacity = (a.sorted_capacity - (long long)a.T * a.topk) / (kMBM - 1);
  return a.expert_parallel && from_capacity > a.E ? from_capacity : a.E;
}

// Tile table of the grouped GEMMs in gemm_wt.cu: up to `tile_rows` rows of one expert per entry, i.e. every expert's
// run of row blocks cut into pieces of that many rows.  One CTA; blocks are scanned 256 at a time, and the last
// block of a run writes its tiles.  With few experts the CTA is what the gather takes, a chain of loads from L2 and of
// cold code: hence one round of loads for a block and its neighbours, the first of them ahead of the block count, runs
// found by a ballot, and loops that stay loops.  8 experts of 2048 x 768, 160 to 400 tokens: 27.1 -> 26.0, 28.0 -> 27.4, 30.1
// -> 29.2 us against loads in turn and two scans by shuffles.  (The padding sought with 23 loads in two rounds, unrolled, in
// place of eight in turn: 28.7 us for the first.)
constexpr int kGatherThreads = 256;
__device__ void moe_tile_table(const int32_t* sorted_ids, const int32_t* expert_ids, const int32_t* num_post_pad,
                               int blocks, int numel, int block, int tile_rows, int4* __restrict__ tiles,
                               int32_t* __restrict__ n_tiles) {
  __shared__ int s_start[kGatherThreads / 32], s_sum[kGatherThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int start_carry = 0, count_carry = 0;
  int e = tid < blocks ? __ldcg(expert_ids + tid) : -1;
  const int used = __ldcg(num_post_pad) / block;
#pragma unroll 1
  for (int base = 0; base < used; base += kGatherThreads) {
    const int i = base + tid;
    if (base > 0 && i < used) e = __ldcg(expert_ids + i);
    if (i >= used) e = -1;
    int before = __shfl_up_sync(0xffffffffu, e, 1), after = __shfl_down_sync(0xffffffffu, e, 1);
    if (lane == 0 && i > 0 && i < used) before = __ldcg(expert_ids + i - 1);
    if (lane == 31 && i + 1 < used) after = __ldcg(expert_ids + i + 1);
    const unsigned begins = __ballot_sync(0xffffffffu, i < used && (i == 0 || before != e));
    if (lane == 31) s_start[warp] = begins != 0 ? i - __clz(begins) : 0;  // the last run that begins in this warp
    const bool ends = e >= 0 && (i + 1 == used || after != e);
    int valid = 0;
    if (ends) {  // valid rows come first in the run's last block: find where its padding starts
      int hi = block;
#pragma unroll 1
      while (valid < hi) {
        const int mid = (valid + hi) / 2;
        if (__ldcg(sorted_ids + (int64_t)i * block + mid) < numel) valid = mid + 1;
        else hi = mid;
      }
    }
    __syncthreads();
    const unsigned own = begins & (0xffffffffu >> (31 - lane));
    int start = own != 0 ? i - lane + 31 - __clz(own) : start_carry;  // first block of this block's run
    for (int w = 0; w < kGatherThreads / 32; ++w) {
      if (w < warp) start = max(start, s_start[w]);
      start_carry = max(start_carry, s_start[w]);
    }
    const int rows = ends ? (i - start) * block + valid : 0;
    const int pieces = (rows + tile_rows - 1) / tile_rows;
    int incl = pieces;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    int pos = count_carry + incl - pieces;
    for (int w = 0; w < kGatherThreads / 32; ++w) {
      if (w < warp) pos += s_sum[w];
      count_carry += s_sum[w];
    }
#pragma unroll 1
    for (int at = 0; at < rows; at += tile_rows)
      tiles[pos++] = make_int4(e, start * block + at, min(tile_rows, rows - at), 0);
    __syncthreads();
  }
  if (tid == 0) n_tiles[0] = count_carry;
}

// x_perm[pos, :] = x[token(pos), :], row_weights[pos] = weights[pair] and inverse[pair] = pos for the rows
// of the used blocks (padding rows are left as they are: what the GEMMs compute from them is stored nowhere).
// One warp per row, eight rows per CTA; a lane keeps four 16-byte loads in flight.  The
// first CTA writes the tile table instead of rows.
constexpr int kGatherRows = kGatherThreads / 32;
__global__ void __launch_bounds__(kGatherThreads, 8)
moe_gather_kernel(const __half* x, const int32_t* sorted_ids,
                  const int32_t* expert_ids, const int32_t* num_post_pad, const float* weights,
                  __half* __restrict__ x_perm, int32_t* __restrict__ inverse, float* __restrict__ row_weights,
                  int4* __restrict__ tiles, int32_t* __restrict__ n_tiles, int64_t capacity,
                  int numel, int topk, int H, int rows_per_block, int tile_rows) {
  pdl_launch_dependents();
  pdl_wait();
  const int block = (int)blockIdx.x - 1;
  if (block < 0) {
    moe_tile_table(sorted_ids, expert_ids, num_post_pad, (int)(capacity / rows_per_block), numel,
                   rows_per_block, tile_rows, tiles, n_tiles);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int64_t pos = (int64_t)block * kGatherRows + (threadIdx.x >> 5);
  // both loads in flight together
  const int post = __ldcg(num_post_pad);
  const int fid = pos < capacity ? __ldcg(sorted_ids + pos) : numel;
  if (pos >= post) return;
  uint4* dst = reinterpret_cast<uint4*>(x_perm + (size_t)pos * H);
  const int units = H / 8;
  if (fid >= numel) return;
  if (lane == 0) {
    inverse[fid] = (int32_t)pos;
    row_weights[pos] = __ldcg(weights + fid);
  }
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(fid / topk) * H);
  int i = lane;
  for (; i + 96 < units; i += 128) {
    const uint4 a = __ldcg(src + i), b = __ldcg(src + i + 32), c = __ldcg(src + i + 64),
                d = __ldcg(src + i + 96);
    dst[i] = a;
    dst[i + 32] = b;
    dst[i + 64] = c;
    dst[i + 96] = d;
  }
  for (; i < units; i += 32) dst[i] = __ldcg(src + i);
}

// out[t] = sum over the slots, in slot order, of y[inverse[t, slot]] in fp32.  A pair that the permutation
// dropped (its expert lives on another rank, or its id is no expert's) has no entry in `inverse`: what
// stands there is left over from other calls.  So an entry counts only if the permuted list has the pair at
// that place, which also keeps every read inside y.  One thread per 8 columns.
__global__ void __launch_bounds__(256)
moe_combine_kernel(const __half* y, const int32_t* inverse, const int32_t* sorted_ids,
                   __half* __restrict__ out, int64_t capacity, int T, int topk, int H) {
  const int units = H / 8;
  const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  if (idx >= (long long)T * units) return;
  const int t = (int)(idx / units), u = (int)(idx % units);
  const int32_t* pos = inverse + (size_t)t * topk;
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = 0.f;
  auto add = [&](const uint4& r) {
    const __half* h = reinterpret_cast<const __half*>(&r);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] += __half2float(h[j]);
  };
  auto fetch = [&](int s) {
    const int p = __ldcg(pos + s);
    const bool inside = p >= 0 && p < capacity;
    const int pair = inside ? __ldcg(sorted_ids + p) : -1;
    const uint4 r = inside ? __ldcg(reinterpret_cast<const uint4*>(y + (size_t)p * H) + u)
                           : make_uint4(0, 0, 0, 0);
    return pair == t * topk + s ? r : make_uint4(0, 0, 0, 0);
  };
  int s = 0;
  for (; s + 4 <= topk; s += 4) {
    const uint4 a = fetch(s), b = fetch(s + 1), c = fetch(s + 2), d = fetch(s + 3);
    add(a);
    add(b);
    add(c);
    add(d);
  }
  for (; s < topk; ++s) add(fetch(s));
  __align__(16) __half o[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) o[j] = __float2half_rn(v[j]);
  *(reinterpret_cast<uint4*>(out + (size_t)t * H) + u) = *reinterpret_cast<uint4*>(o);
}

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

}  // namespace

bool moe_tc_supported(int H, int I, int group) {
  // tiles: gate/up segments of 128 columns (I % 128), 256 hidden columns (H % 256);
  // stages of 64 rows inside one quantisation group; 16-byte TMA row pitches
  return H % 256 == 0 && I % 128 == 0 && (group == 128 || group == 64);
}

namespace {
// Scratch of a call with `rows` permuted rows: gathered activations (later the down projection's
// output), silu(gate) * up, inverse permutation, routed weights by row, tile table.
struct TcScratch {
  size_t act, inverse, weights, tiles, n_tiles, bytes;
  TcScratch(int64_t rows, int64_t pairs, int H, int I) {
    act = align_up((size_t)rows * H * 2, 256);
    inverse = act + align_up((size_t)rows * I * 2, 256);
    weights = inverse + align_up((size_t)pairs * sizeof(int32_t), 256);
    tiles = weights + align_up((size_t)(rows + 32) * sizeof(float), 256);
    n_tiles = tiles + align_up((size_t)(rows / kMBM) * sizeof(int4), 256);
    bytes = n_tiles + 256;
  }
};
int64_t padded_rows(int64_t capacity) { return (capacity + kMBM - 1) / kMBM * kMBM; }
}  // namespace

size_t moe_tc_workspace_bytes(int T, int topk, int E, int H, int I) {
  const int64_t pairs = (int64_t)T * topk;
  return TcScratch(padded_rows(awq_b200_moe_sorted_capacity(pairs, E, kMBM)), pairs, H, I).bytes;
}

size_t moe_tc_layout_bytes(const MoeArgs& a) {
  return TcScratch(padded_rows(a.sorted_capacity), (int64_t)a.T * a.topk, a.H, a.I).bytes;
}

int launch_moe_experts_tc(const MoeArgs& a, void* workspace, size_t workspace_bytes,
                          cudaStream_t stream) {
  if (a.block != kMBM || !moe_tc_supported(a.H, a.I, a.group)) return AWQ_B200_ERR_SHAPE;
  const int numel = a.T * a.topk;
  const int max_rows = moe_tile_rows(numel, routed_experts(a), a.E, a.H, a.I, sm_count() / 2);
  const int64_t rows = padded_rows(a.sorted_capacity);
  const TcScratch at(rows, numel, a.H, a.I);
  if (workspace == nullptr || workspace_bytes < at.bytes) return AWQ_B200_ERR_WORKSPACE;
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  __half* x_perm = reinterpret_cast<__half*>(ws);
  __half* act = reinterpret_cast<__half*>(ws + at.act);
  int32_t* inverse = reinterpret_cast<int32_t*>(ws + at.inverse);
  float* row_weights = reinterpret_cast<float*>(ws + at.weights);
  int4* tiles = reinterpret_cast<int4*>(ws + at.tiles);
  int32_t* n_tiles = reinterpret_cast<int32_t*>(ws + at.n_tiles);

  if (a.expert_parallel) {
    // Most pairs are routed to experts of other ranks, and what an earlier call left of them would cost the
    // combine kernel a row each: one of eight ranks of 128 experts (2048 x 768, top-8), 2500
    // tokens, 93 us without and 76 with this.
    if (cudaMemsetAsync(inverse, 0xFF, (size_t)numel * sizeof(int32_t), stream) != cudaSuccess)
      return AWQ_B200_ERR_LAUNCH;
  }
  if (launch_pdl(moe_gather_kernel, dim3((unsigned)((rows + kGatherRows - 1) / kGatherRows + 1)),
                 dim3(kGatherThreads), 0, stream, a.x, a.sorted_ids, a.expert_ids, a.num_post_pad,
                 a.topk_weights, x_perm, inverse, row_weights, tiles, n_tiles, a.sorted_capacity, numel,
                 a.topk, a.H, a.block, max_rows) != cudaSuccess) {
    cudaGetLastError();
    return AWQ_B200_ERR_LAUNCH;
  }
  if (int rc = launch_wt_grouped(1, max_rows, x_perm, rows, a.w13_q, a.E, a.w13_s, a.w13_z, tiles, n_tiles,
                                 nullptr, act, a.H, 2 * a.I, a.group, a.I, stream))
    return rc;
  if (int rc = launch_wt_grouped(2, max_rows, act, rows, a.w2_q, a.E, a.w2_s, a.w2_z, tiles, n_tiles,
                                 row_weights, x_perm, a.I, a.H, a.group, 0, stream))
    return rc;
  const long long work = (long long)a.T * (a.H / 8);
  if (launch_pdl(moe_combine_kernel, dim3((unsigned)((work + 255) / 256)), dim3(256), 0, stream,
                 (const __half*)x_perm, (const int32_t*)inverse, a.sorted_ids, a.out, a.sorted_capacity, a.T,
                 a.topk, a.H) != cudaSuccess) {
    cudaGetLastError();
    return AWQ_B200_ERR_LAUNCH;
  }
  return AWQ_B200_OK;
}

}  // namespace awq
