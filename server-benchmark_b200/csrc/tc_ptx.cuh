// PTX wrappers shared by the tcgen05 kernels: mbarrier, TMA, tcgen05 fences / MMA / commit /
// TMEM loads, shared-memory matrix descriptors.  Every mbarrier wait is bounded.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace awq {

// First bounded wait that ran out in this translation unit (0 = none).  One copy per .cu file
// that includes this header; each file exports a reader for its own copy.
static __device__ int g_tc_status = 0;

// Host side: read this translation unit's status word; `clear` puts it back to 0 afterwards.
// The word is sticky: it keeps the first wait that ran out until it is cleared.
inline int read_tc_status(int* out, int clear) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_tc_status, sizeof(int)) != cudaSuccess) return AWQ_B200_ERR_LAUNCH;
  if (clear && v != 0) {
    const int zero = 0;
    if (cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int)) != cudaSuccess)
      return AWQ_B200_ERR_LAUNCH;
  }
  *out = v;
  return AWQ_B200_OK;
}

namespace tc {

constexpr uint32_t kSpinLimit = 1u << 20;

// ---- PTX wrappers --------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Two barriers at once, whose latencies overlap.
__device__ __forceinline__ bool mbar_try_wait2(uint32_t bar0, uint32_t parity0, uint32_t bar1, uint32_t parity1) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4;\n\t"
      "and.pred p, p, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar0), "r"(parity0), "r"(bar1), "r"(parity1)
      : "memory");
  return ok != 0;
}
// Non-blocking probe of a phase.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait.  Returns false if the CTA has been aborted (by this thread or another).
__device__ __forceinline__ bool mbar_wait_n(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                            int code, uint32_t limit) {
  if (mbar_try_wait(bar, parity)) return true;  // fast path: the phase is already complete
  for (uint32_t i = 1; i < limit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 31u) == 0 && *abort_flag) return false;
  }
  *abort_flag = 1;
  atomicCAS(&g_tc_status, 0, code);
  return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                          int code) {
  return mbar_wait_n(bar, parity, abort_flag, code, kSpinLimit);
}
// The same for a converged warp, with one answer for all lanes.  The way through a complete phase is a probe, a vote
// and a branch.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "vote.sync.all.pred q, p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  if (ok != 0) return true;
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, code));
}
// About a millisecond, after a wait that gave up.
__device__ __forceinline__ void linger() {
  const long long end = clock64() + 2000000;
  while (clock64() < end) {
  }
}
// True in exactly one lane of a fully active warp (always the same lane).  A tcgen05.mma or
// tcgen05.commit issued this way from a converged warp costs its warp ~25-45 cycles; issued from
// one lane that loops alone while the other 31 are parked elsewhere it was measured at ~150.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}
// contiguous bytes: both addresses and the size multiples of 16
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
// orders plain accesses, to global memory too, before bulk copies
__device__ __forceinline__ void fence_proxy_async_all() {
  asm volatile("fence.proxy.async;" ::: "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1,
                                            int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
// Four rows of a 2-D tensor by index (the map's box is one row high), one below the other.
__device__ __forceinline__ void tma_gather4(uint32_t dst, const CUtensorMap* map, int col, int r0,
                                            int r1, int r2, int r3, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
      "l"(map), "r"(col), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void umma_f16_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   bar)
               : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
      "[%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor (sm_100 format): start address, leading / stride byte
// offsets (all >> 4), version 1, 128-byte swizzle.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo_bytes,
                                              uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version (Blackwell)
  d |= (uint64_t)2 << 61;  // SWIZZLE_128B
  return d;
}

// ---- host: tiled tensor maps ---------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled through the runtime's driver entry point lookup (no link against
// libcuda); nullptr when the driver does not provide it.
inline EncodeTiledFn encode_tiled_fn() {
  // initialised once, thread-safely (function-local static)
  static const EncodeTiledFn fn = [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      return reinterpret_cast<EncodeTiledFn>(sym);
    return static_cast<EncodeTiledFn>(nullptr);
  }();
  return fn;
}

// Row-major 2-D tensor [dim1 rows][dim0 elements], row pitch in bytes, box [box1 x box0].
inline int encode_map_2d(CUtensorMap* m, CUtensorMapDataType dt, const void* base, uint64_t dim0,
                         uint64_t dim1, uint64_t pitch_bytes, uint32_t box0, uint32_t box1,
                         CUtensorMapSwizzle swizzle) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (enc == nullptr) return AWQ_B200_ERR_DRIVER;
  const cuuint64_t dims[2] = {dim0, dim1};
  const cuuint64_t strides[1] = {pitch_bytes};
  const cuuint32_t box[2] = {box0, box1};
  const cuuint32_t estr[2] = {1, 1};
  return enc(m, dt, 2, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? AWQ_B200_OK
             : AWQ_B200_ERR_DRIVER;
}

struct Map3d {
  uint64_t dim[3];
  uint64_t pitch[2];  // bytes between neighbours of dimension 1 / 2
  uint32_t box[3];
};
inline int encode_map_3d(CUtensorMap* m, CUtensorMapDataType dt, const void* base, const Map3d& t,
                         CUtensorMapSwizzle swizzle) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (enc == nullptr) return AWQ_B200_ERR_DRIVER;
  const cuuint64_t dims[3] = {t.dim[0], t.dim[1], t.dim[2]};
  const cuuint64_t strides[2] = {t.pitch[0], t.pitch[1]};
  const cuuint32_t box[3] = {t.box[0], t.box[1], t.box[2]};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, dt, 3, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? AWQ_B200_OK
             : AWQ_B200_ERR_DRIVER;
}

// Row-major fp16 matrix [rows][K] seen as [K / 64][rows][64]; box [2][box_rows][64] with 128-byte
// swizzle: 128 columns (box_k64 x 64) of box_rows rows as adjacent K-major tiles, in one copy.
inline int encode_map_x(CUtensorMap* m, const void* base, uint64_t rows, uint64_t K,
                        uint32_t box_rows, uint32_t box_k64 = 2) {
  return encode_map_3d(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, base,
                       {{64, rows, K / 64}, {K * 2, 128}, {64, box_rows, box_k64}},
                       CU_TENSOR_MAP_SWIZZLE_128B);
}

// ---- shared by the kernels that keep the weight operand in tensor memory (gemm_ts, gemm_wt) ----
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
// 16 lanes x 32 columns (x8: eight groups of four columns): of columns 4 c .. 4 c + 3, thread (g, t) gives row g,
// column t, in v[2 c] and row g + 8 in v[2 c + 1].  The shape decides what a store costs: these take 16 cycles of a
// lane quarter's port, as 16x256b 32 (32x32b: 12, but it wants one weight column per thread).
__device__ __forceinline__ void tmem_st_16x128b(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_16x128b(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
               "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
// 16 lanes x 32 columns as an mma accumulator fragment: of columns 8 k .. 8 k + 7, thread (g, t) gets
// row g, columns 2 t and 2 t + 1, in r[4 k], r[4 k + 1], and row g + 8 in r[4 k + 2], r[4 k + 3].
__device__ __forceinline__ void tmem_ld_16x256b_x4(uint32_t taddr, float (&r)[16]) {
  uint32_t v[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) r[i] = __uint_as_float(v[i]);
}
// The same of 16 columns.
__device__ __forceinline__ void tmem_ld_16x256b_x2(uint32_t taddr, float (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
               : "r"(taddr)
               : "memory");
}
// 8 x 8 fp16 matrix, two neighbouring values of row g per thread (g, t): transposed
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ float4 lds_float4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr));
  return v;
}
// A operand in tensor memory, B through a shared-memory descriptor
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// ---- pairs of CTAs (cluster of two, cta_group::2) -------------------------------------------
// Address of `saddr` of this CTA in the shared memory of cluster rank `rank`.
__device__ __forceinline__ uint32_t map_rank(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
// Four values into another CTA's shared memory, counted by a barrier there (both addresses as map_rank gives them).
__device__ __forceinline__ void st_async_v4(uint32_t dst, const float* v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
               "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async_v2(uint32_t dst, float a, float b, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(dst), "f"(a),
               "f"(b), "r"(bar)
               : "memory");
}
// Arrive on a barrier given by its cluster address (own or peer CTA).  What such arrivals hand over is
// tensor memory, ordered by the tcgen05 fences around them, so the default CTA scope is enough; the
// cluster-scope forms (release / acquire) add memory barriers: 65 against 55 us for the whole kernel
// at K 29568 x N 8192, M = 16.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// One lane's arrivals on a barrier given by its cluster address and on one of this CTA, without a branch.
__device__ __forceinline__ void mbar_arrive_both(uint32_t cluster_bar, uint32_t bar, bool lane) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.u32 p, %2, 0;\n\t"
      "@p mbarrier.arrive.shared::cluster.b64 _, [%0];\n\t"
      "@p mbarrier.arrive.shared::cta.b64 _, [%1];\n\t}" ::"r"(cluster_bar),
      "r"(bar), "r"((uint32_t)lane)
      : "memory");
}
// TMA load into this CTA's shared memory that completes on a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1,
                                                 int c2, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(cluster_bar)
      : "memory");
}
// A 256-row MMA over the pair: rows 0-127 in the leader's tensor memory, 128-255 in the peer's; each
// CTA holds half of B's rows at the same shared-memory offset.
// Arrives on the barrier at this offset in both CTAs (`mask`: their ranks in the cluster) once the pair's MMAs so far
// are complete.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar, uint16_t mask = 3) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(bar),
      "h"(mask)
      : "memory");
}
// One unit of a tile whose A operand lies in tensor memory: eight MMAs of K = 16 over the 128 k of an
// x stage (four steps in each of its two 64-k halves, `half` descriptor units apart), the commit on
// `done` of both CTAs, and a probe of the next unit's barrier whose latency the MMAs hide: the
// predicate is read only behind them, which takes one asm block (a probe of its own costs its warp
// ~100 cycles).  Returns whether the next unit is ready.  One elected lane of the leader.
__device__ __forceinline__ bool umma_unit_pair(uint32_t dcol, uint32_t acol, uint64_t dx,
                                               uint32_t half, uint32_t idesc, uint32_t acc,
                                               uint32_t done, uint32_t next, uint32_t next_parity,
                                               uint16_t mask = 3) {
  uint32_t ready;
  asm volatile(
      "{\n\t.reg .pred t, p, q;\n\t"
      ".reg .b64 d0, d1, d2, d3, d4, d5, d6, d7, h;\n\t"
      ".reg .b32 a1, a2, a3, a4, a5, a6, a7;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 t, [%8], %9;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "setp.eq.b32 q, 0, 0;\n\t"
      "cvt.u64.u32 h, %4;\n\t"
      "mov.b64 d0, %3;\n\t"
      "add.u64 d1, %3, 2;\n\t"
      "add.u64 d2, %3, 4;\n\t"
      "add.u64 d3, %3, 6;\n\t"
      "add.u64 d4, %3, h;\n\t"
      "add.u64 d5, d4, 2;\n\t"
      "add.u64 d6, d4, 4;\n\t"
      "add.u64 d7, d4, 6;\n\t"
      "add.u32 a1, %2, 8;\n\t"
      "add.u32 a2, %2, 16;\n\t"
      "add.u32 a3, %2, 24;\n\t"
      "add.u32 a4, %2, 32;\n\t"
      "add.u32 a5, %2, 40;\n\t"
      "add.u32 a6, %2, 48;\n\t"
      "add.u32 a7, %2, 56;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [%2], d0, %5, p;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [a1], d1, %5, q;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [a2], d2, %5, q;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [a3], d3, %5, q;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [a4], d4, %5, q;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [a5], d5, %5, q;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [a6], d6, %5, q;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%1], [a7], d7, %5, q;\n\t"
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%7], %10;\n\t"
      "selp.u32 %0, 1, 0, t;\n\t}"
      : "=r"(ready)
      : "r"(dcol), "r"(acol), "l"(dx), "r"(half), "r"(idesc), "r"(acc), "r"(done), "r"(next),
        "r"(next_parity), "h"(mask)
      : "memory");
  return ready != 0;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
// Orders no memory: a release waits for this thread's stores to global memory, some 1000 cycles at a kernel's end.
__device__ __forceinline__ void cluster_arrive_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Bounded wait for what other CTAs of the cluster stored into this one (st.async).
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag, int code) {
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok != 0) return true;
    if ((i & 31u) == 31u && *abort_flag) return false;
  }
  *abort_flag = 1;
  atomicCAS(&g_tc_status, 0, code);
  return false;
}
// Four transposed 8 x 8 halfword matrices; lane l gives the address of row l % 8 of matrix l / 8.
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

}  // namespace tc
}  // namespace awq
