// Splitting a list of (tile, stage) units over persistent workers (CTAs or CTA pairs), and handing
// partial tiles from one worker to the next through global scratch.
//
// Every worker takes one contiguous range of `chunk` units and walks it from its last tile to its
// first.  A tile that several workers share is finished by the worker that holds its last stage and
// gets to it last; every other worker does its part of such a tile first and hands an fp32 partial
// tile over behind a flag.  So a worker only waits for workers with smaller block numbers, which were
// started before it and do not wait for it.
#pragma once

#include <chrono>

#include "common.cuh"

namespace awq {

namespace handover {

// Flags of the hand-over, one per CTA and epilogue warp, behind the partial tiles in the caller's scratch,
// which comes with any content.  A flag is raised by storing the token of its launch, a 64-bit number that
// no other launch of the process has and that other data holds with a chance of 2^-64; the one warp that
// waits for it lowers it again (to 0, no token), so a replay of a captured launch, whose token is the same
// every time, does not find it raised.  Nothing outlives the call but these zeros.  Calls that share a
// scratch buffer must not overlap.
constexpr int kMaxCtas = 256;
constexpr int kMaxWarps = 8;
constexpr size_t kFlagBytes = (size_t)kMaxCtas * kMaxWarps * sizeof(unsigned long long);

__device__ __forceinline__ void raise_flag(unsigned long long* flag, unsigned long long token) {
  asm volatile("st.release.gpu.global.b64 [%0], %1;" ::"l"(flag), "l"(token) : "memory");
}
__device__ __forceinline__ unsigned long long read_flag(const unsigned long long* flag) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(flag) : "memory");
  return v;
}
struct Flags {
  unsigned long long* base;  // [CTA][kMaxWarps]
  unsigned long long token;
  __device__ __forceinline__ unsigned long long* at(int cta, int warp) const {
    return base + cta * kMaxWarps + warp;
  }
  __device__ __forceinline__ void raise(int cta, int warp) const { raise_flag(at(cta, warp), token); }
  __device__ __forceinline__ bool raised(int cta, int warp) const { return read_flag(at(cta, warp)) == token; }
  __device__ __forceinline__ void lower(int cta, int warp) const { *at(cta, warp) = 0; }
};

// Two sums and the token of their launch in 16 bytes that are written and read as one, so that they need no flag.  Who
// reads them takes the token away again.
__device__ __forceinline__ void store_marked(uint4* at, unsigned long long value, unsigned long long token) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\t"
      "mov.b128 t, {%1, %2};\n\t"
      "st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(at),
      "l"(value), "l"(token)
      : "memory");
}
__device__ __forceinline__ unsigned long long load_marked(const uint4* at, uint64_t& value) {
  unsigned long long token;
  asm volatile(
      "{\n\t.reg .b128 t;\n\t"
      "ld.relaxed.gpu.global.b128 t, [%2];\n\t"
      "mov.b128 {%0, %1}, t;\n\t}"
      : "=l"(value), "=l"(token)
      : "l"(at)
      : "memory");
  return token;
}
__device__ __forceinline__ void take_mark(uint4* at) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(reinterpret_cast<unsigned long long*>(at) + 1), "l"(0ull)
               : "memory");
}

// Token of a launch: a counter, started by the clock and spread over 64 bits by an odd factor.
inline unsigned long long next_token() {
  static std::atomic<unsigned long long> counter{
      (unsigned long long)std::chrono::system_clock::now().time_since_epoch().count()};
  const unsigned long long token = ++counter * 0x9E3779B97F4A7C15ull;
  return token != 0 ? token : next_token();
}

// Flags of a launch whose partial tiles take `partial_bytes` (a multiple of 8) of `workspace`.
inline Flags make_flags(void* workspace, size_t partial_bytes) {
  return {reinterpret_cast<unsigned long long*>(static_cast<uint8_t*>(workspace) + partial_bytes), next_token()};
}

// A worker's units: segments of consecutive stages of one tile, walked in the same order by every
// role of the kernel.  Strided work (chunk = 0): the whole tiles worker, worker + workers, ...
struct Work {
  int worker, workers, KT, chunk;
  int segs, count;             // segments and units of this worker
  int begin, end;              // chunked: first stage of the lowest tile, end stage of the highest
  int tile0;                   // chunked: the lowest tile
  bool chunked;
  __device__ __forceinline__ Work(int worker_, int workers_, int tiles, int KT_, int chunk_)
      : worker(worker_), workers(workers_), KT(KT_), chunk(chunk_), chunked(chunk_ > 0) {
    if (chunked) {
      const int first = worker * chunk;
      if (first >= tiles * KT) {  // more workers than ranges
        segs = count = begin = end = tile0 = 0;
        return;
      }
      const int last = min(first + chunk, tiles * KT) - 1;
      count = last - first + 1;
      tile0 = first / KT;
      const int top = last / KT;
      segs = top - tile0 + 1;
      begin = first - tile0 * KT;
      end = last - top * KT + 1;
    } else {
      segs = worker < tiles ? (tiles - worker + workers - 1) / workers : 0;
      count = segs * KT;
      tile0 = begin = 0;
      end = KT;
    }
  }
  // Units [first, last) of the list, for workers that hand nothing over through scratch.
  __device__ __forceinline__ static Work range(int first, int last, int KT) { return Work(first, last, KT); }
  __device__ __forceinline__ int tile_id(int seg) const {
    return chunked ? tile0 + segs - 1 - seg : worker + seg * workers;
  }
  __device__ __forceinline__ int k_begin(int seg) const {
    return chunked && seg == segs - 1 ? begin : 0;
  }
  __device__ __forceinline__ int k_end(int seg) const { return chunked && seg == 0 ? end : KT; }
  // Workers before this one that share the tile of a segment which this worker finishes.
  __device__ __forceinline__ int helpers(int seg) const {
    return k_begin(seg) > 0 && k_end(seg) == KT ? worker - tile_id(seg) * KT / chunk : 0;
  }

 private:
  __device__ __forceinline__ Work(int first, int last, int KT_)
      : worker(0), workers(1), KT(KT_), chunk(1), count(last - first), chunked(true) {
    tile0 = first / KT;
    const int top = (last - 1) / KT;
    segs = count > 0 ? top - tile0 + 1 : 0;
    begin = first - tile0 * KT;
    end = last - top * KT;
  }
};

// Two tokens of 32 columns per step: this lane's column of tokens c, c + 1 packed to fp16, then
// neighbouring columns (lanes 2 j, 2 j + 1) meet: the even lane stores the column pair of token c, the
// odd lane that of token c + 1.  Cheap on purpose (pack, shuffle, byte permute, store): epilogue warps
// share their schedulers with the conversion warps and get an issue slot every five or six cycles.
// `dst`: address of this lane's column pair in the row of its first token, number `m`.
template <int COUNT>
__device__ __forceinline__ void store_rows(const float (&v)[COUNT], __half* dst, size_t pitch, int m,
                                           int rows, bool odd) {
  const uint32_t sel = odd ? 0x3276u : 0x5410u;
#pragma unroll
  for (int c = 0; c < COUNT; c += 2) {
    const uint32_t own = as_u32(__floats2half2_rn(v[c], v[c + 1]));
    const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 1);
    if (m + c < rows) *reinterpret_cast<uint32_t*>(dst) = prmt(own, other, sel);
    dst += 2 * pitch;
  }
}

}  // namespace handover
}  // namespace awq
