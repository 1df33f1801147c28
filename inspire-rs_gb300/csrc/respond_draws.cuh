// respond_draws.cuh -- device code that the Respond kernels (respond.cu,
// respond_pair.cu) share: drawing a row's polynomial from its seed by 256
// threads, streaming loads and signed 64-bit sums of products.
#pragma once
#include "expand.cuh"
#include "kernels.h"
#include "respond_common.cuh"

namespace ig {

// Exclusive rank of this thread's `cnt` over 256 threads (eight whole warps,
// named barrier `bar`), and the total.  ws: 8 ints of this call's own (reused
// two calls later at the earliest).
__device__ __forceinline__ int scan_256(int cnt, int* ws, int& total, int bar) {
  const int lane = threadIdx.x & 31, warp = (threadIdx.x & 255) >> 5;
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) ws[warp] = incl;
  named_sync(bar, 256);
  int base = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < 8; w++) {
    const int t = ws[w];
    if (w < warp) base += t;
    total += t;
  }
  return base + incl - cnt;
}

__device__ __forceinline__ int scan_warp(int cnt, int& total) {
  const int lane = threadIdx.x & 31;
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  total = __shfl_sync(0xffffffffu, incl, 31);
  return incl - cnt;
}

__device__ __forceinline__ void load_key(const uint8_t* seed, uint32_t key[8]) {
  const uint32_t* s = reinterpret_cast<const uint32_t*>(seed);
  if ((reinterpret_cast<uintptr_t>(seed) & 3) == 0) {
#pragma unroll
    for (int i = 0; i < 8; i++) key[i] = s[i];
  } else {
#pragma unroll
    for (int i = 0; i < 8; i++)
      key[i] = (uint32_t)seed[4 * i] | ((uint32_t)seed[4 * i + 1] << 8) | ((uint32_t)seed[4 * i + 2] << 16) |
               ((uint32_t)seed[4 * i + 3] << 24);
  }
}

// The eight draws of one keystream block under gen_range(0..q): bit k of the
// mask is set if draw k is accepted, val[k] its value.  zone = (q << lz) - 1
// has 32 low ones (q < 2^32), so lo64(v q) <= zone is decided by the high
// words.
__device__ __forceinline__ unsigned draw8(const uint32_t w[16], uint32_t q, uint32_t zone_hi, uint32_t val[8]) {
  unsigned mask = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const uint64_t hi = (uint64_t)w[2 * k + 1] * q + __umulhi(w[2 * k], q);
    val[k] = (uint32_t)(hi >> 32);
    mask |= ((uint32_t)hi <= zone_hi ? 1u : 0u) << k;
  }
  return mask;
}

__device__ __forceinline__ void put_draws(uint32_t* dst, int p, unsigned mask, const uint32_t val[8]) {
#pragma unroll
  for (int k = 0; k < 8; k++)
    if ((mask >> k) & 1u) {
      if (p < N) dst[p] = val[k];
      p++;
    }
}

// One row by the general routine (threads 0-255), for streams that reject more
// draws than the fast path allows for.
template <int NR>
__device__ __noinline__ bool expand_row_general(const DevParams& P, const uint8_t* seed, uint64_t* cand, uint32_t* a0,
                                                int* ws) {
  return expand_seeded_row<NR>(P, seed, cand, a0, a0 + N, ws, 3, threadIdx.x);
}

// Streaming loads of the contracted shard and the CRS keys: read once per
// query, kept out of L1 (which holds the twiddles and the client's keys).
__device__ __forceinline__ uint4 ld_stream(const uint32_t* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// REDC of a signed sum T: T 2^-32 mod q in [T / 2^32, T / 2^32 + q).
__device__ __forceinline__ uint32_t redc_wide(uint64_t T, uint32_t q, uint32_t qinv) {
  const uint32_t m = (uint32_t)T * qinv;
  return (uint32_t)((T + (uint64_t)m * q) >> 32);
}

// a * b of two signed 32-bit values, as a 64-bit sum's term.
__device__ __forceinline__ uint64_t smul(uint32_t a, uint32_t b) { return (uint64_t)((int64_t)(int32_t)a * (int32_t)b); }

}  // namespace ig
