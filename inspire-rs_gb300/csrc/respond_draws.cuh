// respond_draws.cuh -- device code that the Respond kernels (respond.cu,
// respond_pair.cu) share: drawing a row's polynomial from its seed by 256
// threads, streaming loads and signed 64-bit sums of products.
#pragma once
#include "expand.cuh"
#include "kernels.h"
#include "respond_common.cuh"

namespace ig {

constexpr int QT = 256;         // threads that expand a query's rows together
constexpr int EXPAND_BAR = 10;  // their named barrier (barrier 0 may be waited at by other warps of the CTA)

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
  return expand_seeded_row<NR>(P, seed, cand, a0, a0 + N, ws, 7, threadIdx.x);
}

// Poly::from_seed_moduli (poly.rs:251-281) of the ELL rows by threads 0-255
// (barrier EXPAND_BAR), row t residue r to AH[(t NR + r) N ..].  ws: 23 ints, of which [20 + t] is
// left 1 if row t is complete.
// Draws 0 .. 2047 (blocks 0-255, a thread each) go to residue 0, whose few
// missing values (rejections: 2^28 - q of 2^28 draws) come from the start of
// the next 256 blocks, found by warp 0; residue 1 follows there, and one warp
// per row draws the last ~155 values.  Seven rounds of ChaCha20 for the three
// rows together (one row after the other needs nine, three of them tails of
// one warp).  A row whose stream rejects more than that leaves 0 in
// ok[row]: a general pass redoes it.
template <int NR>
__device__ __forceinline__ void expand_rows(const DevParams& P, const uint8_t* seeds, uint32_t* AH, int* ws) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;  // tid < 256
  const uint32_t q0 = P.r[0].q, z0 = (uint32_t)(P.r[0].zone >> 32);
  const uint32_t q1 = P.r[1].q, z1 = (uint32_t)(P.r[1].zone >> 32);
  int* tot = ws + 16;   // [ELL] values drawn so far: residue 0, then residue 1
  int* ok = ws + 20;    // [ELL]
#pragma unroll 1
  for (int t = 0; t < ELL; t++) {
    uint32_t key[8], w[16], val[8];
    load_key(seeds + 32 * t, key);
    chacha20_block(key, tid, P.one, w);
    const unsigned mask = draw8(w, q0, z0, val);
    int total;
    const int p = scan_256(__popc(mask), ws + 8 * (t & 1), total, EXPAND_BAR);
    put_draws(AH + t * NR * N, p, mask, val);
    if (tid == 0) tot[t] = total;
  }
  named_sync(EXPAND_BAR, QT);
  if (NR == 2) {
#pragma unroll 1
    for (int t = 0; t < ELL; t++) {
      uint32_t key[8], w[16], val[8];
      load_key(seeds + 32 * t, key);
      chacha20_block(key, QT + tid, P.one, w);
      uint32_t* a0 = AH + t * NR * N;
      int start = 0;  // warp 0: draws before it belong to residue 0
      if (warp == 0) {
        const int have = tot[t];
        if (have < N) {  // uniform over the warp
          const unsigned m0 = draw8(w, q0, z0, val);
          int all;
          const int p = have + scan_warp(__popc(m0), all);
          put_draws(a0, p, m0, val);
          // the lane that holds value N - 1 knows where residue 1 starts
          int end = 0, pp = p;
#pragma unroll
          for (int k = 0; k < 8; k++)
            if ((m0 >> k) & 1u) {
              if (pp == N - 1) end = 8 * lane + k + 1;
              pp++;
            }
          start = __reduce_max_sync(0xffffffffu, end);
          if (lane == 0) ok[t] = start != 0;
        } else if (lane == 0) {
          ok[t] = 1;
        }
      }
      unsigned mask = draw8(w, q1, z1, val);
      if (warp == 0) {
        const int skip = start - 8 * lane;  // leading draws of this lane to skip
        if (skip > 0) mask &= skip >= 8 ? 0u : ~((1u << skip) - 1u);
      }
      int total;
      const int p = scan_256(__popc(mask), ws + 8 * ((t + 1) & 1), total, EXPAND_BAR);
      put_draws(a0 + N, p, mask, val);
      if (tid == 0) tot[t] = total;
    }
    named_sync(EXPAND_BAR, QT);
  }
  if (warp < ELL) {  // the tails, one warp per row
    const int t = warp;
    uint32_t key[8], w[16], val[8];
    load_key(seeds + 32 * t, key);
    chacha20_block(key, (NR == 2 ? 2 * QT : QT) + lane, P.one, w);
    const unsigned mask = NR == 2 ? draw8(w, q1, z1, val) : draw8(w, q0, z0, val);
    int all;
    const int have = tot[t];
    const int p = have + scan_warp(__popc(mask), all);
    put_draws(AH + (t * NR + NR - 1) * N, p, mask, val);
    if (lane == 0) ok[t] = (NR == 1 || ok[t]) && have + all >= N;
  }
}

// Serving loop: the query's b rows (u64) are staged in four chunks, one after
// the other in the exchange buffers.  Chunk m covers coefficients i in
// [512 m, 512 m + 512) of the reversed rows, i.e. row words N - i: words
// 512 (3 - m) .. and one pair more (for m = 0 that pair is words 0, 1).
constexpr int CH = 512;
constexpr int CHW = CH + 2;  // u64 words of one polynomial's chunk
static_assert(2 * ELL * CHW * 8 <= 4 * N * 4, "a chunk fits the exchange buffers");

__device__ __forceinline__ void stage_chunk(uint64_t* dst, const uint64_t* brows, int m, uint64_t* bar) {
  mbar_expect_tx(bar, 2 * ELL * CHW * 8);
  const int k0 = N - CH * (m + 1);
#pragma unroll 1
  for (int p = 0; p < 2 * ELL; p++) {
    uint64_t* d = dst + p * CHW;
    const uint64_t* s = brows + (size_t)p * N;
    if (m == 0) {
      bulk_g2s(d, s + k0, CH * 8, bar);
      bulk_g2s(d + CH, s, 16, bar);
    } else {
      bulk_g2s(d, s + k0, CHW * 8, bar);
    }
  }
}

// Where a query's b rows come from: device (or mapped) memory, read where used;
// staged chunks; or staged as a whole.
enum RowSource { ROWS_DIRECT, ROWS_CHUNKS, ROWS_WHOLE };

// The whole rows (96 KiB) on one mbarrier.
__device__ __forceinline__ void stage_rows(uint64_t* dst, const uint64_t* brows, uint64_t* bar) {
  mbar_expect_tx(bar, 2 * ELL * N * 8);
#pragma unroll 1
  for (int p = 0; p < 2 * ELL; p++) bulk_g2s(dst + p * N, brows + (size_t)p * N, N * 8, bar);
}

// The b side of the column products, coefficient 0 only (rlwe/enc.rs:195-208;
// see respond.cu) by 256 threads (whole warps, barrier `named`; staged rows: the
// whole CTA): b0_c = -sum_i d_{c}[i] v[i] with v[0] = q - b[0], v[i] = b[N - i].
// Thread tid takes the coefficient pairs j = tid +
// 256 m, m < 4, of every column, so each row word is read once, straight
// from its buffer (or where it is staged), and every column word once;
// 32 sums (column, residue) per thread, exact in 64 bits (6144 products below
// 2^48), are then transposed and added over the warp by shuffles, five
// halving exchanges, and over the warps in shared memory.
// Returns -1, or the chunk (0: the rows) that did not arrive.
template <RowSource SRC>
__device__ __forceinline__ int column_b0(const DevParams& P, const uint16_t* __restrict__ H, const uint64_t* brows,
                                          uint64_t* stage, uint64_t* bar, uint32_t wait_iters, uint64_t* red,
                                          uint32_t* bpoly, int named = 0) {
  const int tid = threadIdx.x & 255, lane = tid & 31, warp = tid >> 5, gamma = P.gamma;
  const uint32_t* h2 = reinterpret_cast<const uint32_t*>(H) + tid;
  uint64_t acc[32];  // [column][residue]
#pragma unroll
  for (int k = 0; k < 32; k++) acc[k] = 0;
  if (SRC == ROWS_WHOLE) {
    const bool arrived = mbar_wait(bar, 0, wait_iters);
    if (__syncthreads_or(!arrived)) return 0;
  }
#pragma unroll 1
  for (int m = 0; m < 4; m++) {
    uint32_t hw[MAX_GAMMA];
#pragma unroll
    for (int c = 0; c < MAX_GAMMA; c++) hw[c] = c < gamma ? __ldg(h2 + (size_t)c * (N / 2) + QT * m) : 0u;
    uint32_t bv[2][2 * ELL];
    const int i0 = 2 * (tid + QT * m);
    if (SRC == ROWS_CHUNKS) {
      const bool arrived = mbar_wait(bar, m & 1, wait_iters);
      if (__syncthreads_or(!arrived)) return m;
      const uint32_t* s = reinterpret_cast<const uint32_t*>(stage);
#pragma unroll
      for (int p = 0; p < 2 * ELL; p++) {
        bv[0][p] = s[2 * (p * CHW + CH - 2 * tid)];
        bv[1][p] = s[2 * (p * CHW + CH - 2 * tid - 1)];
      }
      if (m < 3) {
        __syncthreads();
        if (tid == 0) {
          // the next chunk's copies (async proxy) follow these reads
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          stage_chunk(stage, brows, m + 1, bar);
        }
      }
    } else {
      const uint32_t* s = reinterpret_cast<const uint32_t*>(SRC == ROWS_WHOLE ? stage : brows);
      const int k0 = i0 ? N - i0 : 0, k1 = N - i0 - 1;
#pragma unroll
      for (int p = 0; p < 2 * ELL; p++) {
        bv[0][p] = SRC == ROWS_WHOLE ? s[2 * (p * N + k0)] : __ldg(s + 2 * (p * N + k0));
        bv[1][p] = SRC == ROWS_WHOLE ? s[2 * (p * N + k1)] : __ldg(s + 2 * (p * N + k1));
      }
    }
    if (i0 == 0) {
#pragma unroll
      for (int p = 0; p < 2 * ELL; p++) bv[0][p] = P.r[p & 1].q - bv[0][p];
    }
#pragma unroll
    for (int c = 0; c < MAX_GAMMA; c++) {
      if (c >= gamma) continue;
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const uint64_t xv = P.delta * (uint64_t)((hw[c] >> (16 * e)) & 0xFFFFu);
        const uint32_t d0 = (uint32_t)xv & 0xFFFFFu, d1 = (uint32_t)(xv >> 20) & 0xFFFFFu, d2 = (uint32_t)(xv >> 40);
        acc[2 * c] += (uint64_t)d0 * bv[e][0] + (uint64_t)d1 * bv[e][2] + (uint64_t)d2 * bv[e][4];
        acc[2 * c + 1] += (uint64_t)d0 * bv[e][1] + (uint64_t)d1 * bv[e][3] + (uint64_t)d2 * bv[e][5];
      }
    }
  }
  // lane l ends with the warp's sum of value l
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < o; k++) {
      const uint64_t send = up ? acc[k] : acc[k + o], keep = up ? acc[k + o] : acc[k];
      acc[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  if (SRC == ROWS_CHUNKS) named_sync(named, QT);  // the last chunk has been read
  red[warp * 32 + lane] = acc[0];
  named_sync(named, QT);
  if (tid < 32) {
    uint64_t s = 0;
#pragma unroll
    for (int w = 0; w < QT / 32; w++) s += red[w * 32 + tid];
    const uint32_t q = P.r[tid & 1].q;
    const uint32_t v = (uint32_t)(s % q);
    bpoly[(tid & 1) * 16 + (tid >> 1)] = v ? q - v : 0;
  }
  named_sync(named, QT);
  return -1;
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
