// ntt_joint.cuh -- negacyclic 2048-point transforms of K polynomials of one
// CRT residue at once, by a group of 128 threads (4 warps), 16 values of each
// polynomial per thread.  Same transforms, layouts and twiddle order as
// ntt2048.cuh (forward output slot s holds a(psi^(2 brv(s) + 1))).
//
// What differs from ntt2048.cuh, and why:
//  * K polynomials share every twiddle load and every address, and give each
//    warp K times the independent butterflies, so that few warps fill the
//    integer multiply-add pipe (64 lane-operations per cycle and SM, a
//    high product costs two).
//  * Both exchanges keep one XOR-swizzled index map, jsw, in place: a thread
//    overwrites exactly the words it read last, so an exchange needs one
//    barrier (between its writes and its reads) instead of two.  Elements
//    [128 b, 128 b + 128) stay in words [128 b, 128 b + 128), and the 8
//    lanes that exchange them second are one warp's, so that exchange only
//    needs __syncwarp.
//  * The inverse reads the forward table: psi^-brv(k) = -psi^brv(3 m - 1 - k)
//    for k in [m, 2m), m a power of two (brv(k) is 2^(10-s) (2 i' + 1), and
//    complementing i' inside its level negates the exponent mod N), so the
//    difference is taken the other way round.  Half the table stays in L1.
//  * The inverse's sums are reduced only where a 32-bit overflow could
//    follow (bounds are tracked per register at compile time).
#pragma once
#include <cstdint>

#include "ntt2048.cuh"

namespace ig {

// Word of element e in an exchange buffer of 2048 words: a permutation of
// each aligned 128-word block that keeps 4-word chunks together.  Accesses by
// a warp at x + 128 r, at 128 b + y + 8 r (x = 8 b + y) and, as 128-bit
// chunks, at 16 x .. 16 x + 15 are all free of bank conflicts.
__device__ __forceinline__ int jsw(int e) { return e ^ (((e >> 5) & 3) << 2) ^ (((e >> 7) & 3) << 3); }

// x in [0, b q) -> [0, max(c, b - c) q)
__device__ __forceinline__ uint32_t csub(uint32_t x, uint32_t cq) { return min(x, x - cq); }

// Exchange accesses.  tr: elements 128 b + y + 8 r; ru: elements 16 x + r.
template <int K>
__device__ __forceinline__ void jx_store_tr(const uint32_t (&v)[K][16], uint32_t* const (&sc)[K], int x) {
  const int e0 = 128 * (x >> 3) + ((x & 7) ^ (((x >> 3) & 3) << 3));
#pragma unroll
  for (int r = 0; r < 16; r++) {
    const int o = (e0 ^ (((r & 3) ^ (r >> 3)) << 3) ^ (((r >> 2) & 1) << 2)) + 32 * (r >> 2);
#pragma unroll
    for (int k = 0; k < K; k++) sc[k][o] = v[k][r];
  }
}
template <int K>
__device__ __forceinline__ void jx_load_tr(uint32_t (&v)[K][16], uint32_t* const (&sc)[K], int x) {
  const int e0 = 128 * (x >> 3) + ((x & 7) ^ (((x >> 3) & 3) << 3));
#pragma unroll
  for (int r = 0; r < 16; r++) {
    const int o = (e0 ^ (((r & 3) ^ (r >> 3)) << 3) ^ (((r >> 2) & 1) << 2)) + 32 * (r >> 2);
#pragma unroll
    for (int k = 0; k < K; k++) v[k][r] = sc[k][o];
  }
}
template <int K>
__device__ __forceinline__ void jx_store_co(const uint32_t (&v)[K][16], uint32_t* const (&sc)[K], int x) {
  const int e0 = x ^ (((x >> 5) & 3) << 2);
#pragma unroll
  for (int r = 0; r < 16; r++) {
    const int o = (e0 ^ ((r & 3) << 3)) + 128 * r;
#pragma unroll
    for (int k = 0; k < K; k++) sc[k][o] = v[k][r];
  }
}
template <int K>
__device__ __forceinline__ void jx_load_co(uint32_t (&v)[K][16], uint32_t* const (&sc)[K], int x) {
  const int e0 = x ^ (((x >> 5) & 3) << 2);
#pragma unroll
  for (int r = 0; r < 16; r++) {
    const int o = (e0 ^ ((r & 3) << 3)) + 128 * r;
#pragma unroll
    for (int k = 0; k < K; k++) v[k][r] = sc[k][o];
  }
}
template <int K>
__device__ __forceinline__ void jx_store_ru(const uint32_t (&v)[K][16], uint32_t* const (&sc)[K], int x) {
  const int e0 = (16 * x) ^ (((x >> 1) & 3) << 2) ^ (((x >> 3) & 3) << 3);
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int k = 0; k < K; k++)
      *reinterpret_cast<uint4*>(sc[k] + (e0 ^ (4 * c))) =
          make_uint4(v[k][4 * c], v[k][4 * c + 1], v[k][4 * c + 2], v[k][4 * c + 3]);
}
template <int K>
__device__ __forceinline__ void jx_load_ru(uint32_t (&v)[K][16], uint32_t* const (&sc)[K], int x) {
  const int e0 = (16 * x) ^ (((x >> 1) & 3) << 2) ^ (((x >> 3) & 3) << 3);
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint4 t = *reinterpret_cast<const uint4*>(sc[k] + (e0 ^ (4 * c)));
      v[k][4 * c] = t.x;
      v[k][4 * c + 1] = t.y;
      v[k][4 * c + 2] = t.z;
      v[k][4 * c + 3] = t.w;
    }
}

// Forward stage S (element r pairs with r + H, twiddle (1 << S) + first +
// (r >> SHIFT)) of K polynomials.
template <int K, int S, int SHIFT>
__device__ __forceinline__ void jfwd_stage(uint32_t (&v)[K][16], TwiddleRef tw, int first, uint32_t q, uint32_t q2) {
  constexpr int CNT = 16 >> SHIFT;
  constexpr int H = (S < 4) ? (8 >> S) : (S < 8 ? (8 >> (S - 4)) : (4 >> (S - 8)));
  uint2 run[CNT];
  tw_run<CNT>(tw, (1 << S) + first, run);
#pragma unroll
  for (int r = 0; r < 16; r++)
    if ((r & H) == 0)
#pragma unroll
      for (int k = 0; k < K; k++) ct_bfly(v[k][r], v[k][r + H], run[r >> SHIFT], q, q2);
}

// Forward transforms, coefficient layout (v[k][r] = a_k[x + 128 r]) in, slot
// layout (v[k][r] = A_k[16 x + r], [0, 14 q)) out.  Inputs below 2^20
// (gadget digits), or below q with FULL.  sc[k]: K exchange buffers of 2048
// words, whose words at this thread's coefficient positions (jsw(x + 128 r))
// must be free to this thread; bar: the group's named barrier.
//
// Bounds (q < 2^28, so 16 q < 2^32): a stage adds at most 2 q, or 1 + B / 16
// to its sums where the twiddled operand is below B q.  Digits: below 8 q +
// 2^20 after stages 0-3; in stages 4-7 only element 14, the one that takes
// the difference three times, could pass 16 q, and is reduced before stage
// 7.  One reduction below 8 q before stages 8-10, which end below 14 q.
template <int K, bool FULL>
__device__ __forceinline__ void jntt_fwd(uint32_t (&v)[K][16], uint32_t* const (&sc)[K], TwiddleRef tw, uint32_t q,
                                         int x, int bar) {
  const uint32_t q2 = 2 * q, q8 = 8 * q;
  jfwd_stage<K, 0, 4>(v, tw, 0, q, q2);
  jfwd_stage<K, 1, 3>(v, tw, 0, q, q2);
  jfwd_stage<K, 2, 2>(v, tw, 0, q, q2);
  jfwd_stage<K, 3, 1>(v, tw, 0, q, q2);
  if (FULL) {
#pragma unroll
    for (int k = 0; k < K; k++) reduce_8q(v[k], q);  // < 9 q -> < 8 q
  }
  jx_store_co<K>(v, sc, x);
  group_sync(bar);
  jx_load_tr<K>(v, sc, x);
  const int b = x >> 3;
  jfwd_stage<K, 4, 4>(v, tw, b, q, q2);
  jfwd_stage<K, 5, 3>(v, tw, b << 1, q, q2);
  jfwd_stage<K, 6, 2>(v, tw, b << 2, q, q2);
#pragma unroll
  for (int k = 0; k < K; k++) v[k][14] = csub(v[k][14], q8);
  jfwd_stage<K, 7, 1>(v, tw, b << 3, q, q2);
#pragma unroll
  for (int k = 0; k < K; k++) reduce_8q(v[k], q);  // < 16 q -> < 8 q
  jx_store_tr<K>(v, sc, x);
  __syncwarp();
  jx_load_ru<K>(v, sc, x);
  jfwd_stage<K, 8, 3>(v, tw, x << 1, q, q2);
  jfwd_stage<K, 9, 2>(v, tw, x << 2, q, q2);
  jfwd_stage<K, 10, 1>(v, tw, x << 3, q, q2);
}

// Inverse stage S.  B[r]: bound of element r in multiples of q, known at
// compile time (the loops unroll); sums that could pass 16 q are avoided by
// reducing an operand above 8 q first.
template <int K, int S, int SHIFT>
__device__ __forceinline__ void jinv_stage(uint32_t (&v)[K][16], int (&B)[16], TwiddleRef fwd, int first, uint32_t q) {
  constexpr int CNT = 16 >> SHIFT;
  constexpr int H = (S < 4) ? (8 >> S) : (S < 8 ? (8 >> (S - 4)) : (4 >> (S - 8)));
  // twiddles (1 << S) + first + c, c < CNT, as -fwd[3 (1 << S) - 1 - that]
  uint2 run[CNT];
  tw_run<CNT>(fwd, (2 << S) - CNT - first, run);
#pragma unroll
  for (int r = 0; r < 16; r++)
    if ((r & H) == 0) {
      if (B[r] + B[r + H] > 16) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
          if (B[r + e * H] > 8) {
#pragma unroll
            for (int k = 0; k < K; k++) v[k][r + e * H] = csub(v[k][r + e * H], 8 * q);
            B[r + e * H] = 8;
          }
        }
      }
      const uint32_t bq = (uint32_t)B[r] * q;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t a = v[k][r], b = v[k][r + H];
        v[k][r] = a + b;
        v[k][r + H] = mul_shoup_lazy(b - a + bq, run[CNT - 1 - (r >> SHIFT)], q);
      }
      B[r] += B[r + H];
      B[r + H] = 2;
    }
}

// Reduce every element to below C q, C = 4 (before an exchange) or 1.
template <int K, int C>
__device__ __forceinline__ void jinv_reduce(uint32_t (&v)[K][16], int (&B)[16], uint32_t q) {
#pragma unroll
  for (int r = 0; r < 16; r++) {
#pragma unroll
    for (int c = 8; c >= C; c >>= 1) {
      if (B[r] > c) {
#pragma unroll
        for (int k = 0; k < K; k++) v[k][r] = csub(v[k][r], (uint32_t)c * q);
        B[r] = c;
      }
    }
  }
}

// Inverse transforms without the n^-1 factor, slot layout ([0, 4 q)) in,
// coefficient layout out, canonical.  `fwd` is the forward table.  sc[k]'s
// words at this thread's slot positions must be free to this thread; it
// reads its coefficient positions last.
template <int K>
__device__ __forceinline__ void jntt_inv(uint32_t (&v)[K][16], uint32_t* const (&sc)[K], TwiddleRef fwd, uint32_t q,
                                         int x, int bar) {
  int B[16];
#pragma unroll
  for (int r = 0; r < 16; r++) B[r] = 4;
  jinv_stage<K, 10, 1>(v, B, fwd, x << 3, q);
  jinv_stage<K, 9, 2>(v, B, fwd, x << 2, q);
  jinv_stage<K, 8, 3>(v, B, fwd, x << 1, q);
  jinv_reduce<K, 4>(v, B, q);
  jx_store_ru<K>(v, sc, x);
  __syncwarp();
  jx_load_tr<K>(v, sc, x);
  const int b = x >> 3;
#pragma unroll
  for (int r = 0; r < 16; r++) B[r] = 4;
  jinv_stage<K, 7, 1>(v, B, fwd, b << 3, q);
  jinv_stage<K, 6, 2>(v, B, fwd, b << 2, q);
  jinv_stage<K, 5, 3>(v, B, fwd, b << 1, q);
  jinv_stage<K, 4, 4>(v, B, fwd, b, q);
  jinv_reduce<K, 4>(v, B, q);
  jx_store_tr<K>(v, sc, x);
  group_sync(bar);
  jx_load_co<K>(v, sc, x);
#pragma unroll
  for (int r = 0; r < 16; r++) B[r] = 4;
  jinv_stage<K, 3, 1>(v, B, fwd, 0, q);
  jinv_stage<K, 2, 2>(v, B, fwd, 0, q);
  jinv_stage<K, 1, 3>(v, B, fwd, 0, q);
  jinv_stage<K, 0, 4>(v, B, fwd, 0, q);
  jinv_reduce<K, 1>(v, B, q);
}

}  // namespace ig
