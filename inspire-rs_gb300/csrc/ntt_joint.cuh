// ntt_joint.cuh -- negacyclic 2048-point transforms of K polynomials of one
// CRT residue at once, by a group of 128 threads (4 warps), 16 values of each
// polynomial per thread.  Same transforms, layouts and twiddle order as
// ntt2048.cuh (forward output slot s holds a(psi^(2 brv(s) + 1))).
//
// What differs from ntt2048.cuh, and why:
//  * K polynomials share every twiddle load and every address, and give each
//    warp K times the independent butterflies, so that few warps fill the
//    integer multiply-add pipe (64 lane-operations per cycle and SM, a
//    high product costs two: at most 16 butterflies per cycle).
//  * One table of centred twiddles w in (-q/2, q/2) with companions
//    w' = round(w 2^32 / q) and signed products: for |a| < 2^31,
//    a w - floor(a w' / 2^32) q = a w mod q in (-|a| / 2^33 q, q + |a| / 2^33 q).
//    The forward butterfly is then a' = (b w + a) - h q, b' = 2a - a': four
//    instructions, none with three different added registers (measured in
//    registers: 14.5 butterflies per cycle and SM, 12.4 as x + t, x - t + 2q
//    on unsigned values); the inverse one takes the difference without an
//    offset (13.9, 11.6 with it).
//  * Values are reduced only where 32 bits would overflow: their bounds are
//    tracked per register at compile time.
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
#pragma once
#include <cstdint>

#include "common.cuh"

namespace ig {

// Word of element e in an exchange buffer of 2048 words: a permutation of
// each aligned 128-word block that keeps 4-word chunks together.  Accesses by
// a warp at x + 128 r, at 128 b + y + 8 r (x = 8 b + y) and, as 128-bit
// chunks, at 16 x .. 16 x + 15 are all free of bank conflicts.
__device__ __forceinline__ int jsw(int e) { return e ^ (((e >> 5) & 3) << 2) ^ (((e >> 7) & 3) << 3); }

// x in [0, b q) -> [0, max(c, b - c) q)
__device__ __forceinline__ uint32_t csub(uint32_t x, uint32_t cq) { return min(x, x - cq); }
// signed x in (-2 c, 2 c) -> [-c, c), c a multiple of q
__device__ __forceinline__ uint32_t centre(uint32_t x, uint32_t c) {
  return x - c + ((uint32_t)((int32_t)x >> 31) & (2 * c));
}

// 2 a - b as additions: the compiler would turn 2 a - b into a multiply-add,
// on the pipe that the transforms are bound by.
__device__ __forceinline__ uint32_t twice_minus(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d + a;
}

// Exchange buffers are addressed by 32-bit shared-memory addresses, a
// multiple of 128 bytes, so that a swizzled access is one XOR away from its
// thread's base.
__device__ __forceinline__ uint32_t jx_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t& jx_at(uint32_t a) {
  return *reinterpret_cast<uint32_t*>(__cvta_shared_to_generic(a));
}
__device__ __forceinline__ uint4& jx_at4(uint32_t a) { return *reinterpret_cast<uint4*>(__cvta_shared_to_generic(a)); }

// Byte offsets of this thread's first element in the three layouts.
__device__ __forceinline__ uint32_t jx_co(int x) { return 4u * (uint32_t)(x ^ (((x >> 5) & 3) << 2)); }
__device__ __forceinline__ uint32_t jx_tr(int x) {
  return 4u * (uint32_t)(128 * (x >> 3) + ((x & 7) ^ (((x >> 3) & 3) << 3)));
}
__device__ __forceinline__ uint32_t jx_ru(int x) {
  return 4u * (uint32_t)((16 * x) ^ (((x >> 1) & 3) << 2) ^ (((x >> 3) & 3) << 3));
}
// Element r's distance from it: an XOR of bits 2-6 and a multiple of 128.
__host__ __device__ constexpr uint32_t jx_co_x(int r) { return 4u * ((r & 3) << 3); }
__host__ __device__ constexpr uint32_t jx_co_o(int r) { return 4u * 128u * (uint32_t)r; }
__host__ __device__ constexpr uint32_t jx_tr_x(int r) { return 4u * ((((r & 3) ^ (r >> 3)) << 3) ^ (((r >> 2) & 1) << 2)); }
__host__ __device__ constexpr uint32_t jx_tr_o(int r) { return 4u * 32u * (uint32_t)(r >> 2); }

template <int K>
__device__ __forceinline__ void jx_store_tr(const uint32_t (&v)[K][16], const uint32_t (&sc)[K], int x) {
#pragma unroll
  for (int r = 0; r < 16; r++)
#pragma unroll
    for (int k = 0; k < K; k++) jx_at(((sc[k] + jx_tr(x)) ^ jx_tr_x(r)) + jx_tr_o(r)) = v[k][r];
}
template <int K>
__device__ __forceinline__ void jx_load_tr(uint32_t (&v)[K][16], const uint32_t (&sc)[K], int x) {
#pragma unroll
  for (int r = 0; r < 16; r++)
#pragma unroll
    for (int k = 0; k < K; k++) v[k][r] = jx_at(((sc[k] + jx_tr(x)) ^ jx_tr_x(r)) + jx_tr_o(r));
}
template <int K>
__device__ __forceinline__ void jx_store_co(const uint32_t (&v)[K][16], const uint32_t (&sc)[K], int x) {
#pragma unroll
  for (int r = 0; r < 16; r++)
#pragma unroll
    for (int k = 0; k < K; k++) jx_at(((sc[k] + jx_co(x)) ^ jx_co_x(r)) + jx_co_o(r)) = v[k][r];
}
template <int K>
__device__ __forceinline__ void jx_load_co(uint32_t (&v)[K][16], const uint32_t (&sc)[K], int x) {
#pragma unroll
  for (int r = 0; r < 16; r++)
#pragma unroll
    for (int k = 0; k < K; k++) v[k][r] = jx_at(((sc[k] + jx_co(x)) ^ jx_co_x(r)) + jx_co_o(r));
}
template <int K>
__device__ __forceinline__ void jx_store_ru(const uint32_t (&v)[K][16], const uint32_t (&sc)[K], int x) {
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int k = 0; k < K; k++)
      jx_at4((sc[k] + jx_ru(x)) ^ (16u * c)) = make_uint4(v[k][4 * c], v[k][4 * c + 1], v[k][4 * c + 2], v[k][4 * c + 3]);
}
template <int K>
__device__ __forceinline__ void jx_load_ru(uint32_t (&v)[K][16], const uint32_t (&sc)[K], int x) {
#pragma unroll
  for (int c = 0; c < 4; c++)
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint4 t = jx_at4((sc[k] + jx_ru(x)) ^ (16u * c));
      v[k][4 * c] = t.x;
      v[k][4 * c + 1] = t.y;
      v[k][4 * c + 2] = t.z;
      v[k][4 * c + 3] = t.w;
    }
}

// The warp's 512 elements of a buffer as coalesced 128-bit words: chunk c of
// lane l is elements 512 w + 128 c + 4 l .. + 3.  Between these and the slot
// layout (jx_store_ru, jx_load_ru) only the warp's own words move.
__device__ __forceinline__ uint32_t jx_lin(int x, int c) {
  return 4u * (uint32_t)jsw(512 * (x >> 5) + 128 * c + 4 * (x & 31));
}

// ---- bounds: element r is below B[r] q / 64 (in absolute value in the
//      forward transform); 32-bit signed values allow 8 q = 512 units ----
constexpr int JB_MAX = 512;

template <int V>
__host__ __device__ constexpr int jb_max(const int (&B)[V]) {
  int m = 0;
  for (int r = 0; r < V; r++) m = B[r] > m ? B[r] : m;
  return m;
}
// After an exchange any value may be any register's.
template <int V>
__host__ __device__ constexpr void jb_level(int (&B)[V]) {
  const int m = jb_max(B);
  for (int r = 0; r < V; r++) B[r] = m;
}
// A forward butterfly's bounds, a' = a + (b w mod q), b' = a - (b w mod q);
// true if a has to be centred first.
__host__ __device__ constexpr bool jb_fwd(int& a, int& b) {
  const int grow = 64 + (b + 31) / 32;  // |b w mod q| <= q (1 + |b| / 2^33)
  const bool c = a + grow > JB_MAX;
  if (c) a = JB_MAX / 2;
  a += grow;
  b = a;
  return c;
}

// Forward stage S (element r pairs with r + H, twiddle (1 << S) + first +
// (r >> SHIFT)) of K polynomials.
template <int K, int S, int SHIFT>
__device__ __forceinline__ void jfwd_stage(uint32_t (&v)[K][16], int (&B)[16], TwiddleRef tw, int first, uint32_t q) {
  constexpr int CNT = 16 >> SHIFT;
  constexpr int H = (S < 4) ? (8 >> S) : (S < 8 ? (8 >> (S - 4)) : (4 >> (S - 8)));
  uint2 run[CNT];
  tw_run<CNT>(tw, (1 << S) + first, run);
#pragma unroll
  for (int r = 0; r < 16; r++)
    if ((r & H) == 0) {
      if (jb_fwd(B[r], B[r + H])) {
#pragma unroll
        for (int k = 0; k < K; k++) v[k][r] = centre(v[k][r], 4 * q);
      }
      const uint2 w = run[r >> SHIFT];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t a = v[k][r], b = v[k][r + H];
        const uint32_t h = (uint32_t)__mulhi((int)b, (int)w.y);
        const uint32_t s = b * w.x + a;
        v[k][r] = s - h * q;
        v[k][r + H] = twice_minus(a, v[k][r]);
      }
    }
}

// Forward transforms, coefficient layout (v[k][r] = a_k[x + 128 r]) in, slot
// layout (v[k][r] = A_k[16 x + r], signed, below JFWD_OUT q / 64) out.
// Inputs in [0, B0 q / 64), B0 = JB_DIGIT for gadget digits.  sc[k]: K exchange
// buffers of 2048 words, whose words at this thread's coefficient positions
// (jsw(x + 128 r)) must be free to this thread; bar: the group's named barrier.
//
// Digits (below 2^20) count as 1/64 q: for q near 2^28 they are 1/256 q, and
// for smaller q every bound, an absolute sum of 2^20 and multiples of q, is
// smaller too.
constexpr int JB_DIGIT = 1, JB_CANON = 64;
constexpr int JFWD_OUT = 416, JFWD_OUT_DIGIT = 336;  // 6.5 q, 5.25 q: what the callers' sums are bounded with

// The bound that the stages below reach: V values per thread, `phases` runs of
// stages on register bits from the highest down, by their counts of stages and
// their highest register bits.
struct JbPhase {
  int stages, top;
};
template <int V, int NP>
__host__ __device__ constexpr int jfwd_bound(int (&B)[V], const JbPhase (&phases)[NP], int first = 0) {
  for (int p = 0; p < NP; p++) {
    if (p) jb_level(B);
    for (int s = p ? 0 : first; s < phases[p].stages; s++) {
      const int H = phases[p].top >> s;
      for (int r = 0; r < V; r++)
        if ((r & H) == 0) jb_fwd(B[r], B[r + H]);
    }
  }
  return jb_max(B);
}
// ... of inputs below b0 q / 64, by 16 values per thread (stages 0-3, 4-7, 8-10)
__host__ __device__ constexpr int jfwd_out(int b0) {
  const JbPhase phases[3] = {{4, 8}, {4, 8}, {3, 4}};
  int B[16] = {};
  for (int r = 0; r < 16; r++) B[r] = b0;
  return jfwd_bound(B, phases);
}
// ... with stage 0 by multiples of both operands (jntt_fwd_scaled)
__host__ __device__ constexpr int jfwd_out_scaled() {
  const JbPhase phases[3] = {{4, 8}, {4, 8}, {3, 4}};
  int B[16] = {};
  for (int r = 0; r < 16; r++) B[r] = r < 8 ? 256 : 128;
  return jfwd_bound(B, phases, 1);
}
static_assert(jfwd_out(JB_CANON) <= JFWD_OUT && jfwd_out_scaled() <= JFWD_OUT, "forward outputs of residues");
static_assert(jfwd_out(JB_DIGIT) <= JFWD_OUT_DIGIT, "forward outputs of digits");
struct NoHook {
  __device__ __forceinline__ void operator()() const {}
};
// Stages 1-10; `hook` runs before stages 8-10 (to issue loads that they hide).
template <int K, class Hook = NoHook>
__device__ __forceinline__ void jntt_fwd_from1(uint32_t (&v)[K][16], int (&B)[16], const uint32_t (&sc)[K],
                                               TwiddleRef tw, uint32_t q, int x, int bar, Hook&& hook = Hook()) {
  jfwd_stage<K, 1, 3>(v, B, tw, 0, q);
  jfwd_stage<K, 2, 2>(v, B, tw, 0, q);
  jfwd_stage<K, 3, 1>(v, B, tw, 0, q);
  jx_store_co<K>(v, sc, x);
  group_sync(bar);
  jx_load_tr<K>(v, sc, x);
  jb_level(B);
  const int b = x >> 3;
  jfwd_stage<K, 4, 4>(v, B, tw, b, q);
  jfwd_stage<K, 5, 3>(v, B, tw, b << 1, q);
  jfwd_stage<K, 6, 2>(v, B, tw, b << 2, q);
  jfwd_stage<K, 7, 1>(v, B, tw, b << 3, q);
  jx_store_tr<K>(v, sc, x);
  __syncwarp();
  jx_load_ru<K>(v, sc, x);
  hook();
  jb_level(B);
  jfwd_stage<K, 8, 3>(v, B, tw, x << 1, q);
  jfwd_stage<K, 9, 2>(v, B, tw, x << 2, q);
  jfwd_stage<K, 10, 1>(v, B, tw, x << 3, q);
}

template <int K, int B0, class Hook = NoHook>
__device__ __forceinline__ void jntt_fwd(uint32_t (&v)[K][16], const uint32_t (&sc)[K], TwiddleRef tw, uint32_t q, int x,
                                         int bar, Hook&& hook = Hook()) {
  int B[16];
#pragma unroll
  for (int r = 0; r < 16; r++) B[r] = B0;
  jfwd_stage<K, 0, 4>(v, B, tw, 0, q);
  jntt_fwd_from1<K>(v, B, sc, tw, q, x, bar, hook);
}

// The same of c times the input, any 32-bit values: stage 0 multiplies both
// of its operands, by c and by c psi^brv(1) (Shoup pairs c, cw).
template <int K>
__device__ __forceinline__ void jntt_fwd_scaled(uint32_t (&v)[K][16], const uint32_t (&sc)[K], TwiddleRef tw, uint2 c,
                                                uint2 cw, uint32_t q, int x, int bar) {
  int B[16];
#pragma unroll
  for (int r = 0; r < 8; r++) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t a = mul_shoup_lazy(v[k][r], c, q), b = mul_shoup_lazy(v[k][r + 8], cw, q);
      v[k][r] = a + b;
      v[k][r + 8] = a - b;
    }
    B[r] = 256;
    B[r + 8] = 128;
  }
  jntt_fwd_from1<K>(v, B, sc, tw, q, x, bar);
}

// A forward output brought to [0, q).
static_assert(JFWD_OUT <= 8 * 64, "jcanon_fwd");
__device__ __forceinline__ uint32_t jcanon_fwd(uint32_t x, uint32_t q) {
  x = min(x, x + 8 * q);  // negative values are large as unsigned ones
  return canon16(x, q);
}

// Inverse stage S on values in [0, B q / 64): differences signed, operands
// below 8 q; a product of d takes q (1 + |d| / 2^33) around [0, q), plus q.
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
#pragma unroll
      for (int e = 0; e < 2; e++) {
        if (B[r + e * H] > JB_MAX) {
#pragma unroll
          for (int k = 0; k < K; k++) v[k][r + e * H] = csub(v[k][r + e * H], 8 * q);
          B[r + e * H] = JB_MAX;
        }
      }
      const uint2 w = run[CNT - 1 - (r >> SHIFT)];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t a = v[k][r], d = v[k][r + H] - a;
        v[k][r] = a + v[k][r + H];
        const uint32_t h = (uint32_t)__mulhi((int)d, (int)w.y);
        const uint32_t s = d * w.x + q;
        v[k][r + H] = s - h * q;
      }
      const int m = B[r] > B[r + H] ? B[r] : B[r + H];
      B[r] += B[r + H];
      B[r + H] = 128 + (m + 31) / 32;
    }
}

// Reduce every element to below C q, C = 4 (before an exchange) or 1.
template <int K, int C>
__device__ __forceinline__ void jinv_reduce(uint32_t (&v)[K][16], int (&B)[16], uint32_t q) {
#pragma unroll
  for (int r = 0; r < 16; r++) {
#pragma unroll
    for (int c = 8; c >= C; c >>= 1) {
      if (B[r] > 64 * c) {
#pragma unroll
        for (int k = 0; k < K; k++) v[k][r] = csub(v[k][r], (uint32_t)c * q);
        B[r] = 64 * c;
      }
    }
  }
}

// Inverse stages 10-1, slot layout ([0, 4 q)) in, coefficient layout out with
// bounds B.  `fwd` is the forward table.  sc[k]'s words at this thread's slot
// positions must be free to this thread; it reads its coefficient positions
// last.
template <int K>
__device__ __forceinline__ void jntt_inv_to1(uint32_t (&v)[K][16], int (&B)[16], const uint32_t (&sc)[K],
                                             TwiddleRef fwd, uint32_t q, int x, int bar) {
#pragma unroll
  for (int r = 0; r < 16; r++) B[r] = 256;
  jinv_stage<K, 10, 1>(v, B, fwd, x << 3, q);
  jinv_stage<K, 9, 2>(v, B, fwd, x << 2, q);
  jinv_stage<K, 8, 3>(v, B, fwd, x << 1, q);
  jinv_reduce<K, 4>(v, B, q);
  jx_store_ru<K>(v, sc, x);
  __syncwarp();
  jx_load_tr<K>(v, sc, x);
  const int b = x >> 3;
#pragma unroll
  for (int r = 0; r < 16; r++) B[r] = 256;
  jinv_stage<K, 7, 1>(v, B, fwd, b << 3, q);
  jinv_stage<K, 6, 2>(v, B, fwd, b << 2, q);
  jinv_stage<K, 5, 3>(v, B, fwd, b << 1, q);
  jinv_stage<K, 4, 4>(v, B, fwd, b, q);
  jinv_reduce<K, 4>(v, B, q);
  jx_store_tr<K>(v, sc, x);
  group_sync(bar);
  jx_load_co<K>(v, sc, x);
#pragma unroll
  for (int r = 0; r < 16; r++) B[r] = 256;
  jinv_stage<K, 3, 1>(v, B, fwd, 0, q);
  jinv_stage<K, 2, 2>(v, B, fwd, 0, q);
  jinv_stage<K, 1, 3>(v, B, fwd, 0, q);
}

// Inverse transforms without the n^-1 factor, canonical.
template <int K>
__device__ __forceinline__ void jntt_inv(uint32_t (&v)[K][16], const uint32_t (&sc)[K], TwiddleRef fwd, uint32_t q,
                                         int x, int bar) {
  int B[16];
  jntt_inv_to1<K>(v, B, sc, fwd, q, x, bar);
  jinv_stage<K, 0, 4>(v, B, fwd, 0, q);
  jinv_reduce<K, 1>(v, B, q);
}

// The same times c, canonical: stage 0 multiplies its sums by c and its
// differences by c psi^-brv(1) (Shoup pairs c, cw), whose products need no
// other reduction.
template <int K>
__device__ __forceinline__ void jntt_inv_scaled(uint32_t (&v)[K][16], const uint32_t (&sc)[K], TwiddleRef fwd, uint2 c,
                                                uint2 cw, uint32_t q, int x, int bar) {
  int B[16];
  jntt_inv_to1<K>(v, B, sc, fwd, q, x, bar);
#pragma unroll
  for (int r = 0; r < 8; r++) {
#pragma unroll
    for (int e = 0; e < 2; e++)
      if (B[r + 8 * e] > JB_MAX) {
#pragma unroll
        for (int k = 0; k < K; k++) v[k][r + 8 * e] = csub(v[k][r + 8 * e], 8 * q);
      }
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t a = v[k][r], b = v[k][r + 8];  // below 8 q
      v[k][r] = reduce_2q(mul_shoup_lazy(a + b, c, q), q);
      v[k][r + 8] = reduce_2q(mul_shoup_lazy(a - b + 8 * q, cw, q), q);
    }
  }
}

}  // namespace ig
