// ntt_team.cuh -- the transforms of ntt_joint.cuh for one polynomial on a team
// of 256 threads, 8 values per thread: half the instructions per thread of the
// 128-thread form, for kernels whose time is the latency of one chain of
// transforms (a lone warp issues one instruction in about seven cycles there,
// whatever the pipes could take).
//
// Signed arithmetic, bounds and the shared table as in ntt_joint.cuh.  Layouts
// of thread t: coefficients v[r] = a[t + 256 r], slots v[r] = A[8 t + r].
// Registers hold three index bits at a time; warp w owns elements [256 w, 256 w
// + 256) from the first exchange of the forward transform on (to the last of
// the inverse), so only that exchange needs the team's barrier:
//   forward: bits 8-10 (stages 0-2) | team | 5-7 (3-5) | warp | 2-4 (6-8) |
//            warp | 0-1 (9, 10)
//   inverse: bits 0-2 (stages 10-8) | warp | 3-5 (7-5) | warp | 6-7 (4, 3) |
//            team | 8-10 (2-0)
// The exchange buffer (2048 words) keeps element e at e ^ ((e >> 5 & 7) << 2),
// which is free of bank conflicts in all these layouts (8 t + r in 128-bit
// chunks) and keeps blocks of 32 together, so exchanges work in place with
// one barrier each.
#pragma once
#include "ntt_joint.cuh"

namespace ig {

constexpr int TEAM = 256;

// Byte offsets of thread t's element 0; element r is an XOR (bits 4-6) and a
// multiple of 128 bytes away.
__device__ __forceinline__ uint32_t jt_co(int t) {  // t + 256 r, and t of any block of 256
  return 4u * (uint32_t)(t ^ (((t >> 5) & 7) << 2));
}
__device__ __forceinline__ uint32_t jt_hi(int t) {  // (t & 31) + 32 r + 256 (t >> 5)
  return 4u * (uint32_t)((t & 31) + 256 * (t >> 5));
}
__device__ __forceinline__ uint32_t jt_mf(int t) {  // (t & 3) + 4 r + 32 (t >> 2)
  return 4u * (uint32_t)((t & 3) + 32 * (t >> 2)) ^ (16u * (uint32_t)((t >> 2) & 7));
}
__device__ __forceinline__ uint32_t jt_mi(int t) {  // (t & 7) + 8 r + 64 (t >> 3)
  return 4u * (uint32_t)((t & 7) + 64 * (t >> 3)) ^ (32u * (uint32_t)((t >> 3) & 3));
}
__device__ __forceinline__ uint32_t jt_ru(int t) {  // 8 t + r
  return 4u * (uint32_t)((8 * t) ^ (((t >> 2) & 7) << 2));
}

#define IG_JT_ACCESS(name, base, expr)                                                             \
  __device__ __forceinline__ void jt_store_##name(const uint32_t (&v)[8], uint32_t sc, int t) {    \
    const uint32_t a = sc + base(t);                                                               \
    _Pragma("unroll") for (int r = 0; r < 8; r++) jx_at(expr) = v[r];                              \
  }                                                                                                \
  __device__ __forceinline__ void jt_load_##name(uint32_t (&v)[8], uint32_t sc, int t) {           \
    const uint32_t a = sc + base(t);                                                               \
    _Pragma("unroll") for (int r = 0; r < 8; r++) v[r] = jx_at(expr);                              \
  }
IG_JT_ACCESS(co, jt_co, a + 1024u * r)                           // bits 8-10 do not move the swizzle
IG_JT_ACCESS(hi, jt_hi, (a ^ (16u * r)) + 128u * r)              // r is bits 5-7
IG_JT_ACCESS(mf, jt_mf, a ^ (16u * r))                           // r is bits 2-4
IG_JT_ACCESS(mi, jt_mi, (a ^ (32u * (r & 3)) ^ (16u * (r >> 2))) + 128u * (r >> 2))  // bits 3-5
#undef IG_JT_ACCESS
__device__ __forceinline__ void jt_store_ru(const uint32_t (&v)[8], uint32_t sc, int t) {
  const uint32_t a = sc + jt_ru(t);
  jx_at4(a) = make_uint4(v[0], v[1], v[2], v[3]);
  jx_at4(a ^ 16u) = make_uint4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ void jt_load_ru(uint32_t (&v)[8], uint32_t sc, int t) {
  const uint32_t a = sc + jt_ru(t);
  const uint4 lo = jx_at4(a), hi = jx_at4(a ^ 16u);
  v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
  v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
}

// Twiddle runs of up to three stages, loaded ahead of the exchange before them.
struct JtRuns {
  uint2 a[1], b[2], c[4];
};

// Stages on register bits 2, 1, 0 (forward) with twiddle indices (1 << s) +
// first, (2 << s) + 2 first, (4 << s) + 4 first.
__device__ __forceinline__ void jt_runs(JtRuns& w, TwiddleRef tw, int s, int first) {
  tw_run<1>(tw, (1 << s) + first, w.a);
  tw_run<2>(tw, (2 << s) + 2 * first, w.b);
  tw_run<4>(tw, (4 << s) + 4 * first, w.c);
}

template <int H, int SH, int CNT>
__device__ __forceinline__ void jt_fwd_stage(uint32_t (&v)[8], int (&B)[8], const uint2 (&run)[CNT], uint32_t q) {
#pragma unroll
  for (int r = 0; r < 8; r++)
    if ((r & H) == 0) {
      if (jb_fwd(B[r], B[r + H])) v[r] = centre(v[r], 4 * q);
      const uint2 w = run[r >> SH];
      const uint32_t a = v[r], b = v[r + H];
      const uint32_t h = (uint32_t)__mulhi((int)b, (int)w.y);
      const uint32_t s = b * w.x + a;
      v[r] = s - h * q;
      v[r + H] = twice_minus(a, v[r]);
    }
}

// (stages 0-2, 3-5, 6-8, 9 and 10)
__host__ __device__ constexpr int jt_fwd_out(int b0) {
  const JbPhase phases[4] = {{3, 4}, {3, 4}, {3, 4}, {2, 2}};
  int B[8] = {};
  for (int r = 0; r < 8; r++) B[r] = b0;
  return jfwd_bound(B, phases);
}
static_assert(jt_fwd_out(JB_CANON) <= JFWD_OUT && jt_fwd_out(JB_DIGIT) <= JFWD_OUT_DIGIT, "forward outputs");

// Forward transform; inputs in [0, B0 q / 64), outputs as jntt_fwd's (signed,
// below JFWD_OUT q / 64).  `hook` runs before the last
// two stages.
template <int B0, class Hook = NoHook>
__device__ __forceinline__ void jt_fwd(uint32_t (&v)[8], uint32_t sc, TwiddleRef tw, uint32_t q, int t, int bar,
                                       Hook&& hook = Hook()) {
  int B[8];
#pragma unroll
  for (int r = 0; r < 8; r++) B[r] = B0;
  JtRuns w;
  jt_runs(w, tw, 0, 0);
  jt_fwd_stage<4, 3, 1>(v, B, w.a, q);
  jt_fwd_stage<2, 2, 2>(v, B, w.b, q);
  jt_fwd_stage<1, 1, 4>(v, B, w.c, q);
  jt_store_co(v, sc, t);
  jt_runs(w, tw, 3, t >> 5);
  team_sync(bar);
  jt_load_hi(v, sc, t);
  jb_level(B);
  jt_fwd_stage<4, 3, 1>(v, B, w.a, q);
  jt_fwd_stage<2, 2, 2>(v, B, w.b, q);
  jt_fwd_stage<1, 1, 4>(v, B, w.c, q);
  jt_store_hi(v, sc, t);
  jt_runs(w, tw, 6, t >> 2);
  __syncwarp();
  jt_load_mf(v, sc, t);
  jb_level(B);
  jt_fwd_stage<4, 3, 1>(v, B, w.a, q);
  jt_fwd_stage<2, 2, 2>(v, B, w.b, q);
  jt_fwd_stage<1, 1, 4>(v, B, w.c, q);
  jt_store_mf(v, sc, t);
  tw_run<2>(tw, 512 + 2 * t, w.b);
  tw_run<4>(tw, 1024 + 4 * t, w.c);
  __syncwarp();
  jt_load_ru(v, sc, t);
  hook();
  jb_level(B);
  jt_fwd_stage<2, 2, 2>(v, B, w.b, q);
  jt_fwd_stage<1, 1, 4>(v, B, w.c, q);
}

// Inverse stage on register bit H, twiddles as -fwd in reverse (ntt_joint.cuh).
template <int H, int SH, int CNT>
__device__ __forceinline__ void jt_inv_stage(uint32_t (&v)[8], int (&B)[8], const uint2 (&run)[CNT], uint32_t q) {
#pragma unroll
  for (int r = 0; r < 8; r++)
    if ((r & H) == 0) {
#pragma unroll
      for (int e = 0; e < 2; e++)
        if (B[r + e * H] > JB_MAX) {
          v[r + e * H] = csub(v[r + e * H], 8 * q);
          B[r + e * H] = JB_MAX;
        }
      const uint2 w = run[CNT - 1 - (r >> SH)];
      const uint32_t a = v[r], d = v[r + H] - a;
      v[r] = a + v[r + H];
      const uint32_t h = (uint32_t)__mulhi((int)d, (int)w.y);
      const uint32_t s = d * w.x + q;
      v[r + H] = s - h * q;
      const int m = B[r] > B[r + H] ? B[r] : B[r + H];
      B[r] += B[r + H];
      B[r + H] = 128 + (m + 31) / 32;
    }
}
template <int C>
__device__ __forceinline__ void jt_inv_reduce(uint32_t (&v)[8], int (&B)[8], uint32_t q) {
#pragma unroll
  for (int r = 0; r < 8; r++) {
#pragma unroll
    for (int c = 8; c >= C; c >>= 1) {
      if (B[r] > 64 * c) {
        v[r] = csub(v[r], (uint32_t)c * q);
        B[r] = 64 * c;
      }
    }
    if (C == 4) B[r] = 256;
  }
}
// Runs of stages s + 2, s + 1, s with first twiddle offsets 4, 2, 1 times
// `first`, from the forward table: indices (2 << S) - CNT - offset.
__device__ __forceinline__ void jt_inv_runs(JtRuns& w, TwiddleRef fwd, int s, int first) {
  tw_run<4>(fwd, (8 << s) - 4 - 4 * first, w.c);
  tw_run<2>(fwd, (4 << s) - 2 - 2 * first, w.b);
  tw_run<1>(fwd, (2 << s) - 1 - first, w.a);
}

// Inverse transform without the n^-1 factor, slots in [0, 4 q) in, canonical
// coefficients out.
__device__ __forceinline__ void jt_inv(uint32_t (&v)[8], uint32_t sc, TwiddleRef fwd, uint32_t q, int t, int bar) {
  int B[8];
#pragma unroll
  for (int r = 0; r < 8; r++) B[r] = 256;
  JtRuns w;
  jt_inv_runs(w, fwd, 8, t);
  jt_inv_stage<1, 1, 4>(v, B, w.c, q);
  jt_inv_stage<2, 2, 2>(v, B, w.b, q);
  jt_inv_stage<4, 3, 1>(v, B, w.a, q);
  jt_inv_reduce<4>(v, B, q);
  jt_store_ru(v, sc, t);
  jt_inv_runs(w, fwd, 5, t >> 3);
  __syncwarp();
  jt_load_mi(v, sc, t);
  jt_inv_stage<1, 1, 4>(v, B, w.c, q);
  jt_inv_stage<2, 2, 2>(v, B, w.b, q);
  jt_inv_stage<4, 3, 1>(v, B, w.a, q);
  jt_inv_reduce<4>(v, B, q);
  jt_store_mi(v, sc, t);
  // stages 4, 3 on bits 6, 7 (register bits 1, 2): twiddles 16 + 2 (t >> 5) + (r >> 2), 8 + (t >> 5)
  tw_run<2>(fwd, 32 - 2 - 2 * (t >> 5), w.b);
  tw_run<1>(fwd, 16 - 1 - (t >> 5), w.a);
  __syncwarp();
  jt_load_hi(v, sc, t);
  jt_inv_stage<2, 2, 2>(v, B, w.b, q);
  jt_inv_stage<4, 3, 1>(v, B, w.a, q);
  jt_inv_reduce<4>(v, B, q);
  jt_store_hi(v, sc, t);
  jt_inv_runs(w, fwd, 0, 0);
  team_sync(bar);
  jt_load_co(v, sc, t);
  jt_inv_stage<1, 1, 4>(v, B, w.c, q);
  jt_inv_stage<2, 2, 2>(v, B, w.b, q);
  jt_inv_stage<4, 3, 1>(v, B, w.a, q);
  jt_inv_reduce<1>(v, B, q);
}

}  // namespace ig
