// respond_common.cuh -- device helpers shared by the Respond kernels
// (respond.cu: one CTA per query; respond_pair.cu: a cluster of two CTAs
// per query, one per CRT residue) and by the kernels that build their tables:
// bulk copies and mbarriers, the layouts of slots, the folded keys.
#pragma once
#include "common.cuh"

namespace ig {

// A 64-bit load the compiler may neither hoist nor keep in a register: used
// to re-read a query's database base pointer where it is needed instead of
// holding it through the kernel.
template <class T>
__device__ __forceinline__ T* reload_ptr(T* const* p) {
  uint64_t v;
  asm volatile("ld.global.nc.u64 %0, [%1];" : "=l"(v) : "l"(p));
  return reinterpret_cast<T*>(v);
}

// L2 prefetch of a contiguous device range with bulk (TMA) prefetches.
__device__ __forceinline__ void prefetch_l2(const void* p, size_t bytes) {
  const char* c = static_cast<const char*>(p);
  for (size_t off = 0; off < bytes; off += 65536) {
    const uint32_t sz = (uint32_t)(bytes - off < 65536 ? bytes - off : 65536);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(c + off), "r"(sz) : "memory");
  }
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// mbarrier with one arrival, visible to the bulk-copy (async) proxy.
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// The single arrival, announcing `bytes` of bulk copies to complete.
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// Bulk copy of `bytes` (a multiple of 16; both addresses 16-byte aligned)
// from global memory -- device or mapped host memory -- into this CTA's shared
// memory, completing on `bar`.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Wait, with an iteration bound, for phase `parity` of `bar` to complete;
// false when the bound ran out (at once for limit 0).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit) {
  for (uint32_t it = 0; it < limit; it++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// ---- slot order of the resident tables ----
// tau_{g^i} in the NTT domain is the slot permutation s -> u with 2brv(u)+1 =
// g^i (2brv(s)+1) mod 2N (inspiring2.rs:208-263).  With g = 2N/gamma + 1 and
// gamma <= 16 a power of two, g^i = 1 + (2N/gamma) i mod 2N, so brv(u) =
// brv(s) + (N/gamma) (i (2brv(s)+1) mod gamma) mod N: only the top four bits
// of brv(s) move, i.e. only the low four bits of s, by an amount that depends
// on s >> 4 alone.  With s = 16 x + l and h = brv4(l), the top four bits of
// brv(s), u is (x, h + rot_rows(gamma, i, x) mod 16).
//
// Tables are therefore stored by run:
//   quads  [l >> 2][x][l & 3]: a thread reads the slots it owns with coalesced
//          128-bit loads (contracted shard, CRS keys);
//   rows   [h][x]: row h + rot of 128 runs, the rotation uniform over 16 runs,
//          so that a warp's load of a rotated slot touches two half lines
//          (client keys, row transforms).
__device__ __forceinline__ uint32_t rot_rows(int gamma, int i, int x) {
  const uint32_t c = 2u * (__brev((uint32_t)x) >> 25) + 1u;  // 2 brv(s) + 1 mod 16
  return (((uint32_t)i * c) & (uint32_t)(gamma - 1)) * (uint32_t)(MAX_GAMMA / gamma);
}
__host__ __device__ constexpr int h_of(int l) { return ((l & 1) << 3) | ((l & 2) << 1) | ((l & 4) >> 1) | ((l & 8) >> 3); }
__host__ __device__ constexpr int quad_word(int l, int x) { return (l >> 2) * 512 + 4 * x + (l & 3); }
__host__ __device__ constexpr int row_word(int h, int x) { return h * 128 + x; }

// Programmatic dependent launch: a launch that allows it may be set up while the
// one before it runs; it waits for that one's end (no wait otherwise) where it
// first needs its results.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A key triple's transforms (any representatives below 6.5 q in absolute value,
// signed), scaled by n^-1 2^32 and with the third gadget digit folded in
// (fold_third_digit_kernel, setup.cu), canonical.
__device__ __forceinline__ void fold_keys(uint32_t (&v)[ELL][16], const ResidueConsts& C) {
  const uint32_t q = C.q;
#pragma unroll
  for (int j = 0; j < 16; j++) {
    uint32_t k[ELL];
#pragma unroll
    for (int e = 0; e < ELL; e++) k[e] = mul_shoup(v[e][j] + 8 * q, C.ninv_mont, C.ninv_mont_p, q);
    v[0][j] = sub_mod(k[0], mul_shoup(k[2], C.d2_z2, C.d2_z2_p, q), q);
    v[1][j] = sub_mod(k[1], mul_shoup(k[2], C.d2_z1, C.d2_z1_p, q), q);
    v[2][j] = mul_shoup(k[2], C.d2_nz2, C.d2_nz2_p, q);
  }
}

__host__ __device__ constexpr int brv_of(int v, int bits) {
  int r = 0;
  for (int i = 0; i < bits; i++) r |= ((v >> i) & 1) << (bits - 1 - i);
  return r;
}

// The DFT of a slot's G values, G_m = sum_i zeta^(i m) f_i with zeta = psi^(2N/G),
// by decimation in frequency: f[k] = G_m, m the bit reversal of k.  Values in
// [0, 2q) both ways.
template <int G>
__device__ __forceinline__ void slot_dft(uint32_t (&f)[G], const ResidueConsts& C) {
  const uint32_t q = C.q, q2 = 2 * q;
#pragma unroll
  for (int len = G; len > 1; len >>= 1)
#pragma unroll
    for (int b = 0; b < G; b += len)
#pragma unroll
      for (int p = 0; p < len / 2; p++) {
        const uint32_t u = f[b + p], v = f[b + p + len / 2];
        f[b + p] = csub(u + v, q2);
        const uint32_t d = u - v + q2;
        f[b + p + len / 2] = p == 0 ? csub(d, q2) : mul_shoup_lazy(d, __ldg(C.fwd + brv_of(2 * N / len * p, LOGN)), q);
      }
}

__device__ __forceinline__ uint32_t u4e(const uint4& v, int e) { return e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w; }

}  // namespace ig
