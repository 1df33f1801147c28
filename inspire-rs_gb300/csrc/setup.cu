// setup.cu -- setup-time GPU kernels: resident database, CRS key table and
// per-client key tables.  All outputs stay in HBM for the lifetime of their
// handles; Respond then reads them without further preprocessing.
#include <algorithm>

#include "kernels.h"
#include "ntt_joint.cuh"
#include "respond_common.cuh"

namespace ig {

namespace {

// encode_database (src/pir/encode_db.rs:106-181): shard s holds entries
// [s*N, s*N + N); column c, coefficient i = little-endian u16 of bytes
// (2c, 2c+1) of that entry (a lone trailing byte is the value itself).
__global__ void columns_from_raw_kernel(const uint8_t* __restrict__ raw, uint64_t n_entries,
                                        int entry_size, int gamma, int nshards,
                                        uint16_t* __restrict__ H) {
  const uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t total = (uint64_t)nshards * N;
  if (idx >= total) return;
  const uint64_t s = idx >> LOGN, i = idx & (N - 1);
  const uint64_t e = idx;  // global entry index = s * N + i
  for (int c = 0; c < gamma; c++) {
    uint16_t v = 0;
    if (e < n_entries) {
      const uint8_t* ent = raw + e * (uint64_t)entry_size;
      const int bo = 2 * c;
      if (bo + 1 < entry_size) v = (uint16_t)(ent[bo] | (ent[bo + 1] << 8));
      else if (bo < entry_size) v = ent[bo];
    }
    H[(s * gamma + c) * N + i] = v;
  }
}

// Contracted database: K * sum_j zeta^(k j) * omega_u^j * NTT(d_t(Delta h_j))[u]
// with omega_u = psi^(2brv(u)+1), zeta = psi^(2n/gamma), K = gamma^-1 n^-1
// 2^32 (Montgomery form, n^-1 pre-applied for the unscaled inverse NTTs of
// the Respond kernel).  Grid: (shard, residue, digit t).
//
// Stored by recursion step i and, within it, by the slot s that R_i takes
// the value at: source slot u contributes the DFT output k = (2brv(u)+1) m_i
// mod gamma, m_i = (gamma - i) mod gamma, to s = tau_i^-1(u), i.e. (rot_rows)
// to row h - rot of the same 16-slot run.  For odd 2brv(u)+1 the map i -> k
// is a bijection: the table is a permutation of the outputs.  A slot's G values
// stay its thread's until they are written, a quad at a time.
// 2^20 entries (512 shards) come from host memory into this form in 1.0 ms, 1.7
// with G products per output and 4-byte stores.
constexpr int ENC_GROUPS = 4;
template <int G>
__global__ void __launch_bounds__(ENC_GROUPS* NTT_GT, 1)
    encode_E_kernel(const DevParams P, const uint16_t* __restrict__ H, uint32_t* __restrict__ E) {
  constexpr int LG = G == 16 ? 4 : G == 8 ? 3 : G == 4 ? 2 : G == 2 ? 1 : 0;
  extern __shared__ __align__(128) uint32_t smem[];
  uint32_t* Dh = smem;  // [G][16 rows h][128]; then the exchange buffers
  const int s = blockIdx.x, r = blockIdx.y, t = blockIdx.z;
  const int tid = threadIdx.x, g = tid >> 7, x = tid & 127;
  const ResidueConsts& C = P.r[r];
  const uint32_t q = C.q;
#pragma unroll 1
  for (int j = g; j < G; j += ENC_GROUPS) {
    const uint16_t* h = H + ((size_t)s * G + j) * N;
    uint32_t v[1][16];
#pragma unroll
    for (int rr = 0; rr < 16; rr++) {
      const uint64_t xv = P.delta * (uint64_t)h[x + 128 * rr];
      v[0][rr] = (uint32_t)(xv >> (ZBITS * t)) & ((1u << ZBITS) - 1);  // digit t < 2^20 < q
    }
    group_sync(1 + g);  // the last transform's reads are done
    const uint32_t sc[1] = {jx_addr(Dh + (G + g) * N)};
    jntt_fwd<1, JB_CANON>(v, sc, sfwd_tw(C), q, x, 1 + g);
#pragma unroll
    for (int rr = 0; rr < 16; rr++) Dh[j * N + row_word(h_of(rr), x)] = jcanon_fwd(v[0][rr], q);
  }
  __syncthreads();
  const uint32_t c = 2u * (__brev((uint32_t)x) >> 25) + 1u;  // 2brv(u)+1 = 256 h + c
  const uint32_t cinv = c * c * c;                           // c^4 = 1 mod 16
#pragma unroll 1
  for (int h = g; h < 16; h += ENC_GROUPS) {
    uint32_t* slot = Dh + row_word(h, x);
    uint32_t f[G];
#pragma unroll
    for (int j = 0; j < G; j++) {
      const uint32_t ex = ((256u * (uint32_t)h + c) * (uint32_t)j) & (2 * N - 1);  // omega_u^j = psi^ex, psi^N = -1
      f[j] = slot[j * N];
      if (j) f[j] = mul_shoup_lazy(f[j], __ldg(C.fwd + brv11(ex & (N - 1))), q);
      if (ex & N) f[j] = 2 * q - f[j];
      if (j) f[j] = csub(f[j], 2 * q);
    }
    slot_dft<G>(f, C);
#pragma unroll
    for (int k = 0; k < G; k++) {
      const uint32_t i = (0u - cinv * (uint32_t)brv_of(k, LG)) & (uint32_t)(G - 1);
      slot[i * N] = mul_shoup(f[k], C.e_scale, C.e_scale_p, q);
    }
  }
  __syncthreads();
  uint32_t* Eo = E + (((size_t)s * 2 + r) * G * ELL + t) * N;
#pragma unroll 1
  for (int i = 0; i < G; i++) {
    const uint32_t rot = rot_rows(G, i, x);
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; j++) w[j] = Dh[i * N + row_word(((uint32_t)h_of(4 * g + j) + rot) & 15u, x)];
    *reinterpret_cast<uint4*>(Eo + (size_t)i * ELL * N + 512 * g + 4 * x) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// OfflinePackingKeys::generate (inspiring2.rs:448-506): w_all_ntt[i][k] =
// NTT-domain automorphism tau_{g^i} of NTT(w_mask[k]) for i < gamma-1, with the
// reference's residue-1 behaviour in compat mode.  Stored times n^-1 2^32.
__global__ void __launch_bounds__(BLOCK) crs_what_kernel(const DevParams P, const uint32_t* __restrict__ wmask,
                                                         uint32_t* __restrict__ what) {
  __shared__ __align__(16) uint32_t W[2][N];
  __shared__ uint32_t SC[2][NTT_SCRATCH];
  const int k = blockIdx.x, tid = threadIdx.x, g = tid >> 7, x = tid & 127;
  const int gamma = P.gamma;
  {
    const ResidueConsts& C = P.r[g];
    uint32_t v[16];
#pragma unroll
    for (int rr = 0; rr < 16; rr++) v[rr] = wmask[((size_t)k * 2 + g) * N + x + 128 * rr];
    ntt_fwd(v, SC[g], fwd_tw(C), C.q, x, 1 + g);
#pragma unroll
    for (int rr = 0; rr < 16; rr++) W[g][16 * x + rr] = canon16(v[rr], C.q);
  }
  __syncthreads();
  for (int i = 0; i + 1 < gamma; i++) {
    const uint32_t tg = gen_pow(gamma, i);
    for (int v = 0; v < N / BLOCK; v++) {
      const int s = tid + BLOCK * v;
      const uint32_t es = 2 * brv11(s) + 1;
      const int u = brv11(((tg * es) & (2 * N - 1)) >> 1);  // table_{g^i}[s]
      uint32_t v0 = W[0][u];
      uint32_t v1 = P.mode == MODE_COMPAT ? compat_residue1(P, v0) : W[1][u];
      v0 = mul_shoup(v0, P.r[0].ninv_mont, P.r[0].ninv_mont_p, P.r[0].q);
      v1 = mul_shoup(v1, P.r[1].ninv_mont, P.r[1].ninv_mont_p, P.r[1].q);
      what[(((size_t)i * ELL + k) * 2 + 0) * N + s] = v0;
      what[(((size_t)i * ELL + k) * 2 + 1) * N + s] = v1;
    }
  }
}

// Key tables with the third gadget digit folded in.  In the NTT domain of
// residue r, the digits of the composite coefficient c = INTT(R) satisfy
// NTT(d0) + z NTT(d1) + z^2 NTT(d2) = R (mod q_r), so for any key triple
// (k0, k1, k2):  k0 NTT(d0) + k1 NTT(d1) + k2 NTT(d2)
//   = (k0 - z^-2 k2) NTT(d0) + (k1 - z^-1 k2) NTT(d1) + (z^-2 k2) R.
// With R kept as n^-1 R (the Respond kernel's R_{i+1}), the third key is
// n z^-2 k2.  src and dst hold ngroups triples [g][k<3][2][N] (any constant
// scaling, applied alike to the three keys), src in slot order, dst in quads
// [l >> 2][x][l & 3].
__global__ void __launch_bounds__(BLOCK) fold_third_digit_kernel(const DevParams P, const uint32_t* src, uint32_t* dst,
                                                                 int ngroups) {
  const size_t per = (size_t)2 * N;
  const size_t total = (size_t)ngroups * per;
  for (size_t idx = (size_t)blockIdx.x * BLOCK + threadIdx.x; idx < total; idx += (size_t)gridDim.x * BLOCK) {
    const size_t g = idx / per, rs = idx - g * per;
    const int r = (int)(rs >> LOGN);
    const ResidueConsts& C = P.r[r];
    const int w = (int)(rs & (N - 1));
    const int x = (w >> 2) & 127, l = ((w >> 9) << 2) | (w & 3);
    const uint32_t* f = src + g * 3 * per + (size_t)r * N + 16 * x + l;
    uint32_t* t = dst + g * 3 * per + rs;
    const uint32_t k0 = f[0], k1 = f[per], k2 = f[2 * per];
    t[0] = sub_mod(k0, mul_shoup(k2, C.d2_z2, C.d2_z2_p, C.q), C.q);
    t[per] = sub_mod(k1, mul_shoup(k2, C.d2_z1, C.d2_z1_p, C.q), C.q);
    t[2 * per] = mul_shoup(k2, C.d2_nz2, C.d2_nz2_p, C.q);
  }
}

// Client key table from y_body: the forward NTT of packing_online
// (inspiring2.rs:1199-1213) of the three y_body[k], times n^-1 2^32, the third
// digit folded in as above, in rows [h][x].  generate_rotations (:1309-1323) is a
// rotation of the rows (rot_rows), which the Respond kernels apply as they read.
// An explicit y_all ((gamma-1) triples of coefficient polys; `rotated`) is
// stored with slot h in row h + rot, where they look for it.  One CTA per triple
// and residue, keys in device or page-locked host memory.  A single query's
// Respond kernel, which needs the table only after the rows' expansion, starts
// meanwhile.  Measured (one query with its keys, host call): 131 us with seeds and
// 125 without; 146 and 155 with an upload, a transform of single polys, a fold in
// place and copies of the rows.
__global__ void __launch_bounds__(NTT_GT) client_keys_kernel(const DevParams P, const uint64_t* __restrict__ keys,
                                                             bool rotated, uint32_t* __restrict__ yhat) {
  __shared__ __align__(128) uint32_t X[ELL][N];
  pdl_trigger();
  const int g = blockIdx.x, r = blockIdx.y, x = threadIdx.x;
  const ResidueConsts& C = P.r[r];
  const uint64_t* src = keys + ((size_t)g * ELL * 2 + r) * N + x;
  uint32_t v[ELL][16];
#pragma unroll
  for (int k = 0; k < ELL; k++)
#pragma unroll
    for (int j = 0; j < 16; j++) v[k][j] = (uint32_t)__ldg(src + (size_t)k * 2 * N + 128 * j);
  const uint32_t sc[ELL] = {jx_addr(X[0]), jx_addr(X[1]), jx_addr(X[2])};
  jntt_fwd<ELL, JB_CANON>(v, sc, sfwd_tw(C), C.q, x, 1);
  fold_keys(v, C);
  const uint32_t rot = rotated ? rot_rows(P.gamma, g, x) : 0;
  uint32_t* o = yhat + ((size_t)g * ELL * 2 + r) * N;
#pragma unroll
  for (int k = 0; k < ELL; k++)
#pragma unroll
    for (int j = 0; j < 16; j++) o[(size_t)k * 2 * N + row_word((h_of(j) + rot) & 15, x)] = v[k][j];
}

}  // namespace

cudaError_t launch_fold_third_digit(const DevParams& P, const uint32_t* src, uint32_t* dst, int ngroups,
                                    cudaStream_t st) {
  if (ngroups <= 0) return cudaSuccess;
  const size_t total = (size_t)ngroups * 2 * N;
  const unsigned blocks = (unsigned)std::min<size_t>((total + BLOCK - 1) / BLOCK, 4096);
  fold_third_digit_kernel<<<blocks, BLOCK, 0, st>>>(P, src, dst, ngroups);
  return cudaGetLastError();
}

cudaError_t launch_columns_from_raw(const uint8_t* raw, uint64_t n_entries, int entry_size, int gamma,
                                    int nshards, uint16_t* H, cudaStream_t st) {
  const uint64_t total = (uint64_t)nshards * N;
  const unsigned blocks = (unsigned)((total + 255) / 256);
  if (blocks) columns_from_raw_kernel<<<blocks, 256, 0, st>>>(raw, n_entries, entry_size, gamma, nshards, H);
  return cudaGetLastError();
}

template <int G>
static constexpr int encode_smem_bytes() {
  return (int)sizeof(uint32_t) * (G + ENC_GROUPS) * N;
}
template <int G>
static cudaError_t set_encode_smem() {
  return cudaFuncSetAttribute(encode_E_kernel<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, encode_smem_bytes<G>());
}
cudaError_t prepare_setup_kernels() {
  const cudaError_t es[] = {set_encode_smem<1>(), set_encode_smem<2>(), set_encode_smem<4>(), set_encode_smem<8>(),
                            set_encode_smem<16>()};
  for (cudaError_t e : es)
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}

template <int G>
static void launch_encode(const DevParams& P, const uint16_t* H, int nshards, uint32_t* E, cudaStream_t st) {
  // grid.x is limited to 2^31-1 shards; y = residue, z = digit
  encode_E_kernel<G><<<dim3(nshards, 2, ELL), ENC_GROUPS * NTT_GT, encode_smem_bytes<G>(), st>>>(P, H, E);
}

cudaError_t launch_encode_E(const DevParams& P, const uint16_t* H, int nshards, uint32_t* E, cudaStream_t st) {
  if (nshards <= 0) return cudaSuccess;
  switch (P.gamma) {
    case 1: launch_encode<1>(P, H, nshards, E, st); break;
    case 2: launch_encode<2>(P, H, nshards, E, st); break;
    case 4: launch_encode<4>(P, H, nshards, E, st); break;
    case 8: launch_encode<8>(P, H, nshards, E, st); break;
    case 16: launch_encode<16>(P, H, nshards, E, st); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_crs_what(const DevParams& P, const uint32_t* wmask, uint32_t* what, cudaStream_t st) {
  if (P.gamma < 2) return cudaSuccess;
  crs_what_kernel<<<ELL, BLOCK, 0, st>>>(P, wmask, what);
  return cudaGetLastError();
}

cudaError_t launch_client_keys(const DevParams& P, const uint64_t* keys, int ntriples, bool rotated, uint32_t* yhat,
                               cudaStream_t st) {
  if (ntriples <= 0) return cudaSuccess;
  client_keys_kernel<<<dim3(ntriples, 2), NTT_GT, 0, st>>>(P, keys, rotated, yhat);
  return cudaGetLastError();
}

}  // namespace ig
