// tree.cu -- tree packing (respond_one_packing / respond_seeded_packed,
// src/pir/respond.rs:213-268, 428-435) on the GPU: pack_lwes
// (src/inspiring/automorph_pack.rs:418-485) over the LWEs sample-extracted at
// coefficient 0 of a query's column products (rlwe/enc.rs:195-208), with the
// CRS's log2(d) Galois key-switching matrices (pir/setup.rs:164-173).
//
// pack_lwes_inner (automorph_pack.rs:171-255) at d = 2048 has 11 levels;
// node (l, s) combines its children (l-1, s) and (l-1, s + 2^(11-l)):
//   s0 = even + X^(d >> l) odd,  s1 = even - X^(d >> l) odd,
//   node = s0 + homomorphic_automorph(s1, 2^l + 1, key[11 - l])
// and a child whose start is past the last LWE is absent (then s0 = s1 =
// even; all-zero subtrees contribute nothing, bit for bit).  With at most 16
// LWEs, levels 1..7 are a chain per LWE and levels 8..11 combine pairs.
//
// homomorphic_automorph (automorph_pack.rs:33-79): tau_t of both parts,
// gadget digits (base 2^20, 3 digits) of tau_t(a), and
//   out = (sum_k digit_k * K[k].a, tau_t(b) + sum_k digit_k * K[k].b).
//
// Both parts of every ciphertext stay in the NTT domain (alpha, beta: NTT
// values times n^-1), where
//  * X^k is a product per slot and tau_t a permutation of slots;
//  * the third digit needs no transform: NTT(d0) + z NTT(d1) + z^2 NTT(d2) =
//    NTT(tau_t a) mod q_r, the permuted alpha, so with the keys folded as for
//    the Respond kernel (K0 - z^-2 K2, K1 - z^-1 K2, n z^-2 K2) a key switch is
//    one inverse transform (of alpha, for the digits) and two forward ones
//    per residue, instead of three and two inverses;
//  * the LWEs' a parts come from the contracted database without digit
//    transforms: with T_i[u] = sum_t E[i,t][u] A_t[u], the Respond kernel's
//    query-only sums, alpha_j[u] = omega_u^-j sum_i zeta^(i c j) T_i[u], c =
//    2brv(u)+1, a length-gamma DFT per slot.
// A thread owns slots 16x .. 16x+15 of its residue; tau_t maps run x to one
// other run, rows h to rows h0 + h t (tau_row), so ciphertexts are kept in rows
// [h][x] and permuted through shared memory without bank conflicts.
//
// Three launches: tree_front_kernel (rows expanded and transformed, the b side;
// four CTAs per query), tree_leaves_kernel (the DFTs, 16 CTAs per query) and
// tree_kernel (all levels).  Ciphertexts that one CTA leaves to another live in a
// per-query global work area (30 of 2 polys x 2 residues).
//
// What bounds it: the integer multiply-add pipe.  A key switch of both residues
// takes 7.4 k cycles of it per SM (6 transforms of 704, the products, the
// digits) and 12.4 k in all, whether one CTA runs on an SM or two.  A batch of 33
// takes 282 us per host call, 224 of them in tree_kernel (4191 key switches in
// 3.5 chains per SM; the fullest SM has 1.4 times the average), 299 us with a
// launch per level from the eighth on.  At 9 queries or fewer (one chain per SM)
// the call takes 125-133 us.
#include "ntt_joint.cuh"
#include "respond_draws.cuh"

namespace ig {
namespace {

constexpr int CT_WORDS = 4 * N;  // one ciphertext: alpha (2 residues), beta (2 residues), rows [h][x]

// Work area of one query: the node (l, s) of levels 7..10 in buffer
// level_base(l) + s: 0..15 level 7 (each LWE's key-switch chain; the leaves
// before), 16..23 level 8, 24..27 level 9, 28..29 level 10; then the LWEs' b
// values, the arrivals at each node of levels 8..11 (node (l, s) at 2^(11-l) + s)
// and whether each row's expansion ended.  The row transforms lie in the
// level-8 nodes' place until the leaves are made.
constexpr int TREE_BUFS = 30;
__host__ __device__ constexpr int level_base(int l) { return l == 7 ? 0 : l == 8 ? 16 : l == 9 ? 24 : 28; }
constexpr size_t WORK_ROWS = (size_t)level_base(8) * CT_WORDS;  // [ELL][2][N]
constexpr size_t WORK_BVALS = (size_t)TREE_BUFS * CT_WORDS;     // [2 residues][16]
constexpr size_t WORK_ARRIVED = WORK_BVALS + 32;                // [16]
constexpr size_t WORK_GOOD = WORK_ARRIVED + 16;                 // [ELL]
constexpr size_t WORK_WORDS = WORK_GOOD + 16;

// ---- the query's rows: expanded and transformed (rows [h][x] in the work
//      area), one CTA per row, and the b side in a fourth ----
// Only this launch lets its successor start early (the leaves' database words
// then arrive meanwhile): tree_kernel's CTAs, started among the leaves', came to
// lie two on an SM while others stayed empty, 179 us instead of 131 for 9
// queries.
template <bool SEEDED>
__global__ void __launch_bounds__(QT, 2) tree_front_kernel(const __grid_constant__ TreeArgs A) {
  __shared__ __align__(128) uint32_t AH[2 * N];  // the row, coefficients
  __shared__ __align__(128) uint32_t X[2 * N];   // candidates of the expansion, then exchange buffers; partial sums
  __shared__ int ws[32];
  __shared__ uint32_t bp[32];
  __shared__ uint8_t seed[32];
  const DevParams& P = A.P;
  const int qi = blockIdx.x >> 2, t = blockIdx.x & 3, tid = threadIdx.x, r = tid >> 7, x = tid & 127;
  uint32_t* W = A.work + (size_t)qi * WORK_WORDS;
  const uint32_t shard = A.shard[qi];
  pdl_trigger();
  if (shard >= (uint32_t)A.nshards) return;  // uniform over the CTA; tree_kernel reports it
  if (t == ELL) {
    if (tid < 16) W[WORK_ARRIVED + tid] = 0;
    column_b0<ROWS_DIRECT>(P, A.H + (size_t)shard * P.gamma * N, A.brows + (size_t)qi * A.brow_stride, nullptr, nullptr, 0,
                     reinterpret_cast<uint64_t*>(X), bp);
    if (tid < 32) W[WORK_BVALS + tid] = bp[tid];
    return;
  }
  uint32_t v[1][16];
  if (SEEDED) {
    if (tid < 32) seed[tid] = A.seeds[((size_t)qi * ELL + t) * 32 + tid];
    __syncthreads();
    const bool good = expand_row_general<2>(P, seed, reinterpret_cast<uint64_t*>(X), AH, ws);
    __syncthreads();
    if (tid == 0) W[WORK_GOOD + t] = good;
#pragma unroll
    for (int j = 0; j < 16; j++) v[0][j] = AH[r * N + x + 128 * j];
  } else {
    if (tid == 0) W[WORK_GOOD + t] = 1;
    const uint64_t* ar = A.arows + (((size_t)qi * ELL + t) * 2 + r) * N + x;
#pragma unroll
    for (int j = 0; j < 16; j++) v[0][j] = (uint32_t)__ldg(ar + 128 * j);
  }
  const ResidueConsts& C = P.r[r];
  const uint32_t sc[1] = {jx_addr(X + r * N)};
  jntt_fwd<1, JB_CANON>(v, sc, sfwd_tw(C), C.q, x, 1 + r);
  uint32_t* o = W + WORK_ROWS + (t * 2 + r) * N + x;
#pragma unroll
  for (int j = 0; j < 16; j++) o[128 * h_of(j)] = jcanon_fwd(v[0][j], C.q);
}

// ---- leaves: alpha_j of every LWE, from the contracted database ----
constexpr int LEAF_RUNS = 16;  // runs x per CTA: one class x >> 4, so that c and the outputs' columns are uniform

template <int G>
__global__ void __launch_bounds__(256) tree_leaves_kernel(const __grid_constant__ TreeArgs A) {
  constexpr int LG = G == 16 ? 4 : G == 8 ? 3 : G == 4 ? 2 : G == 2 ? 1 : 0;
  __shared__ uint32_t As[ELL][16][LEAF_RUNS];
  __shared__ uint32_t F[G][16][LEAF_RUNS];
  const DevParams& P = A.P;
  const int xc = blockIdx.x & 7, r = (blockIdx.x >> 3) & 1, qi = blockIdx.x >> 4;
  const int tid = threadIdx.x, xl = tid & 15;
  const int x = LEAF_RUNS * xc + xl;
  uint32_t* W = A.work + (size_t)qi * WORK_WORDS;
  const uint32_t shard = A.shard[qi];
  if (shard >= (uint32_t)A.nshards) {  // uniform over the CTA; tree_kernel reports it
    pdl_wait();
    return;
  }
  const ResidueConsts& C = P.r[r];
  const uint32_t q = C.q, q2 = 2 * q;
  // the contracted database first: it does not depend on the launch before
  const uint32_t* E = A.E + ((size_t)shard * 2 + r) * ELL * G * N;
  const int qa = (tid >> 4) & 3, i0 = tid >> 6;  // thread (xl, quad qa, every fourth i)
  constexpr int IT = G < 4 ? 1 : G / 4;
  uint4 e[IT][ELL];
#pragma unroll
  for (int k = 0; k < IT; k++)
#pragma unroll
    for (int t = 0; t < ELL; t++)
      if (i0 + 4 * k < G) e[k][t] = ld_stream(E + ((size_t)(i0 + 4 * k) * ELL + t) * N + 512 * qa + 4 * x);
  pdl_wait();
  for (int k = tid; k < ELL * 256; k += 256)
    As[k >> 8][(k >> 4) & 15][k & 15] = W[WORK_ROWS + ((k >> 8) * 2 + r) * N + row_word((k >> 4) & 15, LEAF_RUNS * xc + (k & 15))];
  __syncthreads();
  // T_i at source slots
#pragma unroll
  for (int k = 0; k < IT; k++) {
    const int i = i0 + 4 * k;
    if (i >= G) break;
    const uint32_t rot = rot_rows(G, i, x);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t h = ((uint32_t)h_of(4 * qa + j) + rot) & 15u;
      F[i][h][xl] = redc((uint64_t)u4e(e[k][0], j) * As[0][h][xl] + (uint64_t)u4e(e[k][1], j) * As[1][h][xl] +
                             (uint64_t)u4e(e[k][2], j) * As[2][h][xl],
                         q, C.qinv);
    }
  }
  __syncthreads();
  // G_m = sum_i zeta^(i m) T_i per slot, then alpha_j = omega_u^-j G_(c j)
  const int h = tid >> 4;
  uint32_t f[G];
#pragma unroll
  for (int i = 0; i < G; i++) f[i] = F[i][h][xl];
  slot_dft<G>(f, C);
  const uint32_t c = 2u * (__brev((uint32_t)x) >> 25) + 1u;      // 2brv(u)+1 mod 16, odd
  const uint32_t cinv = (c * c * c) & (uint32_t)(G - 1);         // c^4 = 1 mod 16
  const uint32_t eu = 256u * (uint32_t)h + c;                    // 2brv(u)+1
#pragma unroll
  for (int k = 0; k < G; k++) {
    const int m = brv_of(k, LG);
    const uint32_t j = (cinv * (uint32_t)m) & (uint32_t)(G - 1);
    const uint32_t ex = (0u - eu * j) & (2 * N - 1);  // omega_u^-j = psi^ex, psi^N = -1
    uint32_t w = f[k];
    if (j) w = mul_shoup_lazy(w, __ldg(C.fwd + brv11(ex & (N - 1))), q);
    if (ex & N) w = q2 - w;
    W[(size_t)j * CT_WORDS + (size_t)r * N + row_word(h, x)] = canon4(w, q);
  }
}

// ---- key switches ----
struct SwitchSmem {
  static constexpr int SP = 0;               // [2 r][2 parts][N] s1 in rows, for tau
  static constexpr int XB = SP + 4 * N;      // [2 r][2][N] exchange buffers; the second first has s1's a, coefficients
  static constexpr int TOTAL = XB + 4 * N;
};

// (ra, rb) += homomorphic_automorph((a, b), 2^l + 1, key[11 - l]), everything
// in this thread's slots; a, b in [0, 4q), ra, rb in [0, 2q).  256 threads, group
// r per residue.
__device__ __forceinline__ void key_switch(const TreeArgs& A, uint32_t base, int l, const uint32_t (&a)[16],
                                           const uint32_t (&b)[16], uint32_t (&ra)[16], uint32_t (&rb)[16]) {
  using L = SwitchSmem;
  const DevParams& P = A.P;
  const int r = threadIdx.x >> 7, x = threadIdx.x & 127;
  const ResidueConsts& C = P.r[r];
  const uint32_t q = C.q, qinv = C.qinv, qo = P.r[r ^ 1].q;
  const uint32_t t = (1u << l) + 1u;
  const uint32_t sp = base + 4 * (L::SP + 2 * N * r), xb = base + 4 * (L::XB + 2 * N * r);
  const uint32_t cf = base + 4 * (L::XB + N);
  group_sync(1 + r);  // the last call's reads of the rows are done
#pragma unroll
  for (int j = 0; j < 16; j++) {
    jx_at(sp + 4 * (uint32_t)row_word(h_of(j), x)) = a[j];
    jx_at(sp + 4 * N + 4 * (uint32_t)row_word(h_of(j), x)) = b[j];
  }
  {
    uint32_t c[1][16];
#pragma unroll
    for (int j = 0; j < 16; j++) c[0][j] = a[j];
    const uint32_t sc[1] = {xb};
    jntt_inv<1>(c, sc, sfwd_tw(C), q, x, 1 + r);
#pragma unroll
    for (int j = 0; j < 16; j++) jx_at(cf + 4 * (2 * N * r + x + 128 * j)) = c[0][j];
  }
  __syncthreads();
  // tau_t: coefficient i goes to i t mod 2N, negated past N, so coefficient j
  // comes from j t^-1; digits 0 and 1 of the composite coefficients
  uint32_t ti = t;  // t^-1 mod 2^32, 2N a power of two (Newton: 3 bits, 6, 12)
  ti *= 2u - t * ti;
  ti *= 2u - t * ti;
  ti *= 2u - t * ti;
  uint32_t v[2][16];
#pragma unroll
  for (int j = 0; j < 16; j++) {
    const uint32_t i = (uint32_t)(x + 128 * j) * ti;
    const uint32_t src = cf + 4 * (i & (N - 1)), neg = 0u - ((i >> LOGN) & 1u);
    uint32_t own = jx_at(src + 8 * N * r), oth = jx_at(src + 8 * N * (r ^ 1));
    own = csub((own ^ neg) - neg + (q & neg), q);  // q - own, 0 for 0
    oth = (oth ^ neg) - neg + (qo & neg);
    const uint64_t cc = crt_compose_from(C, qo, own, oth);
    v[0][j] = (uint32_t)cc & 0xFFFFFu;
    v[1][j] = (uint32_t)(cc >> 20) & 0xFFFFFu;
  }
  __syncthreads();  // the coefficients have been read
  const uint32_t* ks = A.ks + (size_t)(11 - l) * 2 * ELL * 2 * N + (size_t)r * N + 4 * x;
  const uint32_t sc2[2] = {xb, xb + 4 * N};
  jntt_fwd<2, JB_DIGIT>(v, sc2, sfwd_tw(C), q, x, 1 + r);  // signed, below 5.25 q
  // tau_t in the NTT domain: slot s takes slot u, 2brv(u)+1 = t (2brv(s)+1) mod
  // 2N.  With brv(s) = 128 h + y: brv(u) = (128 h + y) t + 2^(l-1) mod N, so run
  // and row offset depend on y alone and row h comes from h0 + h t
  const uint32_t y = __brev((uint32_t)x) >> 25;
  const uint32_t bu = y * t + (1u << (l - 1));
  const uint32_t xu = __brev(bu & 127u) >> 25, h0 = bu >> 7;
#pragma unroll
  for (int qd = 0; qd < 4; qd++) {
    uint4 k[2][ELL];
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int e = 0; e < ELL; e++)
        k[p][e] = ld_stream(ks + (size_t)(p * ELL + e) * 2 * N + 512 * qd);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int s = 4 * qd + j;
      const uint32_t at = sp + 4 * ((((h0 + (uint32_t)h_of(s) * t) & 15u) << 7) + xu);
      const uint32_t ta = jx_at(at), tb = jx_at(at + 4 * N);
      // each sum is in (-10.5 q^2, 14.5 q^2): reduced plus q in (0.3 q, 3 q)
      const uint64_t SA = smul(v[0][s], u4e(k[0][0], j)) + smul(v[1][s], u4e(k[0][1], j)) + smul(ta, u4e(k[0][2], j));
      const uint64_t SB = smul(v[0][s], u4e(k[1][0], j)) + smul(v[1][s], u4e(k[1][1], j)) + smul(ta, u4e(k[1][2], j));
      ra[s] = csub(csub(ra[s] + redc_wide(SA, q, qinv) + q, 4 * q), 2 * q);
      rb[s] = csub(csub(csub(rb[s] + tb + redc_wide(SB, q, qinv) + q, 8 * q), 4 * q), 2 * q);
    }
  }
}

// The tree of every query: one CTA per LWE takes it through levels 1..7 (the
// odd children are absent: node(l, s) = node(l-1, s) +
// homomorphic_automorph(node(l-1, s))), then on to the node it is a child of.
// Of a node's two children the CTA that arrives first stores its ciphertext and
// ends, the second takes it from there, so no CTA ever waits and the upper
// levels of the first queries fill the gaps that the last chains leave.  The CTA
// left at the root transforms it back and writes pack_lwes' result
// (automorph_pack.rs:466-484): b_val_z * d added at coefficient z < ncols; one
// LWE alone is returned unpacked (automorph_pack.rs:439-446), (a, b_val at
// coefficient 0).
// CTAS per SM: one, with the registers of both, while every LWE has an SM (9
// queries of 16 take 126 us, 132 with two; 33 take 282, 291 with one).
template <int CTAS>
__global__ void __launch_bounds__(QT, CTAS) tree_kernel(const __grid_constant__ TreeArgs A) {
  extern __shared__ __align__(128) uint32_t smem[];
  __shared__ uint32_t arrived;
  const DevParams& P = A.P;
  const int qi = blockIdx.x / A.ncols;
  int s = blockIdx.x - qi * A.ncols;
  const int r = threadIdx.x >> 7, x = threadIdx.x & 127;
  const uint32_t base = jx_addr(smem);
  pdl_wait();
  if (A.shard[qi] >= (uint32_t)A.nshards) {  // uniform over the CTA
    if (s == 0 && threadIdx.x == 0) A.status[qi] = ERR_INDEX;
    return;
  }
  const ResidueConsts& C = P.r[r];
  const uint32_t q = C.q, q2 = 2 * q;
  uint32_t* W = A.work + (size_t)qi * WORK_WORDS;
  uint32_t* own = W + (size_t)r * N + x;
  uint32_t a[16], b[16];
#pragma unroll
  for (int j = 0; j < 16; j++) {
    a[j] = own[(size_t)s * CT_WORDS + 128 * h_of(j)];
    b[j] = 0;
  }
#pragma unroll 1
  for (int l = A.ncols == 1 ? LOGN + 1 : 1; l <= LOGN; l++) {
    uint32_t sa[16], sb[16];  // s1; a, b become s0
#pragma unroll
    for (int j = 0; j < 16; j++) {
      sa[j] = a[j];
      sb[j] = b[j];
    }
    const int nn = 1 << (LOGN - l);
    if (l >= 8 && (s & (nn - 1)) + nn < A.ncols) {
      const int node = s & (nn - 1);
      const bool odd = s != node;
      if (odd) {  // X^(d >> l) odd: times psi^((d >> l)(2brv(s)+1)), psi^N = -1
        const uint32_t e0 = (uint32_t)nn * (2u * (__brev((uint32_t)x) >> 25) + 1u);
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const uint32_t ex = e0 + (uint32_t)nn * 256u * (uint32_t)h_of(j);
          const uint2 w = __ldg(C.fwd + brv11(ex & (N - 1)));
          a[j] = mul_shoup_lazy(a[j], w, q);
          b[j] = mul_shoup_lazy(b[j], w, q);
          if (ex & N) {
            a[j] = q2 - a[j];
            b[j] = q2 - b[j];
          }
        }
      }
      uint32_t* me = own + (size_t)(level_base(l - 1) + s) * CT_WORDS;
#pragma unroll
      for (int j = 0; j < 16; j++) {
        __stcg(me + 128 * h_of(j), a[j]);
        __stcg(me + 2 * N + 128 * h_of(j), b[j]);
      }
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) arrived = atomicAdd(W + WORK_ARRIVED + nn + node, 1u);
      __syncthreads();
      if (arrived == 0) return;  // uniform over the CTA: the sibling goes on
      __threadfence();
      const uint32_t* sib = own + (size_t)(level_base(l - 1) + (s ^ nn)) * CT_WORDS;
#pragma unroll
      for (int j = 0; j < 16; j++) {
        sa[j] = __ldcg(sib + 128 * h_of(j));
        sb[j] = __ldcg(sib + 2 * N + 128 * h_of(j));
      }
#pragma unroll
      for (int j = 0; j < 16; j++) {  // the odd parts are up to 2q
        const uint32_t ua = a[j], va = sa[j], ub = b[j], vb = sb[j];
        a[j] = csub(ua + va, q2);
        b[j] = csub(ub + vb, q2);
        sa[j] = odd ? va - ua + q2 : ua - va + q2;
        sb[j] = odd ? vb - ub + q2 : ub - vb + q2;
      }
    }
    if (l >= 8) s &= nn - 1;
    key_switch(A, base, l, sa, sb, a, b);
  }
  if (threadIdx.x == 0) {
    bool good = true;
#pragma unroll
    for (int t = 0; t < ELL; t++) good &= W[WORK_GOOD + t] != 0;
    A.status[qi] = good ? 0 : ERR_EXPAND;
  }
  const uint32_t xb = base + 4 * (SwitchSmem::XB + 2 * N * r);
  const uint32_t sc[2] = {xb, xb + 4 * N};
  uint32_t c[2][16];
#pragma unroll
  for (int j = 0; j < 16; j++) {
    c[0][j] = a[j];
    c[1][j] = b[j];
  }
  jntt_inv<2>(c, sc, sfwd_tw(C), q, x, 1 + r);
  uint64_t* out = A.out_a + (size_t)qi * 2 * N + (size_t)r * N + x;
#pragma unroll
  for (int j = 0; j < 16; j++) out[128 * j] = c[0][j];
  const uint32_t* bv = W + WORK_BVALS;
  out = A.out_b + (size_t)qi * 4 * N + (size_t)r * N + x;
  if (A.mode == MODE_CRT_FIXED || A.ncols == 1) {
    if (x < A.ncols)
      c[1][0] = add_mod(c[1][0], (uint32_t)((uint64_t)bv[16 * r + x] * (A.ncols == 1 ? 1 : N) % q), q);
#pragma unroll
    for (int j = 0; j < 16; j++) out[128 * j] = c[1][j];
  } else {
    // compat: the crate adds b_val_z * d to the first d words of the
    // residue-major b vector and rebuilds a polynomial of dimension 2d from
    // all 2d words (Poly::from_coeffs_moduli, math/poly.rs:127-159)
    const uint32_t q0 = P.r[0].q, q1 = P.r[1].q;
    const uint64_t qc = (uint64_t)q0 * q1;
#pragma unroll
    for (int j = 0; j < 16; j++) {
      uint64_t bc = c[1][j];
      if (j == 0 && r == 0 && x < A.ncols) {
        uint64_t v = crt_compose(P, bv[x], bv[16 + x]);
        for (int k = 0; k < LOGN; k++) {  // b_val * d mod q by doubling (q < 2^56)
          v <<= 1;
          if (v >= qc) v -= qc;
        }
        bc += v;
        if (bc >= qc) bc -= qc;
      }
      out[128 * j] = bc % q0;
      out[2 * N + 128 * j] = bc % q1;
    }
  }
}

// Galois key table [key][part a, b][k][residue], quads: each of the log2(d)
// matrices' ELL rows (a, b), NTT-transformed, scaled by n^-1 2^32 and with the
// third digit folded in.  keys[key][k][part][residue][N].  One CTA per (key,
// part) and residue.
__global__ void __launch_bounds__(NTT_GT) galois_prep_kernel(const DevParams P, const uint64_t* __restrict__ keys,
                                                             uint32_t* __restrict__ ks) {
  __shared__ __align__(128) uint32_t X[ELL][N];
  const int key = blockIdx.x >> 1, part = blockIdx.x & 1, r = blockIdx.y, x = threadIdx.x;
  const ResidueConsts& C = P.r[r];
  const uint32_t q = C.q;
  uint32_t v[ELL][16];
#pragma unroll
  for (int k = 0; k < ELL; k++)
#pragma unroll
    for (int j = 0; j < 16; j++)
      v[k][j] = (uint32_t)keys[((((size_t)key * ELL + k) * 2 + part) * 2 + r) * N + x + 128 * j];
  const uint32_t sc[ELL] = {jx_addr(X[0]), jx_addr(X[1]), jx_addr(X[2])};
  jntt_fwd<ELL, JB_CANON>(v, sc, sfwd_tw(C), q, x, 1);
  fold_keys(v, C);
  uint32_t* o = ks + ((size_t)blockIdx.x * ELL * 2 + r) * N;
#pragma unroll
  for (int k = 0; k < ELL; k++)
#pragma unroll
    for (int j = 0; j < 16; j += 4)
      *reinterpret_cast<uint4*>(o + (size_t)k * 2 * N + quad_word(j, x)) =
          make_uint4(v[k][j], v[k][j + 1], v[k][j + 2], v[k][j + 3]);
}

// Static scratch of the allocation-free tree-packing entry: the work areas.
__device__ __align__(256) uint32_t g_tree_noalloc_scratch[TREE_NOALLOC_MAX_QUERIES * WORK_WORDS];

}  // namespace


// Device address of the static scratch in the current device's context.
// Looked up on every call rather than cached: the lookup is cheap and
// allocates nothing, and a cached address would go stale if the context were
// destroyed and re-created (cudaDeviceReset) within the process.
cudaError_t tree_noalloc_scratch(int device, void** ptr) {
  int cur = -1;
  cudaError_t e = cudaGetDevice(&cur);
  if (e != cudaSuccess) return e;
  if (cur != device) return cudaErrorInvalidDevice;  // the caller makes `device` current first
  return cudaGetSymbolAddress(ptr, g_tree_noalloc_scratch);
}

size_t tree_work_words_per_query() { return WORK_WORDS; }

constexpr int SWITCH_BYTES = (int)sizeof(uint32_t) * SwitchSmem::TOTAL;

cudaError_t prepare_tree_kernels() {
  const cudaError_t e = cudaFuncSetAttribute(tree_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SWITCH_BYTES);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(tree_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, SWITCH_BYTES);
}

cudaError_t launch_tree(const TreeArgs& a, bool seeded, cudaStream_t st) {
  if (a.nq <= 0) return cudaSuccess;
  void (*leaves)(TreeArgs) = nullptr;
  switch (a.ncols) {
    case 1: leaves = tree_leaves_kernel<1>; break;
    case 2: leaves = tree_leaves_kernel<2>; break;
    case 4: leaves = tree_leaves_kernel<4>; break;
    case 8: leaves = tree_leaves_kernel<8>; break;
    case 16: leaves = tree_leaves_kernel<16>; break;
    default: return cudaErrorInvalidValue;
  }
  if (seeded) tree_front_kernel<true><<<a.nq * (ELL + 1), QT, 0, st>>>(a);
  else tree_front_kernel<false><<<a.nq * (ELL + 1), QT, 0, st>>>(a);
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(QT);
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(a.nq * 2 * (128 / LEAF_RUNS));
  cudaError_t e = cudaLaunchKernelEx(&cfg, leaves, a);
  if (e != cudaSuccess) return e;
  cfg.gridDim = dim3(a.nq * a.ncols);
  cfg.dynamicSmemBytes = SWITCH_BYTES;
  return cudaLaunchKernelEx(&cfg, a.nq * a.ncols <= a.sm_count ? tree_kernel<1> : tree_kernel<2>, a);
}

cudaError_t launch_galois_prep(const DevParams& P, const uint64_t* keys, int nkeys, uint32_t* ks, cudaStream_t st) {
  if (nkeys <= 0) return cudaSuccess;
  galois_prep_kernel<<<dim3(2 * nkeys, 2), NTT_GT, 0, st>>>(P, keys, ks);
  return cudaGetLastError();
}

}  // namespace ig
