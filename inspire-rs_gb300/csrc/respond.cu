// respond.cu -- fused InsPIRe^2 Respond kernel: one CTA of 256 threads per
// query, two CTAs per SM.
//
// Computes, for one seeded query against one resident shard, exactly what
// respond_seeded_inspiring / respond_inspiring (src/pir/respond.rs:284-398)
// return: the packed RLWE ciphertext (a_hat, b) of packing_online
// (src/inspiring/inspiring2.rs:1185-1222).  The reference's steps are
// regrouped into an equivalent exact dataflow:
//
//  * expand (rgsw/types.rs:315-318): only RGSW rows ELL..2ELL-1 are needed,
//    because the database ciphertext is (0, Delta*h) (rlwe/enc.rs:174-182) and
//    every digit of its zero a-part is 0 (rgsw/external_product.rs:122-147).
//  * b-part of each column product, coefficient 0 only
//    (rlwe/enc.rs:195-208): b0_c = sum_t sum_i d_{c,t}[i] * b'_t[i] with
//    d = base-2^20 digits of Delta*h_c and b'_t the negacyclic reversal of row
//    ELL+t's b, accumulated exactly in 64 bits.
//  * a-part + the first stage of packing_offline (inspiring2.rs:948-982): the
//    per-slot 16x16 monomial inner products, the 1/gamma scaling and the 16
//    NTT-domain automorphisms reduce to a length-gamma DFT per NTT slot, which
//    is folded into the resident database ("E", built in setup.cu); per slot
//    only sum_t E[i,t][s] * A_t[tau_i(s)] remains.
//  * the backward recursion (inspiring2.rs:984-1008) and packing_online run
//    interleaved: each T[i][k] NTT is multiplied into R[i] with the CRS key
//    w_all and into the b accumulator with the client key y_all, the third
//    gadget digit folded into the keys (fold_third_digit_kernel, setup.cu).
//
// Layout.  Group r of 128 threads owns CRT residue r, thread x of it the 16
// NTT slots 16x .. 16x+15 of every polynomial.  The automorphisms tau_{g^i}
// (g = 2N/gamma + 1) permute slots only inside such runs (rot_rows,
// respond_common.cuh), so a recursion step is private to its thread in the
// NTT domain: R_{i+1} and the b accumulator stay in registers, the row
// transforms (AH) in words of shared memory that no other thread reads, and
// the nine products of a slot share two Montgomery reductions.  Threads meet
// only in the transforms' exchanges and, warp to warp, where the composite
// coefficient needs both residues:
//   [A] INTT(R_{i+1}) in registers;
//   [B] the residues swapped through shared memory, digits d0, d1 of the
//       composite coefficients computed by both groups (64-thread barrier);
//   [C] NTT(d0), NTT(d1) together (one set of twiddle loads);
//   [D] R_i = sum_t E A_t + NTT(d0) w'0 + NTT(d1) w'1 + R_{i+1} w'2,
//       b += NTT(d0) y'0 + NTT(d1) y'1 + R_{i+1} y'2.
// Three barriers a step, each over one group or one pair of warps.
//
// What bounds it: the integer multiply-add pipe (64 lane-operations per
// cycle and SM, a high or wide product costs two) is 73 % busy, 86 % in the
// digit transforms; the rest waits on 16 warps' latencies.  Two CTAs of different
// queries share the SM without waiting for each other, and 128 registers a
// thread let each warp keep 16 independent butterflies in flight.  One call of
// 2048 queries takes 1355 us, 1507 us with unsigned butterflies and the step's
// database and CRS words loaded where they are used, 2290 us with one CTA of 24
// warps in step per SM.
#include "ntt_joint.cuh"
#include "respond_draws.cuh"

namespace ig {

namespace {

// Shared memory in u32 words (NR = residues of the a side).  80 KiB and a
// little: two CTAs fit the SM's 164 KiB configuration, which leaves it 92 KiB
// of L1 for the twiddles and the client keys.
template <int NR>
struct Smem {
  static constexpr int AH = 0;                 // [ELL][NR][16 rows h][128] row transforms
  static constexpr int XC = AH + ELL * NR * N; // [4][N] exchange buffers: 2 shared by turns, 1 per residue
  static constexpr int WS = XC + 4 * N;        // [2][8] scan totals, [3] expansion totals, flags
  static constexpr int BP = WS + 32;           // [2][16] the b side
  static constexpr int SEED = BP + 32;         // [ELL * 8] staged seeds (serving loop)
  static constexpr int BAR = SEED + 24;        // the staged rows' mbarrier
  static constexpr int TOTAL = BAR + 8;
  // (the transforms' swizzled accesses XOR address bits 2-6)
  static_assert(AH * 4 % 128 == 0 && XC * 4 % 128 == 0 && BAR % 2 == 0 && TOTAL % 4 == 0,
                "alignment of rows, buffers, mbarrier and whole staged rows");
};

// One query (index qi) by the whole CTA; every return is uniform over the CTA.
// ALONE: the SM is this CTA's, with registers for all of a step's database and
// CRS words at once.  WHOLE (QDB, ALONE): and with shared memory for the whole
// rows, from Smem::TOTAL on.
template <int MODE, bool SEEDED, bool QDB, bool ALONE, bool WHOLE = false>
__device__ __forceinline__ void respond_one(const RespondArgs& A, const int qi) {
  constexpr int NR = MODE == MODE_COMPAT ? 1 : 2;
  using L = Smem<NR>;
  extern __shared__ __align__(128) uint32_t smem[];
  uint32_t* AH = smem + L::AH;
  uint32_t* XC = smem + L::XC;
  int* ws = reinterpret_cast<int*>(smem + L::WS);
  uint32_t* bpoly = smem + L::BP;

  const DevParams& P = A.P;
  const int tid = threadIdx.x, r = tid >> 7, x = tid & 127;
  const int gamma = P.gamma;
  // QDB (serving loop): this query's fields come from its descriptor in
  // device memory, its rows and response from / to pinned host memory;
  // otherwise from the launch's arrays.  Descriptor fields are re-read where
  // used (reload_ptr) rather than held in registers.
  const QueryDesc* D = QDB ? A.qdesc + qi : nullptr;
  const uint32_t shard = QDB ? D->shard : A.shard[qi];
  const int32_t cid = QDB ? D->client : A.client[qi];
  const uint32_t* Ebase = QDB ? D->db.E : A.E;
  const uint16_t* H = (QDB ? D->db.H : A.H) + (size_t)shard * gamma * N;
  const int nshards = QDB ? D->db.nshards : A.nshards;
  auto status_ptr = [&]() -> int32_t* {
    return QDB ? reload_ptr(&D->status) : A.status + qi;
  };
  if (shard >= (uint32_t)nshards || cid < 0 || cid >= A.nclients || A.yhat_table[cid] == nullptr) {
    if (tid == 0) *status_ptr() = ERR_INDEX;
    return;  // uniform over the CTA
  }
  // the a side's residue: this group's, or residue 0 for both in compat mode
  const int sres = MODE == MODE_CRT_FIXED ? r : 0;
  const uint32_t* E = Ebase + ((size_t)shard * 2 + sres) * ELL * gamma * N;
  // The client's key table: a body table (tag bit 0 set: NTT(y_body[k]),
  // ELL polys, 48 KiB) whose rotations are formed by the rows read, or the
  // full table of (gamma-1)*ELL rotated polys (explicit y_all).
  const uintptr_t ytag = reinterpret_cast<uintptr_t>(A.yhat_table[cid]);
  const bool ybody = (ytag & 1) != 0;
  const uint32_t* Y = reinterpret_cast<const uint32_t*>(ytag & ~(uintptr_t)1);
  const ResidueConsts& C = P.r[r];
  const uint32_t q = C.q, qinv = C.qinv, qo = P.r[r ^ 1].q;
  const uint64_t* brows = QDB ? D->brows : A.brows + (size_t)qi * ELL * 2 * N;
  uint64_t* rbar = reinterpret_cast<uint64_t*>(smem + L::BAR);
  uint64_t* stage = reinterpret_cast<uint64_t*>(WHOLE ? smem + L::TOTAL : XC);

  if (tid == 0) {
    if (QDB) mbar_init(rbar);
    // the contracted shard's blocks of the first steps (the rest are
    // prefetched two steps ahead of their use), the raw columns, the keys
    prefetch_l2(H, sizeof(uint16_t) * (size_t)gamma * N);
    const int i0 = gamma >= 3 ? gamma - 3 : 0;
    for (int rr = 0; rr < NR; rr++)
      prefetch_l2(Ebase + (((size_t)shard * 2 + rr) * gamma + i0) * ELL * N,
                  sizeof(uint32_t) * (size_t)(gamma - i0) * ELL * N);
    if (gamma > 1) prefetch_l2(Y, sizeof(uint32_t) * (size_t)(ybody ? 1 : gamma - 1) * ELL * 2 * N);
  }
  const uint8_t* seeds = nullptr;
  if (SEEDED) seeds = QDB ? reinterpret_cast<const uint8_t*>(smem + L::SEED) : A.seeds + (size_t)qi * ELL * 32;
  if (QDB) {
    // the seeds, inline in the query's descriptor
    if (SEEDED && tid < ELL * 32) reinterpret_cast<uint8_t*>(smem + L::SEED)[tid] = D->seeds[tid];
    __syncthreads();  // the mbarrier is initialised, the seeds staged
    if (tid == 0) {
      if (WHOLE) stage_rows(stage, brows, rbar);
      else stage_chunk(stage, brows, 0, rbar);
    }
  }

  // ---- rows ELL..2ELL-1, coefficients, into AH [t][NR][N] ----
  if (SEEDED) {
    expand_rows<NR>(P, seeds, AH, ws);
  } else {
    const uint64_t* ar = A.arows + (size_t)qi * ELL * 2 * N;
#pragma unroll 16
    for (int j = tid; j < ELL * NR * N; j += QT) {
      const int t = j / (NR * N);
      AH[j] = (uint32_t)__ldg(ar + (size_t)t * 2 * N + (j - t * NR * N));
    }
  }

  // ---- the b side ----
  constexpr RowSource SRC = WHOLE ? ROWS_WHOLE : QDB ? ROWS_CHUNKS : ROWS_DIRECT;
  const int missing = column_b0<SRC>(P, H, brows, stage, rbar, A.stage_wait_iters, reinterpret_cast<uint64_t*>(XC), bpoly);
  if (QDB && missing >= 0) {
    // The CTA must not exit while its bulk copies can still write into its
    // shared memory (the next CTA on this SM would own it): a second bounded
    // wait, for the chunk in flight.  If even that runs out, ERR_STAGE_LOST
    // tells the host to drop every result of this launch.
    const int lost = __syncthreads_or(!mbar_wait(rbar, missing & 1, STAGE_DRAIN_ITERS));
    if (tid == 0) *status_ptr() = lost ? ERR_STAGE_LOST : ERR_STAGE;
    return;  // uniform over the CTA
  }
  // ---- rows that the fast expansion left to the general one ----
  if (SEEDED) {
    bool good = true;
#pragma unroll 1
    for (int t = 0; t < ELL; t++)
      if (!ws[20 + t]) {  // uniform; ordered by the b side's barriers
        good &= expand_row_general<NR>(P, seeds + 32 * t, reinterpret_cast<uint64_t*>(XC), AH + t * NR * N, ws);
        __syncthreads();
      }
    if (tid == 0) *status_ptr() = good ? 0 : ERR_EXPAND;
  } else {
    if (tid == 0) *status_ptr() = 0;
  }

  const uint32_t xc = jx_addr(XC);
  // ---- row transforms, into rows h of AH (a slot's words are its thread's).
  //      Consecutive transforms use two exchange buffers by turns: one ends
  //      with reads that another warp's next first writes could overtake ----
  {
    const ResidueConsts& Cs = P.r[sres];
#pragma unroll 1
    for (int t = NR == 2 ? 0 : r, turn = 0; t < ELL; t += NR == 2 ? 1 : 2, turn ^= 1) {
      uint32_t* row = AH + (t * NR + sres) * N;
      uint32_t v[1][16];
      const uint32_t sc[1] = {xc + 4 * N * (turn ? r : 2 + r)};
#pragma unroll
      for (int j = 0; j < 16; j++) v[0][j] = row[x + 128 * j];
      jntt_fwd<1, JB_CANON>(v, sc, sfwd_tw(Cs), Cs.q, x, 1 + r);
#pragma unroll
      for (int j = 0; j < 16; j++) row[128 * h_of(j) + x] = jcanon_fwd(v[0][j], Cs.q);
    }
    if (NR == 1) __syncthreads();  // both groups read the rows of residue 0
  }

  // Row h + rot of a table of rows, [k or t][residue][h][x], is at one byte
  // offset in the client's keys and in AH (without the residue there in
  // compat mode): (h + rot) << 9 in bits 9-12, the rest fixed.
  const uint32_t ah = jx_addr(AH);
  const uint32_t rx = 4u * (uint32_t)x + (uint32_t)r * 4u * N;
  auto row_off = [&](uint32_t rot9, int h) -> uint32_t { return ((rot9 + 512u * (uint32_t)h) & 0x1E00u) | rx; };
  const char* Yb = reinterpret_cast<const char*>(Y);
  const uint32_t* Ex = E + 4 * x;
  const uint32_t* Wx = A.what + r * N + 4 * x;
  // sum_t E[i,t][s] A_t[tau_i(s)] for the four slots l = 4 a + j of this thread
  auto query_only = [&](const uint4& e0, const uint4& e1, const uint4& e2, const uint32_t (&ro)[4], uint64_t T[4]) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t ar = ah + ro[j] - (NR == 1 ? (uint32_t)r * 4u * N : 0u);
      T[j] = (uint64_t)u4e(e0, j) * jx_at(ar) + (uint64_t)u4e(e1, j) * jx_at(ar + 4 * NR * N) +
             (uint64_t)u4e(e2, j) * jx_at(ar + 8 * NR * N);
    }
  };
  // compat mode, residue 1: rebuilt from the residue-0 value as the crate's
  // apply_automorphism_ntt does
  const bool conv1 = MODE == MODE_COMPAT && r == 1;
  auto converted = [&](uint64_t T) -> uint32_t {
    return compat_residue1_ninv(P, redc(T, P.r[0].q, P.r[0].qinv));
  };

  uint32_t R[16], acc[16];  // R_{i+1} and the b accumulator, slot layout
  {
    const uint32_t rot9 = rot_rows(gamma, gamma - 1, x) << 9;
    const uint32_t* e = Ex + (size_t)(gamma - 1) * ELL * N;
#pragma unroll
    for (int a = 0; a < 4; a++) {
      uint64_t T[4];
      const uint32_t ro[4] = {row_off(rot9, h_of(4 * a)), row_off(rot9, h_of(4 * a + 1)),
                              row_off(rot9, h_of(4 * a + 2)), row_off(rot9, h_of(4 * a + 3))};
      query_only(ld_stream(e + 512 * a), ld_stream(e + N + 512 * a), ld_stream(e + 2 * N + 512 * a), ro, T);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int l = 4 * a + j;
        R[l] = conv1 ? converted(T[j]) : redc_wide(T[j], q, qinv);
        acc[l] = 0;
      }
    }
  }

  const uint32_t own = xc + 4 * N * (2 + r);
  uint32_t mine = xc + 4 * N * r, other = xc + 4 * N * (r ^ 1);
#pragma unroll 1
  for (int i = gamma - 2; i >= 0; i--) {
    if (tid == 0 && i >= 2)  // the block that step i - 2 reads
      for (int rr = 0; rr < NR; rr++)
        prefetch_l2(Ebase + (((size_t)shard * 2 + rr) * gamma + (i - 2)) * ELL * N, sizeof(uint32_t) * ELL * N);
    // [A] inverse NTT of R_{i+1} ([0, 3.1 q))
    uint32_t v[2][16];
    {
      uint32_t c[1][16], o[1][16];
#pragma unroll
      for (int j = 0; j < 16; j++) c[0][j] = R[j];
      const uint32_t sc[1] = {own}, sm1[1] = {mine}, so1[1] = {other};
      jntt_inv<1>(c, sc, sfwd_tw(C), q, x, 1 + r);
      // [B] the residues trade coefficients, thread for thread: each writes
      // its own to the buffer it has been using, reads the other group's,
      // and goes on with that buffer.  Digits 0 and 1 of the composite
      // coefficients (gadget_decompose, rgsw/external_product.rs:16-37).
      jx_store_co<1>(c, sm1, x);
      named_sync(3 + (x >> 5), 64);
      jx_load_co<1>(o, so1, x);
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const uint64_t cc = crt_compose_from(C, qo, c[0][j], o[0][j]);
        v[0][j] = (uint32_t)cc & 0xFFFFFu;
        v[1][j] = (uint32_t)(cc >> 20) & 0xFFFFFu;
      }
    }
    // [C] with the first quad (all four) of the step's database and CRS words on
    // its way
    const uint32_t* wi = Wx + (size_t)i * ELL * 2 * N;
    const uint32_t* ei = Ex + (size_t)i * ELL * N;
    uint4 nx[ALONE ? 4 : 1][6];
    auto fetch = [&](int a) {
      uint4(&to)[6] = nx[ALONE ? a : 0];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        to[k] = ld_stream(ei + k * N + 512 * a);
        to[3 + k] = ld_stream(wi + 2 * k * N + 512 * a);
      }
    };
    const uint32_t sc2[2] = {other, own};
    jntt_fwd<2, JB_DIGIT>(v, sc2, sfwd_tw(C), q, x, 1 + r, [&]() {  // signed, below 5.25 q
#pragma unroll
      for (int a = 0; a < (ALONE ? 4 : 1); a++) fetch(a);
    });
    other = mine;
    mine = sc2[0];
    // [D] the nine products of each slot under two reductions, in signed
    // 64-bit sums.  With R in [0, 3.1 q), NTT(d) below 5.25 q and the rest
    // canonical, R's sum is in (-10.5 q^2, 16.6 q^2); q < 2^28, so its
    // reduction plus q is in (0.3 q, 3.1 q).  b's part plus q is in (0.3 q,
    // 2.9 q), and b is kept below 8 q.
    const uint32_t rot9 = rot_rows(gamma, i, x) << 9;
    const char* yi = ybody ? Yb : Yb + (size_t)i * ELL * 2 * N * 4;
#pragma unroll
    for (int a = 0; a < 4; a++) {
      uint64_t T[4];
      uint4 cu[6];
#pragma unroll
      for (int k = 0; k < 6; k++) cu[k] = nx[ALONE ? a : 0][k];
      if (!ALONE && a < 3) fetch(a + 1);
      const uint32_t ro[4] = {row_off(rot9, h_of(4 * a)), row_off(rot9, h_of(4 * a + 1)),
                              row_off(rot9, h_of(4 * a + 2)), row_off(rot9, h_of(4 * a + 3))};
      query_only(cu[0], cu[1], cu[2], ro, T);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int l = 4 * a + j;
        const uint32_t* y = reinterpret_cast<const uint32_t*>(yi + ro[j]);
        const uint32_t y0 = __ldg(y), y1 = __ldg(y + 2 * N), y2 = __ldg(y + 4 * N);
        uint64_t S = conv1 ? 0ull : T[j];
        S += smul(v[0][l], u4e(cu[3], j));
        S += smul(v[1][l], u4e(cu[4], j));
        S += smul(R[l], u4e(cu[5], j));
        const uint64_t B = smul(v[0][l], y0) + smul(v[1][l], y1) + smul(R[l], y2);
        R[l] = redc_wide(S, q, qinv) + (conv1 ? converted(T[j]) : 0u) + q;
        acc[l] = csub(acc[l] + redc_wide(B, q, qinv) + q, 8 * q);
      }
    }
  }

  // ---- outputs: a_hat = INTT(R_0) (inspiring2.rs:1027-1029), b = b_poly +
  //      INTT(sum y_all * bold_t) (inspiring2.rs:1217-1221) ----
  uint64_t* out = QDB ? reload_ptr(&D->out) : A.out + (size_t)qi * 4 * N;
#pragma unroll 1
  for (int part = 0; part < 2; part++) {
    uint32_t o[1][16];
    const uint32_t sc[1] = {part ? mine : own};
#pragma unroll
    for (int j = 0; j < 16; j++) o[0][j] = part ? csub(acc[j], 4 * q) : R[j];
    jntt_inv<1>(o, sc, sfwd_tw(C), q, x, 1 + r);
    if (part && x < gamma) o[0][0] = add_mod(o[0][0], bpoly[16 * r + x], q);
#pragma unroll
    for (int j = 0; j < 16; j++) out[part * 2 * N + r * N + x + 128 * j] = o[0][j];
  }
}

// One query per CTA, two CTAs per SM.
template <int MODE, bool SEEDED, bool QDB>
__global__ void __launch_bounds__(QT, 2) respond_kernel(const __grid_constant__ RespondArgs A) {
  respond_one<MODE, SEEDED, QDB, false>(A, blockIdx.x);
}

// One query per CTA and SM, for seeded batches of at most as many queries as SMs:
// 128 queries take 117 us, 131 with 128 registers a thread (half the register
// file idle, the step's words waited for quad by quad), 77 in compat mode 115
// and 129.  The same for 2048 queries takes 1570 us, 1355 with two CTAs per SM.
template <int MODE, bool QDB>
__global__ void __launch_bounds__(QT, 1) respond_kernel_alone(const __grid_constant__ RespondArgs A) {
  respond_one<MODE, true, QDB, true>(A, blockIdx.x);
}

// The same with the whole rows staged while they are expanded, for large batches
// of few columns whose rows and responses cross the host link (batch_policy.h).
template <int MODE>
__global__ void __launch_bounds__(QT, 1) respond_kernel_whole(const __grid_constant__ RespondArgs A) {
  respond_one<MODE, true, true, true, true>(A, blockIdx.x);
}

// Capped grid (seeded queries, device-resident rows): CTA b answers queries b,
// b + gridDim.x, ... in turn.
template <int MODE>
__global__ void __launch_bounds__(QT, 2) respond_kernel_loop(const __grid_constant__ RespondArgs A) {
#pragma unroll 1
  for (int qi = blockIdx.x; qi < A.nq; qi += gridDim.x) {
    if (qi != (int)blockIdx.x) __syncthreads();  // the previous query's shared memory is no longer read
    respond_one<MODE, true, false, false>(A, qi);
  }
}

}  // namespace

size_t respond_smem_bytes(int mode) {
  return sizeof(uint32_t) * (mode == MODE_COMPAT ? Smem<1>::TOTAL : Smem<2>::TOTAL);
}
static size_t whole_smem_bytes(int mode) { return respond_smem_bytes(mode) + sizeof(uint64_t) * 2 * ELL * N; }

template <int MODE, bool SEEDED, bool QDB>
static cudaError_t set_smem_attr() {
  return cudaFuncSetAttribute(respond_kernel<MODE, SEEDED, QDB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)respond_smem_bytes(MODE));
}
template <int MODE>
static cudaError_t set_loop_smem_attr() {
  return cudaFuncSetAttribute(respond_kernel_loop<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)respond_smem_bytes(MODE));
}

// Launches issue no configuration call (so they can be captured in a CUDA
// graph): the shared-memory attribute of every variant is set once per
// device by prepare_respond_kernels.
template <int MODE>
static cudaError_t launch_whole(const RespondArgs& a, cudaStream_t st) {
  respond_kernel_whole<MODE><<<a.nq, QT, whole_smem_bytes(MODE), st>>>(a);
  return cudaGetLastError();
}
template <int MODE, bool SEEDED, bool QDB>
static cudaError_t launch_one(const RespondArgs& a, cudaStream_t st) {
  respond_kernel<MODE, SEEDED, QDB><<<a.nq, QT, respond_smem_bytes(MODE), st>>>(a);
  return cudaGetLastError();
}
template <int MODE>
static cudaError_t launch_loop(const RespondArgs& a, int ctas, cudaStream_t st) {
  respond_kernel_loop<MODE><<<ctas, QT, respond_smem_bytes(MODE), st>>>(a);
  return cudaGetLastError();
}

template <int MODE>
static cudaError_t set_whole_smem_attr() {
  return cudaFuncSetAttribute(respond_kernel_whole<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)whole_smem_bytes(MODE));
}
template <int MODE, bool QDB>
static cudaError_t set_alone_smem_attr() {
  return cudaFuncSetAttribute(respond_kernel_alone<MODE, QDB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)respond_smem_bytes(MODE));
}

cudaError_t prepare_respond_kernels() {
  const cudaError_t es[] = {
      set_whole_smem_attr<MODE_COMPAT>(),            set_whole_smem_attr<MODE_CRT_FIXED>(),
      set_loop_smem_attr<MODE_COMPAT>(),             set_loop_smem_attr<MODE_CRT_FIXED>(),
      set_alone_smem_attr<MODE_COMPAT, false>(),     set_alone_smem_attr<MODE_COMPAT, true>(),
      set_alone_smem_attr<MODE_CRT_FIXED, false>(),  set_alone_smem_attr<MODE_CRT_FIXED, true>(),
      set_smem_attr<MODE_COMPAT, false, false>(),    set_smem_attr<MODE_COMPAT, true, false>(),
      set_smem_attr<MODE_COMPAT, false, true>(),     set_smem_attr<MODE_COMPAT, true, true>(),
      set_smem_attr<MODE_CRT_FIXED, false, false>(), set_smem_attr<MODE_CRT_FIXED, true, false>(),
      set_smem_attr<MODE_CRT_FIXED, false, true>(),  set_smem_attr<MODE_CRT_FIXED, true, true>()};
  for (cudaError_t e : es)
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}

template <int MODE>
static cudaError_t launch_alone(const RespondArgs& a, cudaStream_t st) {
  if (a.qdesc) respond_kernel_alone<MODE, true><<<a.nq, QT, respond_smem_bytes(MODE), st>>>(a);
  else respond_kernel_alone<MODE, false><<<a.nq, QT, respond_smem_bytes(MODE), st>>>(a);
  return cudaGetLastError();
}

template <int MODE>
static cudaError_t launch_mode(const RespondArgs& a, bool seeded, cudaStream_t st) {
  if (a.qdesc) return seeded ? launch_one<MODE, true, true>(a, st) : launch_one<MODE, false, true>(a, st);
  return seeded ? launch_one<MODE, true, false>(a, st) : launch_one<MODE, false, false>(a, st);
}

cudaError_t launch_respond(const RespondArgs& a, bool seeded, cudaStream_t st, int max_ctas, int pair_max) {
  if (a.nq <= 0) return cudaSuccess;
  if (max_ctas <= 0 && a.nq <= pair_max) return launch_respond_pair(a, seeded, st);
  if (a.whole_rows && max_ctas <= 0 && seeded && a.qdesc)
    return a.P.mode == MODE_COMPAT ? launch_whole<MODE_COMPAT>(a, st) : launch_whole<MODE_CRT_FIXED>(a, st);
  if (max_ctas <= 0 && seeded && a.nq <= a.alone_max)
    return a.P.mode == MODE_COMPAT ? launch_alone<MODE_COMPAT>(a, st) : launch_alone<MODE_CRT_FIXED>(a, st);
  if (max_ctas > 0 && max_ctas < a.nq) {
    if (!seeded || a.qdesc) return cudaErrorInvalidValue;
    return a.P.mode == MODE_COMPAT ? launch_loop<MODE_COMPAT>(a, max_ctas, st)
                                   : launch_loop<MODE_CRT_FIXED>(a, max_ctas, st);
  }
  return a.P.mode == MODE_COMPAT ? launch_mode<MODE_COMPAT>(a, seeded, st) : launch_mode<MODE_CRT_FIXED>(a, seeded, st);
}

}  // namespace ig
