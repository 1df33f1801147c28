// nopacking.cu -- NoPacking Respond.
//
// respond (src/pir/respond.rs:71-115) and respond_seeded (:408-415): for every
// column c of the named shard, column_ciphertexts[c] =
// external_product(trivial_encrypt(h_c), rgsw) (rgsw/external_product.rs:88-150),
// and the combined ciphertext is their sum (respond.rs:102-109).  As in the
// packed path, only RGSW rows ELL..2ELL-1 contribute (the a part of the
// trivial encryption is zero), so a_c = sum_t D_{c,t} * a_t and
// b_c = sum_t D_{c,t} * b_t with D_{c,t} the base-2^20 digit t of Delta*h_c.
//
// With column ciphertexts (nopacking_kernel): 768 threads = six groups of 128;
// group g = 3 r + t owns CRT residue r and row/digit t and keeps NTT(a_t),
// NTT(b_t) of its residue in registers (Montgomery form with n^-1 folded) for
// all columns.  Per column: six digit NTTs and products, then groups
// (r,0)/(r,1) sum the three digits and run the inverse NTTs of a_c / b_c.
//
// Combined ciphertexts only (nopacking_sum_kernel): the NTT is linear, so the
// columns' digits are summed before they are transformed.
#include "ntt_joint.cuh"
#include "respond_draws.cuh"

namespace ig {

namespace {

template <bool SEEDED>
__global__ void __launch_bounds__(RBLOCK, 1) nopacking_kernel(const __grid_constant__ NoPackingArgs A) {
  extern __shared__ __align__(128) uint32_t smem[];
  uint32_t* SC = smem;                        // [RG][NTT_SCRATCH]
  uint32_t* PB = SC + RG * NTT_SCRATCH;       // [2 r][3 t][2 (a,b)][N] products, slot layout (swizzled)
  uint32_t* SUMB = PB + 12 * N;               // [2 r][2 (a,b)][N] running sum over columns (swizzled)
  int* wsb = reinterpret_cast<int*>(SUMB + 4 * N);  // [3][20]
  const DevParams& P = A.P;
  const int ngroups = A.col_groups;
  const int qi = blockIdx.x / ngroups, cg = blockIdx.x - qi * ngroups;
  const int tid = threadIdx.x, g = tid >> 7, x = tid & 127;
  const int r = g / 3, t = g - 3 * r;
  const int gamma = P.gamma;
  const int cper = (gamma + ngroups - 1) / ngroups;
  const int c0 = cg * cper, c1 = min(gamma, c0 + cper);
  const uint32_t shard = A.shard[qi];
  if (shard >= (uint32_t)A.nshards) {
    if (tid == 0 && cg == 0) A.status[qi] = ERR_INDEX;
    return;  // uniform over the CTA
  }
  const uint16_t* H = A.H + (size_t)shard * gamma * N;
  const uint32_t q = P.r[r].q, qinv = P.r[r].qinv;

  // ---- rows ELL..2ELL-1: a_t (expanded or given), b_t ----
  {
    const int st = tid >> 8, lt = tid & 255;
    uint64_t* cand = reinterpret_cast<uint64_t*>(SC) + st * N;  // 3 x 16 KiB within SC
    uint32_t* a0 = PB + st * 2 * N;                              // 3 x 16 KiB within PB
    uint32_t* a1 = a0 + N;
    if (SEEDED) {
      const bool ok = expand_seeded_row<2>(P, A.seeds + ((size_t)qi * ELL + st) * 32, cand, a0, a1, wsb + 20 * st,
                                           7 + st, lt);
      if (lt == 0) wsb[20 * st + 17] = ok;
    } else {
      const uint64_t* ar = A.arows + ((size_t)qi * ELL + st) * 2 * N;
      for (int j = lt; j < 2 * N; j += SUB) a0[j] = (uint32_t)ar[j];
    }
  }
  __syncthreads();
  // the query's status is written once, by one thread
  if (tid == 0 && cg == 0) A.status[qi] = (!SEEDED || (wsb[17] && wsb[37] && wsb[57])) ? 0 : ERR_EXPAND;
  // group (r,t): NTT(a_t mod q_r), NTT(b_t mod q_r), kept as x * n^-1 * 2^32
  uint32_t ah[16], bh[16];
  {
    const ResidueConsts& C = P.r[r];
#pragma unroll
    for (int j = 0; j < 16; j++) ah[j] = PB[t * 2 * N + r * N + x + 128 * j];
    ntt_fwd<false>(ah, SC + g * NTT_SCRATCH, fwd_tw(C), q, x, 1 + g);
    const uint64_t* brow = A.brows + (((size_t)qi * ELL + t) * 2 + r) * N;
#pragma unroll
    for (int j = 0; j < 16; j++) bh[j] = (uint32_t)__ldg(brow + x + 128 * j);
    ntt_fwd<false>(bh, SC + g * NTT_SCRATCH, fwd_tw(C), q, x, 1 + g);
#pragma unroll
    for (int j = 0; j < 16; j++) {
      ah[j] = mul_shoup(ah[j], C.ninv_mont, C.ninv_mont_p, q);
      bh[j] = mul_shoup(bh[j], C.ninv_mont, C.ninv_mont_p, q);
    }
  }
  __syncthreads();  // PB (row staging) is reused for products

  // group (r,0): sum_c a_c; group (r,1): sum_c b_c (NTT domain, n^-1 folded)
  uint32_t* sumb = SUMB + (r * 2 + (t < 2 ? t : 0)) * N;
  if (t < 2) {
    const uint32_t zero[16] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
    store16(sumb, x, zero);
  }
  uint64_t* outc = A.out_columns + (size_t)qi * gamma * 4 * N;

  for (int c = c0; c < c1; c++) {
    // digit t of Delta * h_c, NTT mod q_r, products with this group's row
    uint32_t v[16];
#pragma unroll
    for (int j = 0; j < 16; j++) {
      const uint64_t xv = P.delta * (uint64_t)__ldg(H + (size_t)c * N + x + 128 * j);
      v[j] = (uint32_t)(xv >> (ZBITS * t)) & ((1u << ZBITS) - 1);
    }
    ntt_fwd<false>(v, SC + g * NTT_SCRATCH, fwd_tw(P.r[r]), q, x, 1 + g);  // [0, 14q)
    {
      const int f = (x >> 1) & 3;
      uint32_t* da = PB + ((r * 3 + t) * 2 + 0) * N + 16 * x;
      uint32_t* db = PB + ((r * 3 + t) * 2 + 1) * N + 16 * x;
#pragma unroll
      for (int r4 = 0; r4 < 4; r4++) {
        uint32_t pa[4], pb[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int j = 4 * r4 + e;
          pa[e] = redc_lazy((uint64_t)v[j] * ah[j], q, qinv);
          pb[e] = redc_lazy((uint64_t)v[j] * bh[j], q, qinv);
        }
        *reinterpret_cast<uint4*>(da + 4 * (r4 ^ f)) = make_uint4(pa[0], pa[1], pa[2], pa[3]);
        *reinterpret_cast<uint4*>(db + 4 * (r4 ^ f)) = make_uint4(pb[0], pb[1], pb[2], pb[3]);
      }
    }
    __syncthreads();
    if (t < 2) {  // (r,0): a_c, (r,1): b_c
      const int f = (x >> 1) & 3;
      const uint32_t* p0 = PB + ((r * 3 + 0) * 2 + t) * N + 16 * x;
      const uint32_t* p1 = PB + ((r * 3 + 1) * 2 + t) * N + 16 * x;
      const uint32_t* p2 = PB + ((r * 3 + 2) * 2 + t) * N + 16 * x;
#pragma unroll
      for (int r4 = 0; r4 < 4; r4++) {
        const int o = 4 * (r4 ^ f);
        uint4* sp = reinterpret_cast<uint4*>(sumb + 16 * x + o);
        const uint4 s4 = *sp;
        uint32_t ss[4] = {s4.x, s4.y, s4.z, s4.w};
        const uint4 a4 = *reinterpret_cast<const uint4*>(p0 + o);
        const uint4 b4 = *reinterpret_cast<const uint4*>(p1 + o);
        const uint4 c4 = *reinterpret_cast<const uint4*>(p2 + o);
        const uint32_t aa[4] = {a4.x, a4.y, a4.z, a4.w}, bb[4] = {b4.x, b4.y, b4.z, b4.w},
                       cc[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int j = 4 * r4 + e;
          uint32_t sm = aa[e] + bb[e] + cc[e];  // < 6q
          sm = min(sm, sm - 4 * q);
          sm = min(sm, sm - 2 * q);
          sm = min(sm, sm - q);
          v[j] = sm;
          const uint32_t acc = ss[e] + sm;
          ss[e] = min(acc, acc - q);
        }
        *sp = make_uint4(ss[0], ss[1], ss[2], ss[3]);
      }
      ntt_inv_noscale(v, SC + g * NTT_SCRATCH, inv_tw(P.r[r]), q, x, 1 + g);
      uint64_t* o = outc + ((size_t)c * 2 + t) * 2 * N + (size_t)r * N;
#pragma unroll
      for (int j = 0; j < 16; j++) o[x + 128 * j] = canon2(v[j], q);
    }
    __syncthreads();
  }
  // combined ciphertext = sum of the column ciphertexts (respond.rs:102-109)
  if (ngroups == 1 && t < 2) {
    uint32_t sv[16];
    load16(sumb, x, sv);
    ntt_inv_noscale(sv, SC + g * NTT_SCRATCH, inv_tw(P.r[r]), q, x, 1 + g);
    uint64_t* o = A.out + (size_t)qi * 4 * N + (size_t)t * 2 * N + (size_t)r * N;
#pragma unroll
    for (int j = 0; j < 16; j++) o[x + 128 * j] = canon2(sv[j], q);
  }
}

// The combined ciphertext of one query: sum_c NTT(D_{c,t}) = NTT(sum_c
// D_{c,t} mod q_r), so per residue three digit sums, three a rows and three b
// rows are transformed and two sums of products transformed back.
//
// 512 threads, group (r, s) of 128 owning residue r's side s, and a producer
// warp.  The a groups (s = 0) expand the rows while the b groups sum and
// transform the digits; then each side transforms its rows, multiplies them
// with the digits' transforms (thread for thread in shared memory) and writes
// its half of the response.  Rows may lie in page-locked host memory (the
// producer copies them in small chunks) and the response may be written there.
//
// What bounds it: for rows and responses in host memory the link (measured 210
// GB/s of reads and 200 GB/s of writes, 82 us for the 12.6 and 8.4 MB of 128
// queries together: the kernel takes 93 us); the transforms and the expansion
// alone take 36 us.  128 queries take 111 us per host call, 133 us with the rows
// read where they are used, 200 us copied through device buffers.
struct SumSmem {
  static constexpr int AH = 0;                   // [ELL][2][N] rows' a, coefficients; exchange buffers in turn
  static constexpr int XD = AH + ELL * 2 * N;    // [2 r][ELL][N] the digit sums' exchange buffers, then transforms
  static constexpr int DIG = XD + 2 * ELL * N;   // [ELL][N] digit sums; then XB [2 r][N], the b rows' exchange buffers
  static constexpr int ROWS = DIG + ELL * N;     // [ELL][2][N] u64, the staged b rows
  static constexpr int WS = ROWS + 2 * ELL * 2 * N;  // expansion's workspace, [24] chunks issued
  static constexpr int SEED = WS + 32;           // [ELL * 8] staged seeds
  static constexpr int BARS = SEED + 24;         // [ELL][ROW_CHUNKS] mbarriers
  static constexpr int TOTAL = BARS + 2 * ELL * 8;
};
constexpr int ST = 2 * QT;      // threads of the two sides
constexpr int CHUNK = 512;      // u64 words of a staged chunk (4 KiB)
constexpr int ROW_CHUNKS = 2 * N / CHUNK;
static_assert(ROW_CHUNKS == 8, "mbarriers of SumSmem");

template <bool SEEDED>
__global__ void __launch_bounds__(ST + 32, 1) nopacking_sum_kernel(const __grid_constant__ NoPackingArgs A) {
  using L = SumSmem;
  extern __shared__ __align__(128) uint32_t smem[];
  uint32_t* AH = smem + L::AH;
  uint32_t* DIG = smem + L::DIG;
  uint64_t* rows = reinterpret_cast<uint64_t*>(smem + L::ROWS);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::BARS);
  int* ws = reinterpret_cast<int*>(smem + L::WS);
  const DevParams& P = A.P;
  const int qi = blockIdx.x;
  const int tid = threadIdx.x, s = tid >> 8, r = (tid >> 7) & 1, x = tid & 127, gamma = P.gamma;
  const int bar = 1 + (tid >> 7);  // this group's barrier
  const uint32_t shard = A.shard[qi];
  if (shard >= (uint32_t)A.nshards) {
    if (tid == 0) A.status[qi] = ERR_INDEX;
    return;  // uniform over the CTA
  }
  const uint16_t* H = A.H + (size_t)shard * gamma * N;
  if (tid == ST)
    for (int k = 0; k < ELL * ROW_CHUNKS; k++) mbar_init(bars + k);
  if (tid < ELL) ws[20 + tid] = 1;
  uint8_t* const seeds = reinterpret_cast<uint8_t*>(smem + L::SEED);
  if (SEEDED && tid < ELL * 32) seeds[tid] = A.seeds[(size_t)qi * ELL * 32 + tid];
  __syncthreads();
  const ResidueConsts& C = P.r[r];
  const uint32_t q = C.q, qinv = C.qinv;
  const uint32_t xd = jx_addr(smem + L::XD + r * ELL * N), xb = jx_addr(smem + L::DIG + r * N);
  uint32_t v[1][16], acc[1][16];
#pragma unroll
  for (int j = 0; j < 16; j++) acc[0][j] = 0;
  static_assert(JFWD_OUT * JFWD_OUT <= 3 * 16 * 64 * 64, "q < 2^28: reduced products above -3 q");
  // acc += v times the digit sum t's transform: |v|, |d| < 6.5 q, so products
  // are below 42.3 q^2, reduced below 3.7 q and made positive; acc below 8 q
  auto add_product = [&](int t) {
    uint32_t d[1][16];
    const uint32_t sd[1] = {xd + 4 * N * t};
    jx_load_ru<1>(d, sd, x);
#pragma unroll
    for (int j = 0; j < 16; j++)
      acc[0][j] = csub(acc[0][j] + redc_wide(smul(v[0][j], d[0][j]), q, qinv) + 3 * q, 8 * q);
  };
  bool arrived = true;
  if (s == 2) {
    // the producer: two chunks in flight.  A device read (twiddles, columns)
    // queued behind a long host read waits for all of it: 96 KiB per SM at
    // once from 128 SMs held the other groups up for 50 us.
    if (tid == ST) {
      const uint64_t* src = A.brows + (size_t)qi * A.brow_stride;
      int k = 0;
      for (; k < ELL * ROW_CHUNKS; k++) {
        if (k >= 2) arrived = mbar_wait(bars + k - 2, 0, A.row_wait_iters);
        if (!arrived) break;
        mbar_expect_tx(bars + k, sizeof(uint64_t) * CHUNK);
        bulk_g2s(rows + (size_t)k * CHUNK, src + (size_t)k * CHUNK, sizeof(uint64_t) * CHUNK, bars + k);
      }
      ws[24] = k;
    }
  } else if (s == 0) {
    if (SEEDED) {
      expand_rows<2>(P, seeds, AH, ws);
    } else {
      const uint64_t* ar = A.arows + (size_t)qi * ELL * 2 * N;
#pragma unroll 4
      for (int j = tid; j < ELL * 2 * N; j += QT) AH[j] = (uint32_t)__ldg(ar + j);
    }
    named_sync(EXPAND_BAR, QT);
    named_arrive(7, ST);  // the b groups may look at ws
    const bool redo = SEEDED && !(ws[20] && ws[21] && ws[22]);  // uniform
    if (redo) {
      named_sync(8, ST);  // the b groups are done with the staged rows: room for candidates
      bool good = true;
#pragma unroll 1
      for (int t = 0; t < ELL; t++)
        if (!ws[20 + t]) good &= expand_row_general<2>(P, seeds + 32 * t, rows, AH + t * 2 * N, ws);
      named_sync(EXPAND_BAR, QT);
      if (!good) arrived = false;
    }
    named_sync(5 + r, QT);  // the digits' transforms of this residue are there
#pragma unroll 1
    for (int t = 0; t < ELL; t++) {
      uint32_t* row = AH + (t * 2 + r) * N;
#pragma unroll
      for (int j = 0; j < 16; j++) v[0][j] = row[x + 128 * j];
      group_sync(bar);  // the row is read: its words become its exchange buffer
      const uint32_t sc[1] = {jx_addr(row)};
      jntt_fwd<1, JB_CANON>(v, sc, sfwd_tw(C), q, x, bar);
      add_product(t);
    }
  } else {
    // digit sums: below 2^24 (the transform takes any such sum: for q near
    // 2^28 it is below q / 16, and for smaller q nothing comes near 32 bits)
    const uint32_t* h2 = reinterpret_cast<const uint32_t*>(H) + (tid - QT);
#pragma unroll 1
    for (int m = 0; m < N / 2 / QT; m++) {
      uint32_t sum[2][ELL] = {};
#pragma unroll
      for (int c = 0; c < MAX_GAMMA; c++) {
        if (c >= gamma) continue;
        const uint32_t hw = __ldg(h2 + (size_t)c * (N / 2) + QT * m);
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const uint64_t xv = P.delta * (uint64_t)((hw >> (16 * e)) & 0xFFFFu);
          sum[e][0] += (uint32_t)xv & 0xFFFFFu;
          sum[e][1] += (uint32_t)(xv >> 20) & 0xFFFFFu;
          sum[e][2] += (uint32_t)(xv >> 40);
        }
      }
#pragma unroll
      for (int t = 0; t < ELL; t++)
        *reinterpret_cast<uint2*>(DIG + t * N + 2 * (tid - QT + QT * m)) = make_uint2(sum[0][t], sum[1][t]);
    }
    named_sync(9, QT);
    {
      uint32_t d[ELL][16];
#pragma unroll
      for (int t = 0; t < ELL; t++)
#pragma unroll
        for (int j = 0; j < 16; j++) d[t][j] = DIG[t * N + x + 128 * j];
      named_sync(9, QT);  // DIG is read: its words become the b rows' exchange buffers
      const uint32_t sc[ELL] = {xd, xd + 4 * N, xd + 8 * N};
      jntt_fwd<ELL, JB_CANON>(d, sc, sfwd_tw(C), q, x, bar);
      jx_store_ru<ELL>(d, sc, x);
      named_arrive(5 + r, QT);
    }
#pragma unroll 1
    for (int t = 0; t < ELL; t++) {
      for (int k = 0; k < ROW_CHUNKS; k++)
        if (arrived) arrived = mbar_wait(bars + t * ROW_CHUNKS + k, 0, A.row_wait_iters);
      const uint32_t* row = reinterpret_cast<const uint32_t*>(rows + ((size_t)t * 2 + r) * N);
#pragma unroll
      for (int j = 0; j < 16; j++) v[0][j] = row[2 * (x + 128 * j)];
      if (t) group_sync(bar);  // the last transform's reads are done
      const uint32_t sc[1] = {xb};
      jntt_fwd<1, JB_CANON>(v, sc, sfwd_tw(C), q, x, bar);
      add_product(t);
    }
    named_sync(7, ST);
    if (SEEDED && !(ws[20] && ws[21] && ws[22])) named_arrive(8, ST);
  }
  if (s < 2) {
    // this side's half of the response
#pragma unroll
    for (int j = 0; j < 16; j++) acc[0][j] = csub(acc[0][j], 4 * q);
    {
      const uint32_t sc[1] = {s ? xb : jx_addr(AH + ((ELL - 1) * 2 + r) * N)};
      jntt_inv_scaled<1>(acc, sc, sfwd_tw(C), make_uint2(C.ninv_mont, C.ninv_mont_p), C.ninv_mont_w, q, x, bar);
    }
    uint64_t* o = A.out + (size_t)qi * 4 * N + (size_t)(2 * s + r) * N + x;
#pragma unroll
    for (int j = 0; j < 16; j++) o[128 * j] = acc[0][j];
  }
  // rows that did not arrive within the wait's bound end the query with a
  // status, after another bounded wait for the copies still in flight
  const int late = __syncthreads_or(s != 0 && !arrived), bad = __syncthreads_or(s == 0 && !arrived);
  if (late) {
    bool here = true;  // (the chunks after those issued never come)
    for (int k = 0; k < ws[24] && here; k++) here = mbar_wait(bars + k, 0, STAGE_DRAIN_ITERS);
    const int lost = __syncthreads_or(!here);
    if (tid == 0) A.status[qi] = lost ? ERR_STAGE_LOST : ERR_STAGE;
  } else if (tid == 0) {
    A.status[qi] = bad ? ERR_EXPAND : 0;
  }
}

// Combined ciphertexts of split queries: out[q] = sum_c columns[q][c] mod q_r
// (respond.rs:102-109), in the coefficient domain (the sum commutes with the
// inverse NTT, so this equals the one-CTA path's bits).
__global__ void column_sum_kernel(const DevParams P, int nq, int gamma, const uint64_t* __restrict__ cols,
                                  uint64_t* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;  // over nq * 4N words
  if (i >= (size_t)nq * 4 * N) return;
  const size_t qi = i / (4 * N), w = i - qi * 4 * N;  // w: part (a, b) x residue x coefficient
  const uint32_t q = P.r[(w / N) & 1].q;
  const uint64_t* src = cols + qi * (size_t)gamma * 4 * N + w;
  uint32_t s = 0;
  for (int c = 0; c < gamma; c++) {
    const uint32_t v = s + (uint32_t)src[(size_t)c * 4 * N];
    s = min(v, v - q);
  }
  out[i] = s;
}

}  // namespace

size_t nopacking_smem_bytes() { return sizeof(uint32_t) * ((size_t)RG * NTT_SCRATCH + 16 * N + 64); }

template <bool SEEDED>
static cudaError_t launch_np(const NoPackingArgs& a, cudaStream_t st) {
  if (!a.out_columns) {
    nopacking_sum_kernel<SEEDED><<<a.nq, ST + 32, sizeof(uint32_t) * SumSmem::TOTAL, st>>>(a);
    return cudaGetLastError();
  }
  nopacking_kernel<SEEDED><<<a.nq * a.col_groups, RBLOCK, nopacking_smem_bytes(), st>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && a.col_groups > 1) {
    const size_t words = (size_t)a.nq * 4 * N;
    column_sum_kernel<<<(unsigned)((words + 255) / 256), 256, 0, st>>>(a.P, a.nq, a.P.gamma, a.out_columns, a.out);
    e = cudaGetLastError();
  }
  return e;
}

cudaError_t prepare_nopacking_kernels() {
  const int smem = (int)nopacking_smem_bytes();
  cudaError_t e = cudaFuncSetAttribute(nopacking_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(nopacking_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  const int sum = (int)sizeof(uint32_t) * SumSmem::TOTAL;
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(nopacking_sum_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sum);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(nopacking_sum_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sum);
  return e;
}

cudaError_t launch_nopacking(const NoPackingArgs& a, bool seeded, cudaStream_t st) {
  if (a.nq <= 0) return cudaSuccess;
  if (a.col_groups < 1 || (a.col_groups > 1 && !a.out_columns)) return cudaErrorInvalidValue;
  return seeded ? launch_np<true>(a, st) : launch_np<false>(a, st);
}

}  // namespace ig
