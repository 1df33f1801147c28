// respond_pair.cu -- the Respond kernel for small batches: a cluster of two
// CTAs of 512 threads per query, CTA r computing CRT residue r.
//
// It returns exactly what respond.cu's one-CTA kernel returns (the packed
// ciphertext of respond_seeded_inspiring / respond_inspiring,
// src/pir/respond.rs:284-398, through packing_online,
// src/inspiring/inspiring2.rs:1185-1222), from the same regrouped dataflow
// and the same tables; only the placement differs, for the latency of one
// query.  Of the recursion step (inspiring2.rs:984-1008) only the gadget
// decomposition needs both residues, so each CTA runs one residue's chain and
// the two exchange the 2048 coefficients of INTT(R_{i+1}) once per step
// through distributed shared memory (st.async on the receiver's mbarrier).
//
// Inside a CTA, thread t of both teams of 256 owns slots 8t .. 8t+7, and the
// teams share a step's work so that the chain INTT -> digits -> NTT is as
// short as one team can make it:
//   team 0: [A] INTT(R_{i+1}), coefficients to team 1 and to the peer CTA;
//           [C] NTT(d0); [D] its products, R_i from both teams' sums;
//   team 1: [A] sum_t E A_t + R_{i+1} w'2, b += R_{i+1} y'2;
//           [C] NTT(d1); [D] its products, its sum to team 0.
// Both compute their digit of the composite coefficients themselves ([B]).
// Besides the transforms' own, a step has the wait for the peer, one barrier
// of all threads (team 1's sum) and two that team 1 alone waits for (the
// coefficients, R_i).
//
// What bounds it: latency; a CTA's 316 K warp instructions issue at 1.7 per cycle
// and SM.  A batch of 8 takes 86.5 us, 111 us with 256 threads per CTA and 16
// values a thread (a lone warp issues an instruction every seven cycles, so
// halving each thread's chain pays).
#include "ntt_team.cuh"
#include "respond_draws.cuh"

namespace ig {

namespace {

constexpr int PT = 2 * TEAM;  // threads per CTA

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

// Address of this CTA's shared variable `p` in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_smem(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}

__device__ __forceinline__ void st_peer(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// Every thread of both CTAs: this CTA's earlier writes (local and remote)
// are visible to the peer and the peer's to this CTA afterwards.
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// 16 bytes to the peer's shared memory, completing on its mbarrier.
__device__ __forceinline__ void st_async4(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                   addr),
               "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar)
               : "memory");
}

// Wait, with an iteration bound, for phase `parity` of `bar` and the peer's
// writes that completed it; false when the bound ran out.
__device__ __forceinline__ bool mbar_wait_peer(uint64_t* bar, uint32_t parity, uint32_t limit) {
  for (uint32_t it = 0; it < limit; it++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, "
        "0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Thread 0, which stopped waiting for the peer's coefficients at step `late`:
// waits, with an iteration bound, until those of that and all later steps have
// come.  The mbarriers' phases of steps late and late - 1 are armed; the steps
// after them, which it has not armed, are one more phase each.  What came for
// these before they are announced here counts towards whichever phase is
// current, so the phases' order, not their split by step, is what is waited
// for.
__device__ __noinline__ bool drain_peer(uint64_t* cbar, int late, int gamma) {
  for (int s = late; s >= 0 && s >= late - 1; s--) {
    uint64_t* bar = cbar + (s & 1);
    uint32_t phase = ((gamma - 2 - s) >> 1) & 1;
    for (int more = s >> 1;; more = 0, phase ^= 1) {
      if (!mbar_wait_peer(bar, phase, STAGE_WAIT_ITERS_DEFAULT)) return false;
      if (!more) break;
      mbar_expect_tx(bar, 4 * N * more);
    }
  }
  return true;
}

// Some of the peer's coefficients did not come within the wait's bound (late: in
// thread 0, the caller): the response is wrong and says so.  The CTA's memory is
// not freed while they may still come; if another bounded wait for them runs out
// too, ERR_PEER_LOST tells the host to drop every result of this launch.  (Where
// thread 0 saw every step arrive, nothing is in flight.)  CTA 0 writes the status.
__device__ __noinline__ int peer_missing(uint64_t* cbar, int* misc, int gamma, bool late) {
  const int outcome = late && !drain_peer(cbar, misc[3] - 1, gamma) ? ERR_PEER_LOST : ERR_PEER;
  if (cluster_rank() == 1) st_peer(peer_smem(misc + 6, 0), (uint32_t)outcome);
  return outcome;
}

// Shared-memory layout in u32 words.
struct PairSmem {
  static constexpr int AH = 0;              // [ELL][16 rows h][128] row transforms of the a-side residue (ah_word)
  static constexpr int X = AH + ELL * N;    // [2][N] exchange buffer of each team
  static constexpr int RC = X + 2 * N;      // [2 parity][N] the peer's coefficients, thread by thread
  static constexpr int OC = RC + 2 * N;     // [N] this residue's, for team 1
  static constexpr int S1 = OC + N;         // [N] team 1's sums, for team 0
  static constexpr int RN = S1 + N;         // [N] R_i, for team 1
  static constexpr int ROWS = X;            // until the b side is done: b rows (u64 [ELL][N]) of a staged query
  static constexpr int GEN = X;             // general expansion: 2048 candidates (u64), then both residues [2][N]
  static constexpr int WS = RN + N;         // [2 teams][2][8] scan totals
  static constexpr int TOT = WS + 32;       // [4] values drawn per row
  static constexpr int OK = TOT + 4;        // [4] rows complete
  static constexpr int BP = OK + 4;         // [16] the b side
  static constexpr int SEED = BP + 16;      // [ELL * 8] staged seeds (serving loop)
  static constexpr int MISC = SEED + 24;    // [3] residue 1's stream positions, [1] the last step whose wait thread 0
                                            // ended, [2] flags, [2] drain results by rank, or CTA 1's outcome in [6]
  static constexpr int BARS = MISC + 8;     // mbarriers: the staged rows', then the peer's coefficients' [2 parity]
  static constexpr int TOTAL = BARS + 8;
};
static_assert(2 * ELL * N <= 6 * N, "the staged rows leave RN free");
static_assert(PairSmem::X * 4 % 128 == 0 && PairSmem::BARS % 2 == 0, "alignment of exchange buffers and mbarriers");

// A row transform's word (h, x): neighbouring lanes read rows h and h + 1 at
// the same 16 runs, so odd rows are stored 16 banks away.
__device__ __forceinline__ uint32_t ah_off(uint32_t h, uint32_t x) { return (h << 9) | ((x << 2) ^ ((h & 1u) << 6)); }

constexpr uint32_t NO_START = 0xFFFFFFFFu;

// The b side of this CTA's residue (see respond.cu's column_b0): b0_c =
// -sum_i d_c[i] v[i], v[0] = q - b[0], v[i] = b[N - i]; pitch: u64 words
// between the rows' polynomials.
__device__ __forceinline__ void column_b0_residue(const DevParams& P, const uint16_t* __restrict__ H,
                                                  const uint64_t* rows, size_t pitch, uint32_t q, uint64_t* red,
                                                  uint32_t* bpoly) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, gamma = P.gamma;
  const uint32_t* h2 = reinterpret_cast<const uint32_t*>(H) + tid;
  uint64_t acc[MAX_GAMMA];
#pragma unroll
  for (int c = 0; c < MAX_GAMMA; c++) acc[c] = 0;
#pragma unroll 1
  for (int m = 0; m < N / 2 / PT; m++) {
    uint32_t hw[MAX_GAMMA], bv[2][ELL];
#pragma unroll
    for (int c = 0; c < MAX_GAMMA; c++) hw[c] = c < gamma ? __ldg(h2 + (size_t)c * (N / 2) + PT * m) : 0u;
    const int i0 = 2 * (tid + PT * m);
#pragma unroll
    for (int t = 0; t < ELL; t++) {
      bv[0][t] = (uint32_t)rows[t * pitch + (i0 ? N - i0 : 0)];
      bv[1][t] = (uint32_t)rows[t * pitch + (N - i0 - 1)];
      if (i0 == 0) bv[0][t] = q - bv[0][t];
    }
#pragma unroll
    for (int c = 0; c < MAX_GAMMA; c++) {
      if (c >= gamma) continue;
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const uint64_t xv = P.delta * (uint64_t)((hw[c] >> (16 * e)) & 0xFFFFu);
        const uint32_t d0 = (uint32_t)xv & 0xFFFFFu, d1 = (uint32_t)(xv >> 20) & 0xFFFFFu, d2 = (uint32_t)(xv >> 40);
        acc[c] += (uint64_t)d0 * bv[e][0] + (uint64_t)d1 * bv[e][1] + (uint64_t)d2 * bv[e][2];
      }
    }
  }
  // lanes l and l + 16 end with the warp's sum of column l
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < o; k++) {
      const uint64_t send = up ? acc[k] : acc[k + o], keep = up ? acc[k + o] : acc[k];
      acc[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 16);
  if (lane < 16) red[warp * 16 + lane] = acc[0];
  __syncthreads();
  if (tid < 16) {
    uint64_t s = 0;
#pragma unroll
    for (int w = 0; w < PT / 32; w++) s += red[w * 16 + tid];
    const uint32_t v = (uint32_t)(s % q);
    bpoly[tid] = v ? q - v : 0;
  }
  __syncthreads();
}

template <int MODE, bool SEEDED, bool QDB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PT, 1)
    respond_pair_kernel(const __grid_constant__ RespondArgs A) {
  using L = PairSmem;
  extern __shared__ __align__(128) uint32_t smem[];
  const uint32_t r = cluster_rank(), peer = r ^ 1u;  // this CTA's residue
  const int qi = blockIdx.x >> 1;
  const DevParams& P = A.P;
  const int tid = threadIdx.x, team = tid >> 8, t = tid & 255, lane = tid & 31, warp = tid >> 5;
  const int x = t >> 1, half = t & 1;  // slots 8 t .. 8 t + 7: half of run x
  const int gamma = P.gamma;
  int* ws = reinterpret_cast<int*>(smem + L::WS) + 16 * team;
  int* tot = reinterpret_cast<int*>(smem + L::TOT);
  int* ok = reinterpret_cast<int*>(smem + L::OK);
  int* misc = reinterpret_cast<int*>(smem + L::MISC);
  uint32_t* bpoly = smem + L::BP;

  const QueryDesc* D = QDB ? A.qdesc + qi : nullptr;
  const uint32_t shard = QDB ? D->shard : A.shard[qi];
  const int32_t cid = QDB ? D->client : A.client[qi];
  const int nshards = QDB ? D->db.nshards : A.nshards;
  auto status_ptr = [&]() -> int32_t* { return QDB ? reload_ptr(&D->status) : A.status + qi; };
  // both CTAs read the same fields: every return here is uniform over the cluster
  if (shard >= (uint32_t)nshards || cid < 0 || cid >= A.nclients || A.yhat_table[cid] == nullptr) {
    if (r == 0 && tid == 0) *status_ptr() = ERR_INDEX;
    pdl_wait();
    return;
  }

  // residue of the a side and the query-only terms: this CTA's, or residue 0
  // for both CTAs in compat mode (residue 1 is then rebuilt from it)
  const int sres = MODE == MODE_CRT_FIXED ? (int)r : 0;
  const bool conv1 = MODE == MODE_COMPAT && r == 1;
  const uint16_t* H = (QDB ? D->db.H : A.H) + (size_t)shard * gamma * N;
  const uint32_t* E = (QDB ? D->db.E : A.E) + ((size_t)shard * 2 + sres) * ELL * gamma * N;
  const uintptr_t ytag = reinterpret_cast<uintptr_t>(A.yhat_table[cid]);
  const bool ybody = (ytag & 1) != 0;
  const uint32_t* Y = reinterpret_cast<const uint32_t*>(ytag & ~(uintptr_t)1);
  const ResidueConsts& C = P.r[r];
  const uint32_t q = C.q, qinv = C.qinv, qo = P.r[peer].q;
  const uint64_t* brows = (QDB ? D->brows : A.brows + (size_t)qi * ELL * 2 * N) + (size_t)r * N;

  uint32_t* AH = smem + L::AH;
  uint64_t* rows = reinterpret_cast<uint64_t*>(smem + L::ROWS);
  uint64_t* rbar = reinterpret_cast<uint64_t*>(smem + L::BARS);
  uint64_t* cbar = rbar + 1;  // [2] by step parity
  if (tid == 0) {
    for (int k = 0; k < 3; k++) mbar_init(rbar + k);
    mbar_expect_tx(cbar, 4 * N);
    mbar_expect_tx(cbar + 1, 4 * N);
    misc[3] = gamma - 1;
    misc[6] = 0;
    prefetch_l2(H, sizeof(uint16_t) * (size_t)gamma * N);
    // the contracted shard's blocks of the first three steps (the rest are
    // prefetched two steps ahead of their use in the recursion)
    const int i0 = gamma >= 3 ? gamma - 3 : 0;
    prefetch_l2(E + (size_t)i0 * ELL * N, sizeof(uint32_t) * (size_t)(gamma - i0) * ELL * N);
    if (gamma > 1) prefetch_l2(Y, sizeof(uint32_t) * (size_t)(ybody ? 1 : gamma - 1) * ELL * 2 * N);
  }
  const uint8_t* seeds = nullptr;
  if (SEEDED) seeds = QDB ? reinterpret_cast<const uint8_t*>(smem + L::SEED) : A.seeds + (size_t)qi * ELL * 32;
  if (QDB && SEEDED && tid < ELL * 32) reinterpret_cast<uint8_t*>(smem + L::SEED)[tid] = D->seeds[tid];
  __syncthreads();  // the mbarriers are initialised, the seeds staged
  // the peer's shared memory may be written only once it has started
  cluster_arrive();
  if (QDB && tid == 0) {
    // this residue's b rows (48 KiB) while the rows are expanded
    mbar_expect_tx(rbar, (uint32_t)(sizeof(uint64_t) * ELL * N));
#pragma unroll
    for (int k = 0; k < ELL; k++)
      bulk_g2s(rows + (size_t)k * N, brows + (size_t)2 * k * N, sizeof(uint64_t) * N, rbar);
  }

  // ---- rows ELL..2ELL-1, residue sres, coefficients into AH [row][N]
  //      (expand_rows in respond.cu; rows 0 and 2 by team 0, 1 by team 1):
  //      draws 0 .. 2047 of a row go to residue 0, a warp finds the few it
  //      still misses among the next 256; residue 1's CTA meanwhile draws from
  //      2048 on and learns where to start ----
  if (SEEDED) {
    const uint32_t sq = P.r[sres].q, sz = (uint32_t)(P.r[sres].zone >> 32);
    if (sres == 0) {
#pragma unroll 1
      for (int k = team; k < ELL; k += 2) {
        uint32_t key[8], w[16], val[8];
        load_key(seeds + 32 * k, key);
        chacha20_block(key, t, P.one, w);
        const unsigned mask = draw8(w, sq, sz, val);
        int total;
        const int p = scan_256(__popc(mask), ws + 8 * (k >> 1), total, 1 + team);
        put_draws(AH + k * N, p, mask, val);
        if (t == 0) tot[k] = total;
      }
      // the next 256 draws, by warps of team 1 while team 0 has the third row (a
      // lone warp's ChaCha20 off the path of both CTAs: 1.6 us of a launch)
      const int k = warp - TEAM / 32;
      const bool tail = k >= 0 && k < ELL;
      uint32_t val[8];
      unsigned mask = 0;
      if (tail) {
        uint32_t key[8], w[16];
        load_key(seeds + 32 * k, key);
        chacha20_block(key, 256 + lane, P.one, w);
        mask = draw8(w, sq, sz, val);
      }
      __syncthreads();
      if (MODE == MODE_CRT_FIXED) cluster_wait();
      if (tail) {
        const int have = tot[k];
        uint32_t end = 0;  // draws past the first 2048 that residue 0 takes
        if (have < N) {    // uniform over the warp
          int all;
          const int p = have + scan_warp(__popc(mask), all);
          put_draws(AH + k * N, p, mask, val);
          int pp = p;
#pragma unroll
          for (int e = 0; e < 8; e++)
            if ((mask >> e) & 1u) {
              if (pp == N - 1) end = 8 * lane + e + 1;
              pp++;
            }
          end = __reduce_max_sync(0xffffffffu, end);
          if (end == 0) end = NO_START;
        }
        if (lane == 0) {
          ok[k] = end != NO_START;
          if (MODE == MODE_CRT_FIXED) st_peer(peer_smem(misc + k, peer), end);
        }
      }
      if (MODE == MODE_CRT_FIXED) cluster_sync_all();
    } else {
      uint32_t val[2][8];
      unsigned mask[2] = {0, 0};
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int k = team + 2 * u;
        if (k >= ELL) continue;
        uint32_t key[8], w[16];
        load_key(seeds + 32 * k, key);
        chacha20_block(key, 256 + t, P.one, w);
        mask[u] = draw8(w, sq, sz, val[u]);
      }
      // the last values, one warp per row, from the blocks after these (as above)
      const int k = warp - TEAM / 32;
      const bool tail = k >= 0 && k < ELL;
      uint32_t v8[8];
      unsigned m = 0;
      if (tail) {
        uint32_t key[8], w[16];
        load_key(seeds + 32 * k, key);
        chacha20_block(key, 512 + lane, P.one, w);
        m = draw8(w, sq, sz, v8);
      }
      cluster_wait();
      cluster_sync_all();
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int k = team + 2 * u;
        if (k >= ELL) continue;
        const uint32_t start = (uint32_t)misc[k];
        const int skip = (int)(start == NO_START ? 0u : start) - 8 * t;  // leading draws of this thread to skip
        if (skip > 0) mask[u] &= skip >= 8 ? 0u : ~((1u << skip) - 1u);
        int total;
        const int p = scan_256(__popc(mask[u]), ws + 8 * u, total, 1 + team);
        put_draws(AH + k * N, p, mask[u], val[u]);
        if (t == 0) tot[k] = total;
      }
      __syncthreads();
      if (tail) {
        int all;
        const int p = tot[k] + scan_warp(__popc(m), all);
        put_draws(AH + k * N, p, m, v8);
        if (lane == 0) ok[k] = (uint32_t)misc[k] != NO_START && tot[k] + all >= N;
      }
    }
    if (MODE != MODE_CRT_FIXED) cluster_wait();
  } else {
    const uint64_t* ar = A.arows + (size_t)qi * ELL * 2 * N + (size_t)sres * N;
#pragma unroll
    for (int j = tid; j < ELL * N; j += PT) AH[j] = (uint32_t)__ldg(ar + (size_t)(j >> LOGN) * 2 * N + (j & (N - 1)));
    cluster_wait();
  }

  // the client's keys, read from the recursion on, may be the last launch's work
  pdl_wait();

  // ---- the b side ----
  int missing = 0;
  if (QDB) {
    missing = __syncthreads_or(!mbar_wait(rbar, 0, A.stage_wait_iters));
    if (!missing) column_b0_residue(P, H, rows, N, q, reinterpret_cast<uint64_t*>(smem + L::RN), bpoly);
  } else {
    column_b0_residue(P, H, brows, 2 * N, q, reinterpret_cast<uint64_t*>(smem + L::RN), bpoly);
  }

  // ---- rows that the fast expansion left to the general one (needs the
  //      step buffers, so only once the staged rows are done with) ----
  bool good = true;
  if (SEEDED && !missing) {
#pragma unroll 1
    for (int k = 0; k < ELL; k++)
      if (!ok[k]) {  // uniform; ordered by the b side's barriers
        uint32_t* both = smem + L::GEN + 2 * N;
        uint64_t* cand = reinterpret_cast<uint64_t*>(smem + L::GEN);
        if (team == 0) {
          good &= MODE == MODE_CRT_FIXED ? expand_row_general<2>(P, seeds + 32 * k, cand, both, ws)
                                         : expand_row_general<1>(P, seeds + 32 * k, cand, both, ws);
        }
        __syncthreads();
        for (int j = tid; j < N; j += PT) AH[k * N + j] = both[sres * N + j];
        __syncthreads();
      }
  }

  // ---- the rows' arrival and the expansion, agreed over the cluster ----
  if (tid == 0) {
    const int fl = (missing ? 1 : 0) | (good ? 0 : 2);
    misc[4 + r] = fl;
    st_peer(peer_smem(misc + 4 + r, peer), (uint32_t)fl);
  }
  cluster_sync_all();
  const int flags = misc[4] | misc[5];
  if (QDB && (flags & 1)) {
    // As in the one-CTA kernel: no CTA exits while its own bulk copies can
    // still land; the drain results are agreed before the status is written.
    const int lost = __syncthreads_or(!mbar_wait(rbar, 0, STAGE_DRAIN_ITERS));
    if (tid == 0) {
      misc[6 + r] = lost;
      st_peer(peer_smem(misc + 6 + r, peer), (uint32_t)lost);
    }
    cluster_sync_all();
    if (r == 0 && tid == 0) *status_ptr() = (misc[6] | misc[7]) ? ERR_STAGE_LOST : ERR_STAGE;
    return;  // uniform over the cluster
  }
  if (r == 0 && tid == 0) *status_ptr() = (flags & 2) ? ERR_EXPAND : 0;

  const uint32_t base = jx_addr(smem);
  const uint32_t xb = base + 4 * (L::X + N * team), s1b = base + 4 * L::S1, rnb = base + 4 * L::RN,
                 ocb = base + 4 * L::OC, rcb = base + 4 * L::RC;
  // ---- row transforms into rows h of AH: team 0 rows 0 and 2 (in two
  //      buffers: a transform ends with reads that another warp's next first
  //      writes could overtake), team 1 row 1 ----
  {
    const ResidueConsts& Cs = P.r[sres];
#pragma unroll 1
    for (int k = team; k < ELL; k += 2) {
      uint32_t v[8];
#pragma unroll
      for (int j = 0; j < 8; j++) v[j] = AH[k * N + t + TEAM * j];
      jt_fwd<JB_CANON>(v, k == 2 ? s1b : xb, sfwd_tw(Cs), Cs.q, t, 1 + team);
#pragma unroll
      for (int j = 0; j < 8; j++)
        jx_at(base + 4 * (L::AH + k * N) + ah_off((h_of(j) | (uint32_t)half), x)) = jcanon_fwd(v[j], Cs.q);
    }
    __syncthreads();
  }

  const uint32_t ahb = base + 4 * L::AH;
  // this thread's slots are quads 2 half, 2 half + 1 of run x, rows h_of(j) + half
  const uint32_t* Ex = E + 1024 * half + 4 * x;
  const uint32_t* Wx = A.what + r * N + 1024 * half + 4 * x;
  const uint32_t* Yx = Y + r * N + x;
  // sum_t E[i,t][s] A_t[tau_i(s)] for this thread's slots
  auto query_only = [&](int i, uint32_t rot, uint64_t (&T)[8]) {
    const uint32_t* e = Ex + (size_t)i * ELL * N;
    uint4 ev[6];
#pragma unroll
    for (int k = 0; k < 6; k++) ev[k] = ld_stream(e + (k >> 1) * N + 512 * (k & 1));
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const uint32_t ar = ahb + ah_off((h_of(j) + half + rot) & 15u, x);
      T[j] = (uint64_t)u4e(ev[j >> 2], j & 3) * jx_at(ar) + (uint64_t)u4e(ev[2 + (j >> 2)], j & 3) * jx_at(ar + 4 * N) +
             (uint64_t)u4e(ev[4 + (j >> 2)], j & 3) * jx_at(ar + 8 * N);
    }
  };
  // compat mode, residue 1: rebuilt from the residue-0 value as the crate's
  // apply_automorphism_ntt does
  auto converted = [&](uint64_t T) -> uint32_t {
    return compat_residue1_ninv(P, redc(T, P.r[0].q, P.r[0].qinv));
  };
  uint32_t R[8], acc[8];  // both teams: R_{i+1}; each its part of the b accumulator
  {
    uint64_t T[8];
    query_only(gamma - 1, rot_rows(gamma, gamma - 1, x), T);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      R[j] = conv1 ? converted(T[j]) : redc_wide(T[j], q, qinv);
      acc[j] = 0;
    }
  }

  bool arrived = true;  // every wait for the peer's coefficients so far
#pragma unroll 1
  for (int i = gamma - 2; i >= 0; i--) {
    const int par = i & 1;
    const uint32_t rc = rcb + 4 * N * par;
    const uint32_t rot = rot_rows(gamma, i, x);
    const uint32_t* wi = Wx + ((size_t)i * ELL + team) * 2 * N;
    const uint32_t* yi = Yx + ((ybody ? 0 : (size_t)i * ELL) + team) * 2 * N;
    if (tid == 0 && i >= 2) prefetch_l2(E + (size_t)(i - 2) * ELL * N, sizeof(uint32_t) * ELL * N);
    uint64_t T[8];  // team 1: its part of R_i
    uint32_t c[8], o[8];
    if (team == 0) {
      // [A] inverse NTT of R_{i+1} ([0, 4 q)); coefficients to team 1 and the peer
#pragma unroll
      for (int j = 0; j < 8; j++) c[j] = R[j];
      jt_inv(c, xb, sfwd_tw(C), q, t, 1);
      const uint32_t rem = peer_smem(smem, peer) + (rc - base + jt_ru(t)), rbr = peer_smem(cbar + par, peer);
      st_async4(rem, rbr, c[0], c[1], c[2], c[3]);
      st_async4(rem ^ 16u, rbr, c[4], c[5], c[6], c[7]);
      jt_store_ru(c, ocb, t);
      named_arrive(4, PT);
    } else {
      query_only(i, rot, T);
      if (conv1) {
#pragma unroll
        for (int j = 0; j < 8; j++) T[j] = (uint64_t)converted(T[j]) << 32;
      }
      const uint4 w20 = ld_stream(wi + 2 * N), w21 = ld_stream(wi + 2 * N + 512);
      uint32_t y2[8];
#pragma unroll
      for (int j = 0; j < 8; j++) y2[j] = __ldg(yi + 2 * N + 128 * ((h_of(j) + half + rot) & 15u));
      if (i != gamma - 2) {
        named_sync(5, PT);  // R_{i+1} is there
        jt_load_ru(R, rnb, t);
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        T[j] += smul(R[j], u4e(j < 4 ? w20 : w21, j & 3));
        acc[j] = csub(acc[j] + redc_wide(smul(R[j], y2[j]), q, qinv), 8 * q);
      }
      named_sync(4, PT);
      jt_load_ru(c, ocb, t);
    }
    if (arrived) arrived = mbar_wait_peer(cbar + par, ((gamma - 2 - i) >> 1) & 1, A.peer_wait_iters);
    jt_load_ru(o, rc, t);
    // [B] this team's digit of the composite coefficients
    //     (gadget_decompose, rgsw/external_product.rs:16-37)
    uint32_t v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const uint64_t cc = crt_compose_from(C, qo, c[j], o[j]);
      v[j] = (uint32_t)(team == 0 ? cc : cc >> 20) & 0xFFFFFu;
    }
    // [C] its transform, [D] its products (bounds as in respond.cu)
    uint4 w0, w1;
    uint32_t yv[8];
    jt_fwd<JB_DIGIT>(v, xb, sfwd_tw(C), q, t, 1 + team, [&]() {
      w0 = ld_stream(wi);
      w1 = ld_stream(wi + 512);
#pragma unroll
      for (int j = 0; j < 8; j++) yv[j] = __ldg(yi + 128 * ((h_of(j) + half + rot) & 15u));
    });
    uint32_t s[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      uint64_t S = smul(v[j], u4e(j < 4 ? w0 : w1, j & 3));
      if (team == 1) S += T[j];
      s[j] = redc_wide(S, q, qinv);
    }
    if (team == 1) jt_store_ru(s, s1b, t);
    named_sync(6, PT);
    if (team == 0) {
      uint32_t s1[8];
      jt_load_ru(s1, s1b, t);
      // each part is in (-0.4 q, 2.7 q): their sum plus q is in (0.2 q, 5 q),
      // below 3 q once reduced
#pragma unroll
      for (int j = 0; j < 8; j++) R[j] = csub(s[j] + s1[j] + q, 2 * q);
      if (i > 0) {
        jt_store_ru(R, rnb, t);
        named_arrive(5, PT);
      }
      // both teams have read the peer's coefficients: its next but one step's may
      // come (not announced in a phase that has not ended)
      if (t == 0 && arrived) {
        if (i >= 2) mbar_expect_tx(cbar + par, 4 * N);
        misc[3] = i;
      }
    }
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j] = csub(acc[j] + redc_wide(smul(v[j], yv[j]), q, qinv) + q, 8 * q);
  }

  // ---- outputs: a_hat = INTT(R_0) (inspiring2.rs:1027-1029) by team 0, b =
  //      b_poly + INTT(sum y_all * bold_t) (inspiring2.rs:1217-1221) by team
  //      1, this residue's halves of the response ----
  uint64_t* out = (QDB ? reload_ptr(&D->out) : A.out + (size_t)qi * 4 * N) + (size_t)r * N;
  if (team == 0) jt_store_ru(acc, s1b, t);
  int outcome = 0;
  if (__syncthreads_or(!arrived) && tid == 0) outcome = peer_missing(cbar, misc, gamma, !arrived);
  cluster_arrive();
  uint32_t f[8];
  if (team == 0) {
#pragma unroll
    for (int j = 0; j < 8; j++) f[j] = R[j];
  } else {
    jt_load_ru(f, s1b, t);
#pragma unroll
    for (int j = 0; j < 8; j++) f[j] = csub(csub(f[j] + acc[j], 8 * q), 4 * q);
  }
  jt_inv(f, xb, sfwd_tw(C), q, t, 1 + team);
  if (team == 1 && t < gamma) f[0] = add_mod(f[0], bpoly[t], q);
#pragma unroll
  for (int j = 0; j < 8; j++) out[team * 2 * N + t + TEAM * j] = f[j];

  cluster_wait();  // (the peer sent its last coefficients most of a step before it arrived)
  if (r == 0 && tid == 0) {
    outcome = max(outcome, misc[6]);
    if (outcome) *status_ptr() = outcome;
  }
}

template <int MODE, bool SEEDED, bool QDB>
static cudaError_t set_pair_smem_attr() {
  return cudaFuncSetAttribute(respond_pair_kernel<MODE, SEEDED, QDB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(sizeof(uint32_t) * PairSmem::TOTAL));
}

template <int MODE>
static cudaError_t launch_pair_mode(const RespondArgs& a, bool seeded, cudaStream_t st) {
  void (*kernel)(RespondArgs) = a.qdesc ? (seeded ? respond_pair_kernel<MODE, true, true>
                                                  : respond_pair_kernel<MODE, false, true>)
                                        : (seeded ? respond_pair_kernel<MODE, true, false>
                                                  : respond_pair_kernel<MODE, false, false>);
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(2 * a.nq);
  cfg.blockDim = dim3(PT);
  cfg.dynamicSmemBytes = sizeof(uint32_t) * PairSmem::TOTAL;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = a.after_keys ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

}  // namespace

size_t respond_pair_smem_bytes() { return sizeof(uint32_t) * PairSmem::TOTAL; }

cudaError_t prepare_respond_pair_kernels() {
  const cudaError_t es[] = {
      set_pair_smem_attr<MODE_COMPAT, false, false>(),    set_pair_smem_attr<MODE_COMPAT, true, false>(),
      set_pair_smem_attr<MODE_COMPAT, false, true>(),     set_pair_smem_attr<MODE_COMPAT, true, true>(),
      set_pair_smem_attr<MODE_CRT_FIXED, false, false>(), set_pair_smem_attr<MODE_CRT_FIXED, true, false>(),
      set_pair_smem_attr<MODE_CRT_FIXED, false, true>(),  set_pair_smem_attr<MODE_CRT_FIXED, true, true>()};
  for (cudaError_t e : es)
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}

cudaError_t launch_respond_pair(const RespondArgs& a, bool seeded, cudaStream_t st) {
  if (a.nq <= 0) return cudaSuccess;
  return a.P.mode == MODE_COMPAT ? launch_pair_mode<MODE_COMPAT>(a, seeded, st)
                                 : launch_pair_mode<MODE_CRT_FIXED>(a, seeded, st);
}

}  // namespace ig
