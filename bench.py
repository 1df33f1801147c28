"""Benchmark: batched InsPIRe^2 Respond on one GB300 (or N replicas).

Workload (the metric's configuration): a 2^24-entry x 32-byte database of
uniform random bytes (seed 1) encoded resident in HBM (8192 shards of 2048
entries), d = 2048, CRT q = [268369921, 249561089], p = 2^16; each step is one
launch answering B = 128 seeded queries (real client queries made by the
library's device-side client -- inspire_client_keygen_device and
inspire_query_seeded_device -- each routed to a uniformly drawn shard), with
per-client packing keys resident.  Metric: Respond queries/s.  Every timed
response is decrypted and extracted on the device with its client's key.

  value : device-resident inputs, CUDA-event time of the Respond launches
          (each step: LAUNCHES_PER_STEP launches of B queries spread over
          --streams CUDA streams, so consecutive batches overlap on the SMs).
  e2e   : the serving loop (inspire_server_submit / poll) saturated from
          host buffers: query rows copied into pinned slots, read by the GPU,
          responses written back to pinned host memory, all inside the timed
          region.  The synchronous host-buffer batch call
          (inspire_respond_seeded_batch) is reported beside it.
  serving: Poisson arrivals at swept rates through the same loop, submitted
          at their arrival times by the library's native driver
          (inspire_server_drive), p50/p99 latency from the scheduled arrival;
          the mixed workload adds 8 resident databases of 2^18..2^26 entries.
  small batches (batch_sweep_qps, plain_single_query_host): launches of at
          most pair_threshold queries run on the two-CTA cluster kernel (one
          SM per CRT residue); *_one_cta repeats them on one CTA per query.

Usage: python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(ROOT, "inspire-rs_gb300")
for p in (ROOT, PKG):
    if p not in sys.path:
        sys.path.insert(0, p)

N = 2048
ENTRY = 32
GAMMA = 16
LOG2_ENTRIES = 24
BATCH = 128
LAUNCHES_PER_STEP = 16  # one step answers LAUNCHES_PER_STEP * BATCH queries
POOL_BATCHES = 32       # distinct staged batches, cycled
QUERY_POOL = 256        # distinct real seeded queries (device-side clients)
N_CLIENTS = 32          # registered clients (own keys), QUERY_POOL / N_CLIENTS queries each
STREAMS = 4             # CUDA streams the timed launches alternate over
REFERENCE_BUDGET_S = 150.0
SERVE_RATE_FRACS = (0.25, 0.5, 0.75, 0.9)  # open-loop offered rates, fractions of the saturated e2e rate
SERVE_DURATION_S = 1.5
MIXED_LOG2_SIZES = (18, 19, 20, 21, 22, 23, 24, 26)  # served workload: 8 databases
W_SEED = bytes(range(100, 132))
METRIC = "Respond queries/s (batched InsPIRe^2, seeded queries, InspiRING packing)"
# algorithmic bytes per query (raw shard 64 KiB + query b-rows 48 KiB + y_body 48 KiB + response 32 KiB)
ALG_BYTES_PER_QUERY = 192 * 1024
# exact modular multiplies per query of the crate's algorithm (counted before any
# regrouping): 68 transforms per residue x 1024 x 11 butterflies (~0.77 M) + ~0.93 M
# pointwise products per residue, two residues
MULMODS_PER_QUERY = 3.4e6
# multiplies the Respond kernels execute per query (gamma = 16, two residues): per residue
# 50 transforms (3 row NTTs, 15 x (one inverse + two digit NTTs), 2 output inverses) x
# 11 264 butterflies = 563 K, 15 x 6 key products x 2048 = 184 K, 16 query-only terms x
# 3 x 2048 = 98 K; then 31 K CRT compositions and 197 K exact products of the b side
EXECUTED_MULMODS_PER_QUERY = 1.92e6
# resident database bytes one query reads: contracted form 768 KiB + raw columns 64 KiB
DB_BYTES_PER_QUERY = (768 + 64) * 1024
# dram__bytes_read.sum + dram__bytes_write.sum of one B=128 batch call (one Respond
# launch), from one ncu capture on the 2^20-entry database: 109.7 + 2.6 MB
NCU_TRAFFIC_PER_LAUNCH_B128 = 112.3e6


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [x.strip() for x in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx.append(float(parts[2]))
            except ValueError:
                continue
            for nm, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": max(mx), "reasons": sorted(reasons),
                "samples": len(sm)}


def reference_query_pool(ctx, pack, n_queries, seed):
    """Seeded queries and y_body from the oracle's restatement of the crate's
    client (query.rs:43-85, inspiring2.rs:640-707), for the reference arm."""
    from oracle import oracle as O

    client = O.Client(ctx, seed=seed, rng_seed=seed + 1000)
    rng = np.random.default_rng(seed)
    locals_ = rng.integers(0, N, size=n_queries)
    seeds = np.zeros((n_queries, 6, 32), dtype=np.uint8)
    brows = np.zeros((n_queries, 6, 2 * N), dtype=np.uint64)
    for k, li in enumerate(locals_):
        seeds[k], brows[k] = client.query_seeded(int(li))
    y_body, _ = client.packing_keys(pack)
    return client, locals_, seeds, brows, y_body


class DeviceClients:
    """n_clients clients made on the device: secret keys and packing key
    bodies (inspire_client_keygen_device), per_client seeded queries each
    (inspire_query_seeded_device) of uniform local indices; query k belongs to
    client k // per_client.  Responses are checked with extract()."""

    def __init__(self, inspire, crs, torch, dev, n_clients, per_client, seed):
        self.inspire, self.crs, self.torch, self.dev = inspire, crs, torch, dev
        key = np.random.default_rng(seed).integers(0, 256, size=32, dtype=np.uint8).tobytes()
        sp = torch.cuda.current_stream(dev).cuda_stream
        self.d_sk = torch.zeros((n_clients, 2 * N), dtype=torch.int64, device=dev)
        d_yb = torch.zeros((n_clients, 3, 2 * N), dtype=torch.int64, device=dev)
        inspire.client_keygen_device(crs, key, 0, n_clients, self.d_sk.data_ptr(), d_yb.data_ptr(), sp)
        nq = n_clients * per_client
        self.locals_ = np.random.default_rng(seed + 1).integers(0, N, size=nq)
        self.client_of = np.repeat(np.arange(n_clients), per_client)
        d_idx = torch.from_numpy(self.locals_.astype(np.int32)).to(dev)
        d_seeds = torch.zeros((nq, 6, 32), dtype=torch.uint8, device=dev)
        d_brows = torch.zeros((nq, 6, 2 * N), dtype=torch.int64, device=dev)
        d_status = torch.full((nq,), -1, dtype=torch.int32, device=dev)
        for c in range(n_clients):
            sl = slice(c * per_client, (c + 1) * per_client)
            inspire.query_seeded_device(crs, self.d_sk[c].data_ptr(), key, c * per_client, per_client,
                                        d_idx[sl].data_ptr(), d_seeds[sl].data_ptr(), d_brows[sl].data_ptr(),
                                        d_status[sl].data_ptr(), sp)
        torch.cuda.synchronize()
        assert not d_status.cpu().numpy().any(), "query generation reported a nonzero status"
        self.seeds = d_seeds.cpu().numpy()
        self.brows = d_brows.cpu().numpy().view(np.uint64)
        self.y_bodies = d_yb.cpu().numpy().view(np.uint64)
        self.n_clients = n_clients

    def extract(self, client, d_ct):
        """decrypt + extract_inspiring of the device responses d_ct [n][2][2N]
        (int64 tensor) with `client`'s key, on the device; entries as numpy."""
        torch = self.torch
        d_ct = d_ct.contiguous()
        n = d_ct.shape[0]
        d_ent = torch.zeros((n, ENTRY), dtype=torch.uint8, device=self.dev)
        self.inspire.pir.extract_inspiring_device(self.crs, self.d_sk[client].data_ptr(), d_ct.data_ptr(), n, ENTRY,
                                                  d_ent.data_ptr(), torch.cuda.current_stream(self.dev).cuda_stream)
        torch.cuda.synchronize()
        return d_ent.cpu().numpy()

    def extract_host(self, client, cts):
        """The same for host responses cts [n][2][2N] (u64)."""
        cts = np.ascontiguousarray(cts, dtype=np.uint64).reshape(-1, 2, 2 * N)
        return self.extract(client, self.torch.from_numpy(cts.view(np.int64)).to(self.dev))


def cpu_baseline(db_raw, pool, mode, budget_s=12.0, max_queries=200):
    """Oracle (C restatement of the crate) respond_seeded_inspiring with
    PackParams / OfflinePackingKeys built once, OpenMP over the 16 columns,
    on the same queries and packing keys as the GPU run."""
    from oracle import oracle as O

    ctx = O.Ctx()
    omode = O.MODE_CRT_FIXED if mode == "crt_fixed" else O.MODE_COMPAT
    pack = O.Pack(ctx, GAMMA, W_SEED, mode=omode)
    locals_, seeds, brows, y_body = pool
    rng = np.random.default_rng(99)
    nshards = (len(db_raw) // ENTRY) // N
    t0 = time.perf_counter()
    done = 0
    while done < max_queries and (time.perf_counter() - t0) < budget_s:
        k = done % len(locals_)
        shard = ctx.encode_shard(db_raw, ENTRY, int(rng.integers(0, nshards)))
        rgsw = ctx.expand_rgsw(seeds[k], brows[k])
        ctx.respond_inspiring(shard, rgsw, W_SEED, mode=omode, pack=pack, y_body=y_body)
        done += 1
    dt = time.perf_counter() - t0
    return done / dt, done, dt


def kernel_microbench(inspire, crs, torch, dev, reps=20):
    """Kernel microbenchmark configuration: batched NTT / inverse NTT over both
    CRT moduli on 4096 seeded uniform polynomials (u32), and RGSW x RLWE
    external products on 1024 seeded pairs, in the crate's data semantics."""
    q = crs.params.crt_moduli
    g = torch.Generator(device="cpu").manual_seed(4)
    polys = torch.stack([torch.randint(0, q[0], (4096, N), generator=g, dtype=torch.int64),
                         torch.randint(0, q[1], (4096, N), generator=g, dtype=torch.int64)], 1).to(torch.int32).to(dev)
    cts = torch.stack([torch.randint(0, q[0], (1024, 2, N), generator=g, dtype=torch.int64),
                       torch.randint(0, q[1], (1024, 2, N), generator=g, dtype=torch.int64)], 2).to(torch.int32).to(dev)
    rg = torch.stack([torch.randint(0, q[0], (1024, 6, 2, N), generator=g, dtype=torch.int64),
                      torch.randint(0, q[1], (1024, 6, 2, N), generator=g, dtype=torch.int64)], 3).to(torch.int32).to(dev)
    out = torch.empty_like(cts)
    st = torch.cuda.current_stream(dev)
    sp = st.cuda_stream
    res = {}
    for name, fn in (("ntt_forward_4096x2", lambda: inspire.ntt_forward_device(crs, polys.data_ptr(), 4096, sp)),
                     ("ntt_inverse_4096x2", lambda: inspire.ntt_inverse_device(crs, polys.data_ptr(), 4096, sp)),
                     ("external_product_1024", lambda: inspire.external_product_device(
                         crs, cts.data_ptr(), rg.data_ptr(), out.data_ptr(), 1024, sp))):
        for _ in range(3):
            fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        for _ in range(reps):
            fn()
        e1.record(st)
        torch.cuda.synchronize()
        res[name + "_us"] = e0.elapsed_time(e1) * 1e3 / reps
    # exact modular-multiply rate probe: the integer roofline denominator
    sink = torch.empty(152 * 8 * 256, dtype=torch.int32, device=dev)
    best = None
    for _ in range(4):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        nmm = inspire.pir.mulmod_rate_device(crs, 152 * 8, 4096, sink.data_ptr(), sp)
        e1.record(st)
        torch.cuda.synchronize()
        dt = e0.elapsed_time(e1) / 1e3
        best = dt if best is None else min(best, dt)
    res["mulmod_rate_tps"] = nmm / best / 1e12  # 10^12 modular multiplies per second
    # integer tensor cores: INT8 MMA rate (mma.sync m16n8k32 s8 -> s32; the
    # tcgen05 INT8 kind does not exist for sm_103a), exactness checked
    ga = torch.Generator(device="cpu").manual_seed(8)
    a8 = torch.randint(-128, 128, (16, 32), generator=ga, dtype=torch.int8)
    b8 = torch.randint(-128, 128, (32, 8), generator=ga, dtype=torch.int8)
    da, db_ = a8.to(dev), b8.to(dev)
    dout = torch.zeros(4 * 16 * 8, dtype=torch.int32, device=dev)
    best = None
    for _ in range(4):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        nops = inspire.pir.int8_mma_rate_device(crs, 152 * 8, 4096, da.data_ptr(), db_.data_ptr(), dout.data_ptr(), sp)
        e1.record(st)
        torch.cuda.synchronize()
        dt = e0.elapsed_time(e1) / 1e3
        best = dt if best is None else min(best, dt)
    want = 4096 * (a8.to(torch.int64) @ b8.to(torch.int64))
    res["int8_mma_tops"] = nops / best / 1e12
    res["int8_mma_exact"] = bool(torch.equal(dout.cpu().view(4, 16, 8).to(torch.int64), want.expand(4, 16, 8)))
    # bytes moved per NTT launch: read + write of 4096 x 2 x 2048 u32
    byts = 2 * 4096 * 2 * N * 4
    res["ntt_forward_gbs"] = byts / (res["ntt_forward_4096x2_us"] * 1e-6) / 1e9
    res["transforms_per_s"] = 8192 / (res["ntt_forward_4096x2_us"] * 1e-6)
    res["external_products_per_s"] = 1024 / (res["external_product_1024_us"] * 1e-6)
    return res


def client_bench(inspire, crs, torch, dev, reps=3):
    """The device-side client and setup kernels, timed with CUDA events on the
    launching stream: seeded query generation (query_seeded) and decrypt +
    extract_inspiring of 4096 queries / responses per launch, key generation
    of 1024 clients per launch, and setup's public keys (15 key-switching
    matrices + 2048 crs_a vectors) for one secret key."""
    st = torch.cuda.current_stream(dev)
    sp = st.cuda_stream
    key = bytes(range(64, 96))
    nq, ncl = 4096, 1024
    d_sk = torch.zeros((ncl, 2 * N), dtype=torch.int64, device=dev)
    d_yb = torch.zeros((ncl, 3, 2 * N), dtype=torch.int64, device=dev)
    d_idx = torch.arange(nq, dtype=torch.int32, device=dev) % N
    d_seeds = torch.zeros((nq, 6, 32), dtype=torch.uint8, device=dev)
    d_brows = torch.zeros((nq, 6, 2 * N), dtype=torch.int64, device=dev)
    d_qst = torch.zeros(nq, dtype=torch.int32, device=dev)
    q = crs.params.crt_moduli
    g = torch.Generator(device="cpu").manual_seed(12)
    d_ct = torch.stack([torch.randint(0, q[0], (nq, 2, N), generator=g, dtype=torch.int64),
                        torch.randint(0, q[1], (nq, 2, N), generator=g, dtype=torch.int64)], 2).reshape(nq, 2, 2 * N)
    d_ct = d_ct.to(dev)
    d_ent = torch.zeros((nq, ENTRY), dtype=torch.uint8, device=dev)
    d_ks = torch.zeros((15, 6, 2 * N), dtype=torch.int64, device=dev)
    d_crs_a = torch.zeros((N, 2 * N), dtype=torch.int64, device=dev)
    d_kst = torch.zeros(16, dtype=torch.int32, device=dev)
    ops = (("client_keygen", ncl, lambda: inspire.client_keygen_device(crs, key, 0, ncl, d_sk.data_ptr(),
                                                                       d_yb.data_ptr(), sp)),
           ("query_gen", nq, lambda: inspire.query_seeded_device(crs, d_sk[0].data_ptr(), key, 0, nq, d_idx.data_ptr(),
                                                                  d_seeds.data_ptr(), d_brows.data_ptr(),
                                                                  d_qst.data_ptr(), sp)),
           ("extract", nq, lambda: inspire.pir.extract_inspiring_device(crs, d_sk[0].data_ptr(), d_ct.data_ptr(), nq,
                                                                         ENTRY, d_ent.data_ptr(), sp)),
           ("setup_keys", 1, lambda: inspire.setup_keygen_device(crs, key, d_sk[0].data_ptr(), d_ks.data_ptr(),
                                                                 d_crs_a.data_ptr(), d_kst.data_ptr(), sp)))
    res = {"workload": f"device-side client: {ncl} client keys, {nq} seeded queries and {nq} extractions per "
                       "launch; setup's public keys for one secret key"}
    for name, n, fn in ops:
        fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        for _ in range(reps):
            fn()
        e1.record(st)
        torch.cuda.synchronize()
        dt = e0.elapsed_time(e1) / 1e3 / reps
        res[name + "_ms"] = dt * 1e3
        if n > 1:
            res[name + "_per_s"] = n / dt
    assert not d_qst.cpu().numpy().any() and not d_kst.cpu().numpy().any(), "client kernels reported a nonzero status"
    return res


def reference_arm(args):
    """The crate's Respond path restated on the host cores: respond_seeded_inspiring
    exactly as respond.rs:391-398 runs it, including PackParams::new (brute-force
    automorphism tables) and OfflinePackingKeys::generate per query."""
    from oracle import oracle as O

    ws, rank, _ = dist_env()
    if rank != 0:
        return
    ctx = O.Ctx()
    pack_tmp = O.Pack(ctx, GAMMA, W_SEED, mode=O.MODE_COMPAT)
    pool = reference_query_pool(ctx, pack_tmp, 8, 7)
    client, locals_, seeds, brows, y_body = pool
    rng = np.random.default_rng(1)
    shard_db = rng.integers(0, 256, size=N * ENTRY, dtype=np.uint8)
    shard = ctx.encode_shard(shard_db, ENTRY, 0)
    # one faithful query takes seconds (PackParams::new searches 2048 tables by
    # brute force), so the run stops at REFERENCE_BUDGET_S and reports the
    # number of steps it timed
    times = []
    nwarm = min(args.warmup, 5)  # W as asked, at most 5 queries of the budget
    budget_t0 = time.perf_counter()
    for step in range(nwarm + args.steps):
        k = step % len(locals_)
        t0 = time.perf_counter()
        rgsw = ctx.expand_rgsw(seeds[k], brows[k])
        ctx.respond_inspiring(shard, rgsw, W_SEED, mode=O.MODE_COMPAT, pack=None, y_body=y_body)
        dt = time.perf_counter() - t0
        if step >= nwarm:
            times.append(dt)
        if time.perf_counter() - budget_t0 > REFERENCE_BUDGET_S and times:
            break
    total = sum(times)
    qps = len(times) / total
    cores = os.cpu_count()
    line = {
        "impl": "reference", "metric": METRIC, "value": qps, "unit": "queries/s", "n_gpus": args.gpus,
        "steps": len(times), "warmup": nwarm, "ms_per_step": 1e3 * total / len(times),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32/u64 modular integer",
        "data": "synthetic",
        "config": {"workload": "InsPIRe^2 respond, d=2048 CRT [268369921,249561089], p=2^16, 32-B entries, "
                               "one seeded query per step (the crate answers one query per call)",
                   "mode": "compat (the crate's own semantics)"},
        "cpu_baseline": {"value": qps, "unit": "queries/s", "cores": cores, "kind": "port",
                         "sample": f"{len(times)} queries, one per step (time-budgeted to {REFERENCE_BUDGET_S:.0f} s), "
                                   "PackParams::new + OfflinePackingKeys rebuilt per query as respond.rs:360-361 do"},
        "e2e": {"value": qps, "unit": "queries/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=100)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--launches-per-step", type=int, default=LAUNCHES_PER_STEP)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--batch", type=int, default=BATCH)
    ap.add_argument("--log2-entries", type=int, default=LOG2_ENTRIES)
    ap.add_argument("--mode", default="crt_fixed", choices=["crt_fixed", "compat"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--streams", type=int, default=STREAMS)
    ap.add_argument("--no-serve", action="store_true")
    ap.add_argument("--no-mixed", action="store_true")
    args = ap.parse_args()
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        reference_arm(args)
        return

    import torch

    ws, rank, local = dist_env()
    if ws > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl")
    dev = torch.device("cuda", local)
    torch.cuda.set_device(dev)

    import build_lib

    if rank == 0:
        build_lib.build()
    if ws > 1:
        torch.distributed.barrier()

    import inspire

    B = args.batch
    n_entries = 1 << args.log2_entries
    nshards = n_entries // N
    # each rank holds its own partition of n_entries entries (weak scaling)
    rng = np.random.default_rng(1 + rank)
    db_raw = rng.integers(0, 256, size=n_entries * ENTRY, dtype=np.uint8)
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16), W_SEED, GAMMA, mode=args.mode, device=local)
    t0 = time.perf_counter()
    edb = inspire.EncodedDatabase(crs, db_raw, ENTRY)
    torch.cuda.synchronize()
    setup_s = time.perf_counter() - t0

    clients = DeviceClients(inspire, crs, torch, dev, N_CLIENTS, QUERY_POOL // N_CLIENTS, 3 + 101 * rank)
    client_of, locals_, seeds, brows = clients.client_of, clients.locals_, clients.seeds, clients.brows
    y_body = clients.y_bodies[0]
    cids = np.array([crs.register_client(inspire.ClientPackingKeys(y_body=yb)) for yb in clients.y_bodies], np.int32)
    qcid = cids[client_of]  # registered client id of each pool query
    c0 = client_of == 0  # client 0's queries (paths that take one client)
    pool = (locals_[c0], seeds[c0], brows[c0], y_body)

    L = args.launches_per_step
    nb = POOL_BATCHES
    qrng = np.random.default_rng(5 + rank)
    pool_idx = qrng.integers(0, len(locals_), size=(nb, B))
    shard_ids = qrng.integers(0, nshards, size=(nb, B)).astype(np.uint32)

    # device-resident inputs of nb distinct batches (rows ELL..2ELL-1 only)
    d_seeds = torch.from_numpy(np.ascontiguousarray(seeds[pool_idx][:, :, 3:6, :])).to(dev)
    d_brows = torch.from_numpy(np.ascontiguousarray(brows[pool_idx][:, :, 3:6, :]).view(np.int64)).to(dev)
    d_shard = torch.from_numpy(shard_ids.view(np.int32)).to(dev)
    d_client = torch.from_numpy(np.ascontiguousarray(qcid[pool_idx])).to(dev)
    d_out = torch.zeros((nb, B, 2, 2 * N), dtype=torch.int64, device=dev)
    d_status = torch.zeros((nb, B), dtype=torch.int32, device=dev)
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)  # > 129 MB L2
    stream = torch.cuda.current_stream(dev)
    sp = stream.cuda_stream
    side = [torch.cuda.Stream(dev) for _ in range(max(1, args.streams))]

    def launch(s, n=B, st=None):
        s %= nb
        inspire.respond_seeded_batch_device(crs, edb, n, d_shard[s].data_ptr(), d_seeds[s].data_ptr(),
                                            d_brows[s].data_ptr(), d_client[s].data_ptr(), d_out[s].data_ptr(),
                                            d_status[s].data_ptr(), sp if st is None else st.cuda_stream)

    def step_launches(k, e_start, e_end):
        """One step: L launches alternating over the side streams, bracketed
        by events on the main stream."""
        e_start.record(stream)
        for st in side:
            st.wait_event(e_start)
        for j in range(L):
            launch(k * L + j, B, side[j % len(side)])
        for st in side:
            e = torch.cuda.Event()
            e.record(st)
            stream.wait_event(e)
        e_end.record(stream)

    for s in range(args.warmup):
        step_launches(s, torch.cuda.Event(), torch.cuda.Event())
    torch.cuda.synchronize()
    if ws > 1:
        torch.distributed.barrier()
    evs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    with ClockSampler(local) as clk:
        time.sleep(0.3)
        torch.cuda.synchronize()
        wall0 = time.perf_counter()
        for k in range(args.steps):
            flush.fill_(k & 0xFF)  # evict the previous step's shards from L2 (untimed)
            step_launches(k, *evs[k])
        torch.cuda.synchronize()
        wall = time.perf_counter() - wall0
    if ws > 1:
        torch.distributed.barrier()
    step_ms = [a.elapsed_time(b) for a, b in evs]
    kern_s = sum(step_ms) / 1e3
    if ws > 1:
        t = torch.tensor([kern_s], device=dev)
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        kern_s = float(t.item())
    value = ws * B * L * args.steps / kern_s

    # the same step captured once as a CUDA graph (2-stream fork/join inside)
    # and replayed: launch costs leave the host path
    value_graph = None
    if ws == 1:
        cap = torch.cuda.Stream(dev)
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=cap):
            e_fork = torch.cuda.Event()
            e_fork.record(cap)
            for st in side:
                st.wait_event(e_fork)
            for j in range(L):
                launch(j, B, side[j % len(side)])
            for st in side:
                e_join = torch.cuda.Event()
                e_join.record(st)
                cap.wait_event(e_join)
        gev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
        graph.replay()
        torch.cuda.synchronize()
        for k in range(args.steps):
            flush.fill_(k & 0xFF)
            gev[k][0].record(stream)
            graph.replay()
            gev[k][1].record(stream)
        torch.cuda.synchronize()
        value_graph = B * L * args.steps / (sum(a.elapsed_time(b) for a, b in gev) / 1e3)

    # capped grid: one launch per step answers all L * B queries with one CTA
    # per SM, each CTA taking queries in turn (no idle SMs until the last round)
    value_grid = None
    if ws == 1 and nb % L == 0:
        n_sm = torch.cuda.get_device_properties(dev).multi_processor_count
        flat = lambda t: t.view(-1, *t.shape[2:])
        f_shard, f_seeds, f_brows = flat(d_shard), flat(d_seeds), flat(d_brows)
        f_client, f_out, f_status = flat(d_client), flat(d_out), flat(d_status)

        def grid_step(k):
            b0 = (k * L) % nb * B
            inspire.respond_seeded_batch_device(crs, edb, L * B, f_shard[b0].data_ptr(), f_seeds[b0].data_ptr(),
                                                f_brows[b0].data_ptr(), f_client[b0].data_ptr(), f_out[b0].data_ptr(),
                                                f_status[b0].data_ptr(), sp, max_ctas=n_sm)

        for k in range(args.warmup):
            grid_step(k)
        torch.cuda.synchronize()
        gev2 = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
        for k in range(args.steps):
            flush.fill_(k & 0xFF)
            gev2[k][0].record(stream)
            grid_step(k)
            gev2[k][1].record(stream)
        torch.cuda.synchronize()
        value_grid = L * B * args.steps / (sum(a.elapsed_time(b) for a, b in gev2) / 1e3)

    # one wave per launch: the same step shape with launches of one query per
    # SM (152 on GB300) instead of B, drawn from the same pool, responses into
    # a scratch buffer
    value_wave = value_one_call = None
    if ws == 1:
        n_sm = torch.cuda.get_device_properties(dev).multi_processor_count
        tot = nb * B
        if n_sm <= tot:
            flat = lambda t: t.view(-1, *t.shape[2:])
            f_shard, f_seeds, f_brows, f_client = flat(d_shard), flat(d_seeds), flat(d_brows), flat(d_client)
            w_out = torch.empty_like(flat(d_out))
            w_status = torch.zeros(tot, dtype=torch.int32, device=dev)

            def wave_step(k, e_start, e_end):
                e_start.record(stream)
                for st in side:
                    st.wait_event(e_start)
                for j in range(L):
                    b0 = ((k * L + j) * n_sm) % (tot - n_sm + 1)
                    inspire.respond_seeded_batch_device(crs, edb, n_sm, f_shard[b0].data_ptr(),
                                                        f_seeds[b0].data_ptr(), f_brows[b0].data_ptr(),
                                                        f_client[b0].data_ptr(), w_out[b0].data_ptr(),
                                                        w_status[b0].data_ptr(), side[j % len(side)].cuda_stream)
                for st in side:
                    e = torch.cuda.Event()
                    e.record(st)
                    stream.wait_event(e)
                e_end.record(stream)

            for k in range(args.warmup):
                wave_step(k, torch.cuda.Event(), torch.cuda.Event())
            torch.cuda.synchronize()
            wev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
                   for _ in range(args.steps)]
            for k in range(args.steps):
                flush.fill_(k & 0xFF)
                wave_step(k, *wev[k])
            torch.cuda.synchronize()
            assert not w_status.cpu().numpy().any(), "one-wave launches reported a nonzero status"
            value_wave = L * n_sm * args.steps / (sum(a.elapsed_time(b) for a, b in wev) / 1e3)

            # the whole step as one batch call (L * B queries, one CTA each)
            def one_call(k):
                b0 = ((k * L * B) % (tot - L * B + 1)) if tot > L * B else 0
                inspire.respond_seeded_batch_device(crs, edb, L * B, f_shard[b0].data_ptr(), f_seeds[b0].data_ptr(),
                                                    f_brows[b0].data_ptr(), f_client[b0].data_ptr(),
                                                    w_out[b0].data_ptr(), w_status[b0].data_ptr(), sp)

            if L * B <= tot:
                for k in range(args.warmup):
                    one_call(k)
                torch.cuda.synchronize()
                oev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
                       for _ in range(args.steps)]
                for k in range(args.steps):
                    flush.fill_(k & 0xFF)
                    oev[k][0].record(stream)
                    one_call(k)
                    oev[k][1].record(stream)
                torch.cuda.synchronize()
                assert not w_status.cpu().numpy().any(), "the one-call step reported a nonzero status"
                value_one_call = L * B * args.steps / (sum(a.elapsed_time(b) for a, b in oev) / 1e3)
            del w_out

    # correctness of what was timed: statuses, then every response of the nb
    # pool batches decrypted and extracted on the device with its client's key
    # must equal its database entry
    status = d_status.cpu().numpy()
    assert not status.any(), "respond kernel reported a nonzero status"
    owner = client_of[pool_idx].reshape(-1)
    flat_out = d_out.view(nb * B, 2, 2 * N)
    got_flat = np.zeros((nb * B, ENTRY), np.uint8)
    for ci in range(clients.n_clients):
        sel = np.nonzero(owner == ci)[0]
        if sel.size:
            got_flat[sel] = clients.extract(ci, flat_out[torch.from_numpy(sel).to(dev)])
    got_all = got_flat.reshape(nb, B, ENTRY)
    gi_all = shard_ids.astype(np.int64) * N + locals_[pool_idx].astype(np.int64)
    verified = 0
    if args.mode == "crt_fixed":
        want_all = db_raw.reshape(-1, ENTRY)[gi_all]
        verified = int(np.all(got_all == want_all, axis=2).sum())
        assert verified == nb * B, f"{nb * B - verified} timed responses failed to decrypt"

    # batch-size sweep (single query = the plain GPU path): launches of at
    # most pair_threshold queries run on the two-CTA cluster kernel, the rest
    # on one CTA per query; the second sweep forces one CTA per query
    pair_threshold = crs.pair_threshold

    def batch_sweep():
        out = {}
        for bs in (1, 8, 32, 128):
            if bs > B:
                continue
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            reps = 20 if bs < 32 else 5
            e0.record(stream)
            for r in range(reps):
                launch(r, bs)
            e1.record(stream)
            torch.cuda.synchronize()
            out[str(bs)] = bs * reps / (e0.elapsed_time(e1) / 1e3)
        return out

    sweep = batch_sweep()
    crs.pair_threshold = 0
    sweep_one_cta = batch_sweep()
    crs.pair_threshold = pair_threshold
    # C4 same-shard variant: every query of the launch names shard 0 (the
    # shard's contracted form is read once into L2 and shared)
    same_shard = None
    if B >= 1:
        d_shard0 = torch.zeros_like(d_shard[0])
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for r in range(5):
            inspire.respond_seeded_batch_device(crs, edb, B, d_shard0.data_ptr(), d_seeds[r].data_ptr(),
                                                d_brows[r].data_ptr(), d_client[r].data_ptr(), d_out[r].data_ptr(),
                                                d_status[r].data_ptr(), sp)
        e1.record(stream)
        torch.cuda.synchronize()
        same_shard = B * 5 / (e0.elapsed_time(e1) / 1e3)

    micro = kernel_microbench(inspire, crs, torch, dev)
    client_side = client_bench(inspire, crs, torch, dev) if rank == 0 else None
    codec = wire_bench(inspire, crs, seeds[0], brows[0], y_body, d_out[0, 0].cpu().numpy().view(np.uint64)
                       .reshape(2, 2 * N))

    # end to end through the host-buffer C ABI call, pinned host memory
    h_seeds = torch.empty((B, 6, 32), dtype=torch.uint8, pin_memory=True)
    h_brows = torch.empty((B, 6, 2 * N), dtype=torch.int64, pin_memory=True)
    h_out = torch.empty((B, 2, 2 * N), dtype=torch.int64, pin_memory=True)
    hs, hb, ho = h_seeds.numpy(), h_brows.numpy().view(np.uint64), h_out.numpy().view(np.uint64)
    e2e_times = []
    for k in range(args.warmup + args.steps):
        s = k % nb
        hs[:] = seeds[pool_idx[s]]
        hb[:] = brows[pool_idx[s]]
        t0 = time.perf_counter()
        _respond_into(crs, edb, shard_ids[s], hs, hb, qcid[pool_idx[s]], ho)
        dt = time.perf_counter() - t0
        if k >= args.warmup:
            e2e_times.append(dt)
    e2e_s = sum(e2e_times)
    if ws > 1:
        t = torch.tensor([e2e_s], device=dev)
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        e2e_s = float(t.item())
    sync_call_qps = ws * B * args.steps / e2e_s  # one host-buffer call of B queries per step
    h2d = B * (4 + 4 + 32 * 3 + 3 * 2 * N * 8)
    d2h = B * (2 * 2 * N * 8 + 4)

    # plain single-query path: one synchronous host-buffer call per query
    def single_calls():
        lat = []
        for k in range(200):
            s = k % nb
            hs1, hb1, ho1 = hs[:1], hb[:1], ho[:1]
            hs1[:] = seeds[pool_idx[s, :1]]
            hb1[:] = brows[pool_idx[s, :1]]
            t0 = time.perf_counter()
            _respond_into(crs, edb, shard_ids[s, :1], hs1, hb1, qcid[pool_idx[s, :1]], ho1)
            lat.append(time.perf_counter() - t0)
        lat = np.array(lat[10:]) * 1e3
        return {"qps": float(1e3 / lat.mean()), "p50_ms": float(np.percentile(lat, 50)),
                "p99_ms": float(np.percentile(lat, 99))}

    plain = dict(single_calls(), path="inspire_respond_seeded_batch with n=1 from host buffers (page-locked), one "
                                      "call at a time; two-CTA cluster kernel (one SM per CRT residue)")
    crs.pair_threshold = 0
    plain_one_cta = dict(single_calls(), path="the same call on the one-CTA kernel")
    crs.pair_threshold = pair_threshold

    c3 = c3_bench(inspire, crs, seeds[c0], brows[c0], y_body) if rank == 0 else None
    shard_files = shard_file_bench(inspire, crs, seeds[c0], brows[c0], y_body) if rank == 0 else None
    tree = tree_bench(inspire, crs, edb, nshards, clients, seeds[c0], brows[c0], torch, dev, B) if rank == 0 else None
    nopack = nopacking_bench(inspire, crs, edb, nshards, seeds, brows, B) if rank == 0 else None

    serving = None
    e2e_value = sync_call_qps
    e2e_kind = "synchronous host-buffer batch call (inspire_respond_seeded_batch), B queries per call"
    if not args.no_serve:
        serving = serve_bench(inspire, crs, edb, nshards, clients, client_of, qcid, locals_, seeds, brows, db_raw, B,
                              args, torch, dev)
        closed = serving["closed_loop"]["achieved_qps"]
        if ws > 1:
            t = torch.tensor([closed], device=dev)
            torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MIN)
            closed = float(t.item())
        if closed * ws > e2e_value:
            e2e_value = closed * ws
            e2e_kind = ("serving loop saturated from host buffers (inspire_server_submit/poll_batch): rows copied "
                        "into pinned slots, read by the GPU over the host link, responses written to pinned host "
                        "memory; per-step byte counts are for B queries")

    http = None
    if not args.no_serve and rank == 0:
        http = http_bench(inspire, crs, edb, db_raw, nshards, clients, seeds, brows)

    peaks_path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    peaks = json.load(open(peaks_path)) if os.path.exists(peaks_path) else {}
    hbm_peak = peaks.get("hbm_gbs", 6800.0)
    mean_kernel_s = kern_s / (args.steps * L)
    achieved_gbs = ALG_BYTES_PER_QUERY * B / mean_kernel_s / 1e9
    resident_bytes = edb.device_bytes

    if rank == 0:
        cpu = None
        if not args.no_cpu_baseline and ws == 1:
            qps, nq, dt = cpu_baseline(db_raw, pool, args.mode)
            cpu = {"value": qps, "unit": "queries/s", "cores": os.cpu_count(), "kind": "port",
                   "sample": f"{nq} queries in {dt:.1f} s (oracle C restatement, PackParams/OfflinePackingKeys "
                             f"hoisted, OpenMP over 16 columns)"}
        line = {
            "metric": METRIC, "value": value, "unit": "queries/s", "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1e3 * kern_s / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u32 modular integer (exact)", "data": "synthetic",
            "config": {"workload": f"batched InsPIRe^2 respond: 2^{args.log2_entries} entries x 32 B resident "
                                   f"({nshards} shards), B={B} seeded queries per launch, uniform shard ids",
                       "step": f"{L} batch calls x {B} queries (one Respond launch each) over "
                               f"{len(side)} streams",
                       "streams": len(side),
                       "queries": f"{QUERY_POOL} distinct real seeded queries from {N_CLIENTS} clients generated "
                                  "on the device (keys, packing keys and queries; packing keys registered and "
                                  "resident); each launch slot draws one with its own uniform shard id",
                       "mode": args.mode, "global_batch": B * ws, "ring_dim": N,
                       "crt_moduli": [268369921, 249561089], "p": 65536,
                       "l2": "flushed between timed steps (256 MiB write); resident DB 6.5 GiB > L2",
                       "db_setup_s": setup_s, "db_device_bytes": resident_bytes},
            "e2e": {"value": e2e_value, "unit": "queries/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                    "path": e2e_kind, "sync_batch_call_qps": sync_call_qps},
            "roofline": {"bound": "hbm", "achieved": achieved_gbs, "peak": hbm_peak, "unit": "GB/s",
                         "frac": achieved_gbs / hbm_peak,
                         "traffic": NCU_TRAFFIC_PER_LAUNCH_B128 if B == 128 else None,
                         "note": "algorithmic bytes 192 KiB/query; the kernel is bound by integer issue, see int_roofline"},
            "int_roofline": {"bound": "integer pipes", "achieved": value * MULMODS_PER_QUERY / 1e12,
                             "peak": micro["mulmod_rate_tps"], "unit": "10^12 modular multiplies/s",
                             "frac": value * MULMODS_PER_QUERY / 1e12 / micro["mulmod_rate_tps"],
                             "executed_per_query": EXECUTED_MULMODS_PER_QUERY,
                             "frac_executed": value * EXECUTED_MULMODS_PER_QUERY / 1e12 / micro["mulmod_rate_tps"],
                             "note": "achieved/frac: the crate's algorithm, 3.4 M exact 28-bit modular multiplies "
                                     "per query; frac_executed: the 1.92 M the kernels execute after regrouping; "
                                     "peak = the rate probe (independent lazy Shoup multiply chains, all SMs)"},
            "cpu_baseline": cpu,
            "clocks": clk.summary(),
            "gpu_launches": args.steps * L,  # one Respond launch per device-row batch call
            "verified_responses": verified,
            "value_cuda_graph": value_graph,
            "value_capped_grid": value_grid,
            "value_one_wave": value_wave,
            "value_one_call": value_one_call,
            "db_scan_gbs": value * DB_BYTES_PER_QUERY / 1e9,
            "batch_sweep_qps": sweep,
            "batch_sweep_qps_one_cta": sweep_one_cta,
            "pair_threshold": pair_threshold,
            "plain_single_query_qps": sweep.get("1"),
            "plain_single_query_host": plain,
            "plain_single_query_host_one_cta": plain_one_cta,
            "same_shard_batch_qps": same_shard,
            "c3_single_query": c3,
            "shard_files": shard_files,
            "tree_packing": tree,
            "nopacking": nopack,
            "batched_over_plain": value / plain["qps"],
            "p50_ms": None if serving is None else serving["headline"]["p50_ms"],
            "p99_ms": None if serving is None else serving["headline"]["p99_ms"],
            "serving": serving,
            "http_serving": http,
            "kernel_microbench": micro,
            "client_side": client_side,
            "wire_codec": codec,
            "wall_s_timed_region": wall,
        }
        print(json.dumps(line), flush=True)
    if ws > 1:
        torch.distributed.destroy_process_group()


def http_bench(inspire, crs, edb, db_raw, nshards, clients, seeds, brows, n_bodies=48, duration_s=2.0):
    """The HTTP front end (the crate's /query_seeded route) on loopback:
    SeededClientQuery JSON bodies with the client's packing keys inline, as
    the crate's client posts them, from spawned client processes over
    keep-alive connections.  The library's native server (csrc/http.cu):
    closed loop at 1, 8, 32 and 64 connections, then Poisson arrivals at
    50 % and 90 % of the best closed-loop rate; the Python server
    (inspire.http_server.PirHttpServer) closed loop at 8 connections.  One
    reply per distinct body is decrypted first and checked against the
    database entry."""
    import http.client
    import json as _json

    from inspire import http_load
    from inspire.http_server import GpuBackend, NativeHttpServer, PirHttpServer

    rng = np.random.default_rng(17)
    picks = []
    bodies = []
    for _ in range(n_bodies):
        i = int(rng.integers(0, len(clients.locals_)))
        sid = int(rng.integers(0, nshards))
        picks.append((i, sid))
        bodies.append(http_load.seeded_query_json(sid, seeds[i], brows[i], clients.y_bodies[clients.client_of[i]]))

    def verify(srv):
        host, port = srv.address
        conn = http.client.HTTPConnection(host, port, timeout=60)
        ok = 0
        for (i, sid), body in zip(picks, bodies):
            conn.request("POST", "/query_seeded", body=body, headers={"Content-Type": "application/json"})
            r = conn.getresponse()
            data = r.read()
            if r.status != 200:
                continue
            ct = _json.loads(data)["response"]["ciphertext"]
            cts = np.array([ct["a"]["coeffs"], ct["b"]["coeffs"]], dtype=np.uint64)
            got = clients.extract_host(int(clients.client_of[i]), cts[None])[0]
            gi = sid * N + int(clients.locals_[i])
            ok += int(np.array_equal(got, db_raw[gi * ENTRY:(gi + 1) * ENTRY]))
        conn.close()
        return ok

    res = {"route": "POST /query_seeded (SeededClientQuery JSON, packing keys inline)",
           "body_bytes": len(bodies[0]), "distinct_bodies": n_bodies,
           "resident_client_keys": "cached by y_body (the first query of a client registers its keys)"}
    native = NativeHttpServer(crs, edb, max_batch=128, max_inflight=4, capacity=4096)
    try:
        ok = verify(native)
        closed = [http_load.run_load(native.url, bodies, c, duration_s=duration_s) for c in (1, 8, 32, 64)]
        best = max(c["achieved_rps"] for c in closed)
        open_loop = [dict(http_load.run_load(native.url, bodies, 64, duration_s=duration_s, rate=f * best), load_frac=f)
                     for f in (0.5, 0.9)]
    finally:
        native.close()
    res["native"] = {"server": "csrc/http.cu (C++ thread per connection; native JSON codecs; GPU serving loop)",
                     "verified_replies": ok, "closed_loop": closed, "open_loop": open_loop}
    backend = GpuBackend(crs, edb, max_batch=128, max_inflight=4, capacity=4096)
    py = PirHttpServer(backend).start()
    try:
        ok = verify(py)
        closed = [http_load.run_load(py.url, bodies, 8, duration_s=duration_s)]
    finally:
        py.close()
        backend.close()
    res["python"] = {"server": "inspire.http_server.PirHttpServer (http.server thread per connection)",
                     "verified_replies": ok, "closed_loop": closed}
    return res


def shard_file_bench(inspire, crs, seeds, brows, y_body, log2_entries=20):
    """Setup from files: a 2^20-entry database written as the crate's binary
    shard files (save_shards_binary layout) to a temporary directory and read
    back into HBM with inspire_db_load_shards (page cache warm), checked by
    answering one query from both databases."""
    import shutil
    import tempfile

    rng = np.random.default_rng(6)
    raw = np.frombuffer(rng.bytes((1 << log2_entries) * ENTRY), dtype=np.uint8)
    edb = inspire.EncodedDatabase(crs, raw, ENTRY)
    d = tempfile.mkdtemp(prefix="inspire_shards_")
    try:
        t0 = time.perf_counter()
        edb.save_shards(d)
        save_s = time.perf_counter() - t0
        files = os.listdir(d)
        nbytes = sum(os.path.getsize(os.path.join(d, f)) for f in files)
        inspire.EncodedDatabase.load_shards(crs, d).close()  # warm the page cache
        t0 = time.perf_counter()
        edb2 = inspire.EncodedDatabase.load_shards(crs, d)
        load_s = time.perf_counter() - t0
        q = inspire.SeededClientQuery(7, seeds[0], brows[0],
                                      inspiring_packing_keys=inspire.ClientPackingKeys(y_body=y_body))
        r1 = inspire.respond_seeded_inspiring(crs, edb, q)
        r2 = inspire.respond_seeded_inspiring(crs, edb2, q)
        same = bool(np.array_equal(r1.ciphertext.a, r2.ciphertext.a) and np.array_equal(r1.ciphertext.b, r2.ciphertext.b))
        edb2.close()
    finally:
        shutil.rmtree(d, ignore_errors=True)
        edb.close()
    assert same, "database loaded from shard files answers differently"
    return {"workload": f"2^{log2_entries} entries x 32 B as {len(files)} shard files ({nbytes / 2**20:.0f} MiB), "
                        "read into HBM (contracted form built on the GPU), page cache warm",
            "load_s": load_s, "load_gbs": nbytes / load_s / 1e9, "save_s": save_s, "same_response": same}


def c3_bench(inspire, crs, seeds, brows, y_body, n=60):
    """C3: plain single-query InsPIRe^2 on 2^20 entries x 32 B resident, one
    query at a time through respond_seeded_inspiring with the packing keys in
    the query (the crate's per-request path: the server rotates y_body for
    every query), latency per call."""
    rng = np.random.default_rng(5)
    raw = np.frombuffer(rng.bytes((1 << 20) * ENTRY), dtype=np.uint8)
    edb = inspire.EncodedDatabase(crs, raw, ENTRY)
    nsh = edb.num_shards
    keys = inspire.ClientPackingKeys(y_body=y_body)
    lat = []
    for k in range(n):
        q = inspire.SeededClientQuery(int(rng.integers(0, nsh)), seeds[k % len(seeds)], brows[k % len(brows)],
                                      inspiring_packing_keys=keys)
        t0 = time.perf_counter()
        inspire.respond_seeded_inspiring(crs, edb, q)
        lat.append(time.perf_counter() - t0)
    edb.close()
    lat = np.array(lat[5:]) * 1e3
    return {"workload": "2^20 entries x 32 B, one seeded query per call, keys in the query",
            "qps": float(1e3 / lat.mean()), "p50_ms": float(np.percentile(lat, 50)),
            "p99_ms": float(np.percentile(lat, 99))}


def tree_bench(inspire, crs, edb, nshards, clients, seeds, brows, torch, dev, B, n_single=20, reps=3):
    """Tree packing (respond_seeded_packed) on the same resident database:
    the CRS's Galois keys made on the device for client 0's secret key, one
    query per host call (latency), and batches of B queries per call."""
    key = bytes(range(200, 232))
    d_keys = torch.zeros((11, 6, 2 * N), dtype=torch.int64, device=dev)
    d_st = torch.zeros(11, dtype=torch.int32, device=dev)
    inspire.galois_keygen_device(crs, key, clients.d_sk[0].data_ptr(), d_keys.data_ptr(), d_st.data_ptr(),
                                 torch.cuda.current_stream(dev).cuda_stream)
    torch.cuda.synchronize()
    assert not d_st.cpu().numpy().any(), "Galois key generation reported a nonzero status"
    crs.load_galois_keys(d_keys.cpu().numpy().view(np.uint64))
    rng = np.random.default_rng(8)
    lat = []
    for k in range(n_single + 3):
        j = k % len(seeds)
        q = inspire.SeededClientQuery(int(rng.integers(0, nshards)), seeds[j], brows[j])
        t0 = time.perf_counter()
        inspire.respond_seeded_packed(crs, edb, q)
        if k >= 3:
            lat.append(time.perf_counter() - t0)
    lat = np.array(lat) * 1e3
    sid = rng.integers(0, nshards, size=B).astype(np.uint32)
    pick = rng.integers(0, len(seeds), size=B)
    sd, br = seeds[pick], brows[pick]
    plen = crs.params.plen

    def run_batch(sd, br, outs):
        inspire.respond_seeded_packed_batch(crs, edb, sid, sd, br, *outs)  # warm-up
        t0 = time.perf_counter()
        for _ in range(reps):
            inspire.respond_seeded_packed_batch(crs, edb, sid, sd, br, *outs)
        return B * reps / (time.perf_counter() - t0)

    pageable_qps = run_batch(sd, br, ())
    with pinned_copies(inspire, [sd, br], [((B, plen), np.uint64), ((B, 2 * plen), np.uint64)]) as (ins, outs):
        pinned_qps = run_batch(*ins, outs)
    return {"workload": f"respond_seeded_packed on the resident database, 16 columns, d = 2048 (127 key "
                        f"switches per query); Galois keys made on the device",
            "single_query_p50_ms": float(np.percentile(lat, 50)), "single_query_p99_ms": float(np.percentile(lat, 99)),
            "batch": B, "batch_qps": pinned_qps, "batch_qps_pageable": pageable_qps,
            "note": "host-buffer calls (batch_qps: page-locked query and response arrays; batch_qps_pageable: "
                    "ordinary numpy arrays); at d = 2048 with two CRT primes the crate's tree-packed responses do "
                    "not decrypt, so this path is measured for parity with the crate, not used for retrieval"}


class pinned_copies:
    """Page-locked copies of the input arrays and page-locked output arrays
    of the given shapes, freed on exit."""

    def __init__(self, inspire, inputs, out_shapes):
        self.bufs = []
        self.ins = []
        for a in inputs:
            pb = inspire.pir.PinnedBuffer(a.shape, a.dtype)
            pb.array[...] = a
            self.bufs.append(pb)
            self.ins.append(pb.array)
        self.outs = []
        for shape, dt in out_shapes:
            pb = inspire.pir.PinnedBuffer(shape, dt)
            self.bufs.append(pb)
            self.outs.append(pb.array)

    def __enter__(self):
        return self.ins, self.outs

    def __exit__(self, *exc):
        self.ins = self.outs = None
        for pb in self.bufs:
            pb.close()
        return False


def nopacking_bench(inspire, crs, edb, nshards, seeds, brows, B, reps=3):
    """The NoPacking variant (respond_seeded, combined ciphertext only) on the
    same resident database: batches of B queries per host-buffer call."""
    rng = np.random.default_rng(9)
    sid = rng.integers(0, nshards, size=B).astype(np.uint32)
    pick = rng.integers(0, len(seeds), size=B)
    sd, br = seeds[pick], brows[pick]

    def run_batch(sd, br, out=None):
        inspire.respond_seeded_nopacking_batch(crs, edb, sid, sd, br, out)  # warm-up
        t0 = time.perf_counter()
        for _ in range(reps):
            inspire.respond_seeded_nopacking_batch(crs, edb, sid, sd, br, out)
        return B * reps / (time.perf_counter() - t0)

    pageable_qps = run_batch(sd, br)
    with pinned_copies(inspire, [sd, br], [((B, 2, crs.params.plen), np.uint64)]) as (ins, outs):
        pinned_qps = run_batch(*ins, outs[0])
    # the crate's respond_seeded: one query per call, with its 16 column
    # ciphertexts (the columns split over 16 CTAs)
    lat = []
    for k in range(23):
        q = inspire.SeededClientQuery(int(sid[k % B]), sd[k % B], br[k % B])
        t0 = time.perf_counter()
        inspire.respond_seeded(crs, edb, q)
        if k >= 3:
            lat.append(time.perf_counter() - t0)
    lat = np.array(lat) * 1e3
    return {"workload": f"respond_seeded (NoPacking) on the resident database, 16 columns, batches of {B} "
                        "queries per host-buffer call (rows copied in, combined ciphertexts copied out; "
                        "batch_qps with page-locked arrays, batch_qps_pageable with ordinary numpy arrays)",
            "batch": B, "batch_qps": pinned_qps, "batch_qps_pageable": pageable_qps,
            "single_query_with_columns_p50_ms": float(np.percentile(lat, 50)),
            "single_query_with_columns_p99_ms": float(np.percentile(lat, 99))}


def serve_bench(inspire, crs, edb, nshards, clients, client_of, qcid, locals_, seeds, brows, db_raw, B, args, torch,
                dev):
    """Serving-loop measurements: saturated closed loop (the e2e number),
    open-loop Poisson sweeps with p50/p99 latency on the 2^24-entry database,
    and the mixed served workload over 8 databases of 2^18..2^26 entries."""
    from inspire import serving as sv

    # the distinct real queries in pinned rows; one submit call carries up to
    # 256 of them (each names its own shard)
    pool = sv.QueryPool(seeds, brows, locals_, pinned=True, client_ids=qcid)
    cid = int(qcid[0])  # unused when the pool names each query's client
    main = [sv.Target(edb, nshards, 1.0)]
    ws, _, _ = dist_env()
    if ws == 1:
        tuned = sv.autotune(lambda **kw: inspire.Server(crs, capacity=8192, **kw), main, pool, cid)
    else:  # ranks share the node's host cores: one default configuration, no search
        tuned = {"best": {"max_batch": 256, "max_inflight": 4, "batch_wait_us": 100}, "table": []}
    cfg = tuned["best"]
    srv = inspire.Server(crs, capacity=8192, **cfg)

    def check(samples, raws, targets_nshards):
        for d, shard, pidx, out in samples[:16]:
            gi = shard * N + int(locals_[pidx])
            got = clients.extract_host(int(client_of[pidx]), out)[0]
            if args.mode == "crt_fixed":
                assert np.array_equal(got, raws[d][gi * ENTRY:(gi + 1) * ENTRY]), "served response failed to decrypt"

    sv.run(srv, main, pool, cid, rate=None, n_queries=8192, n_threads=4)  # warm-up

    def closed_run(server, targets, n_threads):
        st0 = server.stats()
        res = sv.run(server, targets, pool, cid, rate=None, n_queries=1 << 17, n_threads=n_threads, keep_outputs=True,
                     closed_chunk=256)
        st1 = server.stats()
        res["mean_batch"] = (st1["completed"] - st0["completed"]) / max(1, st1["batches"] - st0["batches"])
        res["submitter_threads"] = n_threads
        return res

    def burst_run(server, n=8192):
        """One thread submits n queries back to back (pool-sized calls, rows
        borrowed), then collects them: the loop's rate without per-call
        Python overhead on the collection side."""
        from inspire.pir import now_ns

        rng = np.random.default_rng(3)
        sh = rng.integers(0, nshards, size=n).astype(np.uint32)
        tickets = []
        t0 = now_ns()
        k = 0
        while k < n:
            m = min(pool.q, n - k)
            t, rc = server.submit(edb, sh[k:k + m], pool.seeds[:m], pool.b_rows[:m], pool.client_ids[:m], borrow=True)
            tickets.append(t)
            k += len(t)
        done = server.poll_batch(np.concatenate(tickets))
        return {"n": n, "achieved_qps": n / ((done.max() - t0) / 1e9)}

    burst_run(srv)  # warm-up
    burst = burst_run(srv)
    closed = max((closed_run(srv, main, t) for t in (4, 8)), key=lambda r: r["achieved_qps"])
    check(closed.pop("samples"), [db_raw], None)
    cap = closed["achieved_qps"]
    # open loop: arrivals submitted by the library's native driver (a
    # scripting-language submitter adds its own scheduling delay), one
    # sample of responses checked per run
    sv.run_native(srv, main, pool, cid, rate=0.25 * cap, duration_s=0.5, seed=10)  # warm-up
    sweep = []
    for frac in SERVE_RATE_FRACS:
        r = sv.run_native(srv, main, pool, cid, rate=frac * cap, duration_s=SERVE_DURATION_S, seed=11,
                          keep_outputs=True)
        check(r.pop("samples"), [db_raw], None)
        r["load_frac"] = frac
        sweep.append(r)
    head = next((r for r in sweep if r["load_frac"] == 0.75), sweep[-1])
    out = {"config": {**cfg, "capacity": 8192, "submitter_threads": closed["submitter_threads"],
                      "autotune": tuned["table"],
                      "query_rows": "pinned host memory, borrowed (read in place by the GPU)",
                      "arrivals": "Poisson, offered rate = fraction x saturated closed-loop rate; submitted at "
                                  "their arrival times by the library's native driver (inspire_server_drive)",
                      "database": f"{nshards * N} entries x 32 B"},
           "closed_loop": closed, "burst": burst, "open_loop": sweep,
           "headline": {"p50_ms": head["p50_ms"], "p99_ms": head["p99_ms"], "offered_qps": head["offered_qps"],
                        "achieved_qps": head["achieved_qps"], "load_frac": head["load_frac"]}}
    srv.close()

    if not args.no_mixed and ws == 1:
        rng = np.random.default_rng(21)
        dbs, raws, targets = [], [], []
        t0 = time.perf_counter()
        for lg in MIXED_LOG2_SIZES:
            raw = np.frombuffer(rng.bytes((1 << lg) * ENTRY), dtype=np.uint8)
            db = inspire.EncodedDatabase(crs, raw, ENTRY)
            dbs.append(db)
            raws.append(raw)
            targets.append(sv.Target(db, (1 << lg) // N, float(1 << lg)))
        torch.cuda.synchronize()
        setup = time.perf_counter() - t0
        srv = inspire.Server(crs, capacity=8192, **cfg)
        sv.run(srv, targets, pool, cid, rate=None, n_queries=8192, n_threads=4)  # warm-up
        mclosed = closed_run(srv, targets, closed["submitter_threads"])
        check(mclosed.pop("samples"), raws, None)
        mcap = mclosed["achieved_qps"]
        sv.run_native(srv, targets, pool, cid, rate=0.25 * mcap, duration_s=0.5, seed=10)  # warm-up
        msweep = []
        for frac in (0.5, 0.75, 0.9):
            r = sv.run_native(srv, targets, pool, cid, rate=frac * mcap, duration_s=SERVE_DURATION_S, seed=12,
                              keep_outputs=True)
            check(r.pop("samples"), raws, None)
            r["load_frac"] = frac
            msweep.append(r)
        out["mixed"] = {"databases_log2_entries": list(MIXED_LOG2_SIZES),
                        "device_bytes": int(sum(d.device_bytes for d in dbs)), "setup_s": setup,
                        "query_index": "uniform over all entries of all databases",
                        "closed_loop": mclosed, "open_loop": msweep}
        srv.close()
        for d in dbs:
            d.close()
    pool.close()
    return out


def wire_bench(inspire, crs, seeds, brows, y_body, out_ct, reps=50):
    """Host cost of the HTTP wire formats through the native codecs: parse a
    real SeededClientQuery JSON body (with y_body keys), write the JSON reply
    and the bincode ServerResponse of a real response (one core)."""
    import json as _json

    from inspire import wire

    P = crs.params
    q = crs.params.crt_moduli

    def poly(c):
        return {"coeffs": [int(x) for x in c], "moduli": list(q), "q": q[0] * q[1], "dim": N,
                "crt_q0_inv_mod_q1": pow(q[0], q[1] - 2, q[1]), "is_ntt": False}

    body = _json.dumps({"shard_id": 7, "rgsw_ciphertext": {
        "rows": [{"seed": [int(b) for b in seeds[i]], "b": poly(brows[i])} for i in range(6)],
        "gadget": {"base": 1 << 20, "len": 3, "q": q[0] * q[1]}}, "packing_mode": "inspiring",
        "inspiring_packing_keys": {"y_body": [poly(p) for p in y_body], "full_key": False, "num_to_pack": 16}},
        separators=(",", ":")).encode()
    resp = inspire.ServerResponse(inspire.RlweCiphertext(out_ct[0], out_ct[1]), [])
    res = {"query_json_bytes": len(body)}
    for name, fn in (("parse_query_json", lambda: wire.seeded_query_from_json(P, body)),
                     ("write_response_json", lambda: wire.query_response_to_json(P, resp, 1)),
                     ("write_response_bincode", lambda: wire.server_response_to_bincode(P, resp))):
        fn()
        t0 = time.perf_counter()
        for _ in range(reps):
            fn()
        res[name + "_us"] = (time.perf_counter() - t0) / reps * 1e6
    res["response_json_bytes"] = len(wire.query_response_to_json(P, resp, 1))
    res["response_bincode_bytes"] = len(wire.server_response_to_bincode(P, resp))
    res["parse_query_json_mb_s"] = len(body) / res["parse_query_json_us"]
    return res


def _respond_into(crs, edb, shard_ids, seeds, brows, client_ids, out):
    """inspire_respond_seeded_batch into a caller-owned (pinned) output."""
    import ctypes as C

    from inspire.pir import _check

    sid = np.ascontiguousarray(shard_ids, dtype=np.uint32)
    cids = np.ascontiguousarray(client_ids, dtype=np.int32)
    v = C.c_void_p
    _check(crs.L.inspire_respond_seeded_batch(crs.h, edb.h, len(sid), sid.ctypes.data_as(v), seeds.ctypes.data_as(v),
                                              brows.ctypes.data_as(v), cids.ctypes.data_as(v), out.ctypes.data_as(v)))


if __name__ == "__main__":
    main()
