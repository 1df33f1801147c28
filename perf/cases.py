"""What the server's Respond path is timed on: the calls that a user of this
framework makes, over the sizes that they meet.

Each kind below is one public entry point.  Databases, columns, batch sizes
and modes are those of this repository's tests and benchmark: 32-byte entries
(16 columns of 16 bits) and smaller ones, 1024 to 2^20 entries resident (a
query reads one shard of 2048 entries whatever the database's size, and 2^20
entries are already larger than the L2 cache), 1 to 2048 queries per call,
both semantics of the NTT-domain automorphism ("crt_fixed", whose responses
decrypt, and "compat", the crate's bits).

All results are whole numbers (residues modulo the two CRT primes), computed
exactly, so they are the same bit for bit whatever the schedule.
"""
import os
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "inspire-rs_gb300"))

import inspire  # noqa: E402

N = 2048
ELL = 3
MODULI = (268369921, 249561089)
KEY_SETS = 16  # clients whose packing keys are registered; a batch mixes them
SUBMITTERS = 4  # threads of a served burst, each with its share of the queries


def listed():
    return [
        # one unseeded query with its keys, the crate's smallest database: the host call's latency
        {"name": "full query, 2^10", "kind": "full", "entries": 1024, "entry_size": 32, "mode": "crt_fixed"},
        # one seeded query with its keys, as the HTTP server answers it: the host call's latency
        {"name": "seeded query, 2^20", "kind": "one", "entries": 1 << 20, "entry_size": 32, "mode": "crt_fixed"},
        # a small batch on device buffers, registered clients: fewer queries than SMs
        {"name": "batch of 8", "kind": "batch", "n": 8, "entries": 1 << 20, "entry_size": 32, "mode": "crt_fixed"},
        # an odd batch with the crate's own semantics, and a database whose last shard is partial
        {"name": "batch of 77, compat", "kind": "batch", "n": 77, "entries": 1000003, "entry_size": 32,
         "mode": "compat"},
        # the benchmark's batch
        {"name": "batch of 128", "kind": "batch", "n": 128, "entries": 1 << 20, "entry_size": 32,
         "mode": "crt_fixed"},
        # one call with many waves of queries: the rate of a full GPU
        {"name": "batch of 2048", "kind": "batch", "n": 2048, "entries": 1 << 20, "entry_size": 32,
         "mode": "crt_fixed"},
        # a burst through the serving loop: rows read from, and responses written to, page-locked host memory
        {"name": "served burst of 601", "kind": "serve", "n": 601, "entries": 1 << 20, "entry_size": 32,
         "mode": "crt_fixed"},
        # NoPacking, combined ciphertexts, page-locked host buffers
        {"name": "NoPacking batch of 128", "kind": "nopack", "n": 128, "entries": 1 << 20, "entry_size": 32,
         "mode": "crt_fixed"},
        # tree packing (11 levels of key switches per query), page-locked host buffers
        {"name": "tree batch of 33", "kind": "tree", "n": 33, "entries": 1 << 20, "entry_size": 32,
         "mode": "crt_fixed"},
        # the transforms by themselves, both directions; the large one is the kernel benchmark's size
        {"name": "NTT of 4096", "kind": "ntt", "n": 4096, "inverse": False},
        {"name": "inverse NTT of 301", "kind": "ntt", "n": 301, "inverse": True},
        # general RLWE x RGSW products, the kernel benchmark's size
        {"name": "1024 external products", "kind": "product", "n": 1024},
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread over the logarithm, often odd."""
    v = int(round(lo * (hi / lo) ** rng.random()))
    return min(hi, max(lo, v | 1 if rng.random() < 0.5 else v))


def draw(rng):
    kind = rng.choice(["full", "one", "batch", "batch", "batch", "batch", "serve", "nopack", "tree", "ntt", "ntt",
                       "product"])
    if kind == "ntt":
        return {"kind": kind, "n": _log(rng, 1, 4096), "inverse": rng.random() < 0.5}
    if kind == "product":
        return {"kind": kind, "n": _log(rng, 1, 1024)}
    case = {"kind": kind, "entries": _log(rng, 1024, 1 << 20), "entry_size": rng.choice([32, 32, 32, 31, 16, 15]),
            "mode": rng.choice(["crt_fixed", "crt_fixed", "compat"])}
    most = {"batch": 2048, "serve": 601, "nopack": 128, "tree": 33}.get(kind)
    if most:
        case["n"] = _log(rng, 100 if kind == "serve" else 1, most)
    return case


def _uniform(gen, *lead):
    """Uniform residue polynomials (*lead, 2, N), int64: RLWE ciphertexts and
    key-switching rows are uniform to everyone without the secret key."""
    return torch.stack([torch.randint(0, q, (*lead, N), generator=gen, device="cuda") for q in MODULI], dim=-2)


def _host(t, *shape):
    return t.reshape(*shape).cpu().numpy().view(np.uint64)


class _Pinned(np.ndarray):
    """A view of page-locked memory; `owner` keeps it allocated as long as the view or one of its own is held."""


def _pinned(shape, dtype):
    buf = inspire.PinnedBuffer(shape, dtype)
    view = buf.array.view(_Pinned)
    view.owner = buf
    return view


def _pinned_copy(a):
    view = _pinned(a.shape, a.dtype)
    view[...] = a
    return view


def _seed_bytes(gen, *shape):
    return torch.randint(0, 256, shape, dtype=torch.uint8, generator=gen, device="cuda")


def _stream():
    return torch.cuda.current_stream().cuda_stream


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("ntt", "product"):
        s["crs"] = inspire.ServerCrs(inspire.InspireParams(p=1 << 16), bytes(32), 16)
        n = s["n"] = case["n"]
        if kind == "ntt":
            # in place, and a transform of uniform residues is uniform again: every pass is one on new values
            s["polys"] = _uniform(gen, n).to(torch.int32).contiguous()
        else:
            s["ct"] = _uniform(gen, n, 2).to(torch.int32).contiguous()
            s["rgsw"] = _uniform(gen, n, 2 * ELL, 2).to(torch.int32).contiguous()
            s["out"] = torch.zeros((n, 2, 2, N), dtype=torch.int32, device="cuda")
        return s

    entry = case["entry_size"]
    w_seed = _seed_bytes(gen, 32).cpu().numpy().tobytes()
    crs = s["crs"] = inspire.ServerCrs(inspire.InspireParams(p=1 << 16), w_seed, inspire.num_columns(entry),
                                       mode=case["mode"])
    raw = _seed_bytes(gen, case["entries"] * entry).cpu().numpy()
    db = s["db"] = inspire.EncodedDatabase(crs, raw, entry)
    n = s["n"] = case.get("n", 1)
    shard = torch.randint(0, db.num_shards, (n,), dtype=torch.int32, generator=gen, device="cuda")
    plen = crs.params.plen
    if kind == "full":
        keys = inspire.ClientPackingKeys(y_body=_host(_uniform(gen, ELL), ELL, plen))
        s["query"] = inspire.ClientQuery(int(shard[0]), _host(_uniform(gen, 2 * ELL, 2), 2 * ELL, 2, plen),
                                         inspiring_packing_keys=keys)
        return s
    seeds = _seed_bytes(gen, n, 2 * ELL, 32)
    b_rows = _uniform(gen, n, 2 * ELL)
    if kind == "one":
        keys = inspire.ClientPackingKeys(y_body=_host(_uniform(gen, ELL), ELL, plen))
        s["query"] = inspire.SeededClientQuery(int(shard[0]), seeds[0].cpu().numpy(),
                                               _host(b_rows, 2 * ELL, plen), inspiring_packing_keys=keys)
        return s
    if kind in ("batch", "serve"):
        clients = [crs.register_client(inspire.ClientPackingKeys(y_body=y))
                   for y in _host(_uniform(gen, min(n, KEY_SETS), ELL), min(n, KEY_SETS), ELL, plen)]
        client = [clients[k % len(clients)] for k in range(n)]
    if kind == "batch":
        s["shard"] = shard
        s["seeds"] = seeds[:, ELL:].contiguous()
        s["b_rows"] = b_rows[:, ELL:].contiguous()
        s["client"] = torch.tensor(client, dtype=torch.int32, device="cuda")
        s["out"] = torch.zeros((n, 2, plen), dtype=torch.int64, device="cuda")
        s["status"] = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        return s
    s["shards"] = shard.cpu().numpy().astype(np.uint32)
    s["seeds"] = _pinned_copy(seeds.cpu().numpy())
    s["b_rows"] = _pinned_copy(_host(b_rows, n, 2 * ELL, plen))
    if kind == "serve":
        s["client"] = np.array(client, np.int32)
        # the serving configuration that the benchmark's tuner picks
        s["server"] = inspire.Server(crs, max_batch=152, max_inflight=8, capacity=max(n, 152), batch_wait_us=25)
        s["threads"] = ThreadPoolExecutor(SUBMITTERS)
        s["parts"] = [(n * t // SUBMITTERS, n * (t + 1) // SUBMITTERS) for t in range(SUBMITTERS)]
        s["out"] = _pinned((n, 2, plen), np.uint64)
    elif kind == "nopack":
        s["out"] = _pinned((n, 2, plen), np.uint64)
    else:
        crs.load_galois_keys(_host(_uniform(gen, 11, 2 * ELL), 11, 2 * ELL, plen))
        s["out_a"], s["out_b"] = _pinned((n, plen), np.uint64), _pinned((n, 2 * plen), np.uint64)
    return s


def _serve(s, lo, hi):
    """One submitter's share of a burst."""
    tickets, _ = s["server"].submit(s["db"], s["shards"][lo:hi], s["seeds"][lo:hi], s["b_rows"][lo:hi],
                                    s["client"][lo:hi], borrow=True)
    s["server"].poll_batch(tickets, s["out"][lo:hi])


def run(s):
    kind, crs = s["kind"], s["crs"]
    if kind == "ntt":
        call = inspire.ntt_inverse_device if s["case"]["inverse"] else inspire.ntt_forward_device
        call(crs, s["polys"].data_ptr(), s["n"], _stream())
        return s["polys"]
    if kind == "product":
        inspire.external_product_device(crs, s["ct"].data_ptr(), s["rgsw"].data_ptr(), s["out"].data_ptr(), s["n"],
                                        _stream())
        return s["out"]
    if kind == "full":
        r = inspire.respond_inspiring(crs, s["db"], s["query"])
        return {"a": r.ciphertext.a, "b": r.ciphertext.b}
    if kind == "one":
        r = inspire.respond_seeded_inspiring(crs, s["db"], s["query"])
        return {"a": r.ciphertext.a, "b": r.ciphertext.b}
    if kind == "batch":
        inspire.respond_seeded_batch_device(crs, s["db"], s["n"], s["shard"].data_ptr(), s["seeds"].data_ptr(),
                                            s["b_rows"].data_ptr(), s["client"].data_ptr(), s["out"].data_ptr(),
                                            s["status"].data_ptr(), _stream())
        return {"responses": s["out"], "status": s["status"]}
    if kind == "serve":
        list(s["threads"].map(lambda part: _serve(s, *part), s["parts"]))
        return s["out"].view(np.int64)
    if kind == "nopack":
        return inspire.respond_seeded_nopacking_batch(crs, s["db"], s["shards"], s["seeds"], s["b_rows"], s["out"])
    a, b = inspire.respond_seeded_packed_batch(crs, s["db"], s["shards"], s["seeds"], s["b_rows"], s["out_a"],
                                               s["out_b"])
    return {"a": a, "b": b}


def work(case):
    """Bytes: the query's rows (the second half of the RGSW ciphertext, 64-bit
    words), the client's key body, the shard's raw columns and the response.
    Operations: two per modular multiply-add of the transforms and products
    that the protocol's steps consist of."""
    kind, n = case["kind"], case.get("n", 1)
    poly = 2 * N  # words of one polynomial, both residues
    transform = 2 * 11 * (N // 2)  # multiply-adds of one polynomial's transform
    if kind == "ntt":
        return {"bytes": n * 2 * 4 * poly, "flops": n * 2 * transform}
    if kind == "product":
        return {"bytes": n * 4 * poly * (2 + 4 * ELL + 2),
                "flops": n * 2 * (transform * (2 * ELL + 4 * ELL + 2) + poly * 4 * ELL)}
    gamma = (case["entry_size"] + 1) // 2
    rows = 8 * poly * ELL * (2 if kind == "full" else 1)
    shard = 2 * gamma * N
    front = transform * 2 * ELL + poly * 2 * ELL * gamma
    if kind == "nopack":
        return {"bytes": n * (rows + shard + 16 * poly), "flops": n * 2 * (front + transform * (ELL + 2))}
    if kind == "tree":
        switches = 8 * gamma - 1  # levels 1 to 7 for each column, then the pairs
        return {"bytes": n * (rows + shard + 16 * poly) + 11 * 4 * ELL * 4 * poly,
                "flops": n * 2 * (front + switches * (transform * (ELL + 2) + poly * 2 * ELL))}
    keys = 8 * poly * ELL
    steps = gamma - 1
    return {"bytes": n * (rows + shard + keys + 16 * poly),
            "flops": n * 2 * (front + poly * ELL * gamma + transform * (4 * steps + 2) + poly * 2 * ELL * steps)}


# ---- the transforms and products in 64-bit integer arithmetic, with torch alone ----


def _roots(q):
    """psi^brv(k), k < N, for the first primitive 2N-th root that small bases give."""
    g = next(g for g in range(2, q) if pow(g, (q - 1) // 2, q) == q - 1)
    psi = pow(g, (q - 1) // (2 * N), q)
    return [pow(psi, int(format(k, "011b")[::-1], 2), q) for k in range(N)]


def _forward(a, q):
    """Negacyclic NTT along the last axis, bit-reversed slots."""
    roots = torch.tensor(_roots(q), device=a.device)
    shape, m, t = a.shape, 1, N // 2
    while m < N:
        a = a.reshape(-1, m, 2, t)
        v = a[:, :, 1] * roots[m:2 * m].reshape(1, m, 1) % q
        a = torch.stack([(a[:, :, 0] + v) % q, (a[:, :, 0] - v) % q], dim=2)
        m, t = 2 * m, t // 2
    return a.reshape(shape)


def _inverse(a, q):
    roots = torch.tensor([pow(w, -1, q) for w in _roots(q)], device=a.device)
    shape, m, t = a.shape, N // 2, 1
    while m:
        a = a.reshape(-1, m, 2, t)
        a = torch.stack([(a[:, :, 0] + a[:, :, 1]) % q,
                         (a[:, :, 0] - a[:, :, 1]) * roots[m:2 * m].reshape(1, m, 1) % q], dim=2)
        m, t = m // 2, 2 * t
    return a.reshape(shape) * pow(N, -1, q) % q


def exact(case, seed):
    """The transforms and the products.  The responses' residues, whole
    numbers too, have no short restatement here."""
    if case["kind"] == "ntt":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        a = _uniform(gen, case["n"])
        out = []
        for r, q in enumerate(MODULI):
            if case["inverse"]:  # slots in Montgomery form, R = 2^64
                out.append(_inverse(a[:, r] * pow(2, -64, q) % q, q))
            else:
                out.append(_forward(a[:, r], q) * pow(2, 64, q) % q)
        return torch.stack(out, dim=-2).to(torch.int32)
    if case["kind"] == "product":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        n = case["n"]
        ct, rgsw = _uniform(gen, n, 2), _uniform(gen, n, 2 * ELL, 2)
        q0, q1 = MODULI
        whole = ct[:, :, 0] + q0 * ((ct[:, :, 1] - ct[:, :, 0]) * pow(q0, -1, q1) % q1)
        out = []
        for r, q in enumerate(MODULI):
            total = 0
            for row in range(2 * ELL):
                digit = (whole[:, row // ELL] >> (20 * (row % ELL))) & ((1 << 20) - 1)
                total = (total + _forward(digit, q)[:, None] * _forward(rgsw[:, row, :, r], q)) % q
            out.append(_inverse(total, q))
        return torch.stack(out, dim=-2).to(torch.int32)
    return None
