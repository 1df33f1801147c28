"""The Respond kernels under other CRT moduli, bit-exact against the oracle
(src/pir/respond.rs:284-398): primes just above a power of two, whose seeded
expansion rejects half of its draws (gen_range's zone, poly.rs:251-281) and
takes the kernel's general expansion; primes just below one, which take the
fast one; small primes, below which the 2^20 gadget digits barely fit; and
residue 1's modulus above residue 0's.  Together they reach the ends of the
transforms' lazy ranges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
W_SEED = bytes(range(31, 63))


def _is_prime(v):
    return all(v % d for d in range(2, int(v ** 0.5) + 1))


def _primes(start, step, count):
    """The first `count` primes = 1 (mod 2N) from `start` on, in steps of +-2N."""
    out, v = [], (start // (2 * N)) * (2 * N) + 1
    while len(out) < count:
        v += step * 2 * N
        if _is_prime(v):
            out.append(v)
    return out


MODULI = {
    "half of the draws rejected": _primes(1 << 27, 1, 2),
    "residue 1 rejects half": [_primes(1 << 28, -1, 1)[0], _primes(1 << 27, 1, 1)[0]],
    "just below 2^28": _primes(1 << 28, -1, 2),
    "second modulus larger": [249561089, 268369921],
    "just below 2^21": _primes(1 << 21, -1, 2),
    "just above 2^20": _primes(1 << 20, 1, 2),
}


@pytest.mark.parametrize("entry", [2, 8, 32])
@pytest.mark.parametrize("mode", ["crt_fixed", "compat"])
@pytest.mark.parametrize("which", list(MODULI))
def test_respond_other_moduli(oracle_mod, which, mode, entry):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    O, moduli = oracle_mod, MODULI[which]
    if moduli[0] >= 2 * moduli[1]:
        moduli = moduli[::-1]
    gamma = entry // 2
    rng = np.random.default_rng(len(which) + entry)
    ctx = O.Ctx(moduli=moduli)
    omode = O.MODE_CRT_FIXED if mode == "crt_fixed" else O.MODE_COMPAT
    pack = O.Pack(ctx, gamma, W_SEED, mode=omode)
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16, crt_moduli=tuple(moduli)), W_SEED, gamma, mode=mode)
    db = rng.integers(0, 256, size=(N + 700) * entry, dtype=np.uint8)
    edb = inspire.EncodedDatabase(crs, db, entry)
    n = 3
    polys = lambda k: np.concatenate([rng.integers(0, q, size=(k, N), dtype=np.uint64) for q in moduli], axis=1)  # noqa: E731
    b_rows = polys(6 * n).reshape(n, 6, 2 * N)
    b_rows[0] = np.repeat(np.array(moduli, np.uint64) - 1, N)  # the largest residues
    y_body = polys(3)
    seeds = rng.integers(0, 256, size=(n, 6, 32), dtype=np.uint8)
    shard_ids = [0, 1, 1]
    shards = [ctx.encode_shard(db, entry, s) for s in range(2)]
    want = np.stack([ctx.respond_inspiring(shards[s], ctx.expand_rgsw(sd, br), W_SEED, mode=omode, pack=pack,
                                           y_body=y_body)
                     for s, sd, br in zip(shard_ids, seeds, b_rows)])
    cid = crs.register_client(inspire.ClientPackingKeys(y_body=y_body))
    for threshold in (0, 3):  # one CTA per query, then the two-CTA cluster
        crs.pair_threshold = threshold
        host = inspire.respond_seeded_batch(crs, edb, shard_ids, seeds, b_rows, [cid] * n)
        assert np.array_equal(host, want)
        d = [torch.from_numpy(a).cuda() for a in (np.array(shard_ids, np.int32), seeds[:, 3:].copy(),
                                                  b_rows[:, 3:].copy().view(np.int64), np.full(n, cid, np.int32))]
        out = torch.zeros((n, 2, 2 * N), dtype=torch.int64, device="cuda")
        status = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        inspire.respond_seeded_batch_device(crs, edb, n, *[t.data_ptr() for t in d], out.data_ptr(),
                                            status.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert not status.cpu().numpy().any()
        assert np.array_equal(out.cpu().numpy().view(np.uint64), want)
