"""NoPacking batches in ordinary memory on either side of the count up to which
their rows are gathered, and with only the rows or only the responses
page-locked, bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
PLEN = 2 * N
ENTRY = 8


@pytest.mark.parametrize("n", [1, 5, 6, 64, 65])
def test_gathered_and_copied(oracle_mod, n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    rng = np.random.default_rng(n)
    ctx = oracle_mod.Ctx()
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16), bytes(32), ENTRY // 2)
    db = rng.integers(0, 256, size=2 * N * ENTRY, dtype=np.uint8)
    edb = inspire.EncodedDatabase(crs, db, ENTRY)
    k = 3
    b_rows = np.concatenate([rng.integers(0, q, size=(k, 6, N), dtype=np.uint64) for q in (268369921, 249561089)], axis=2)
    seeds = rng.integers(0, 256, size=(k, 6, 32), dtype=np.uint8)
    shards = np.array([0, 1, 1])
    want = np.stack([ctx.respond_nopacking(ctx.encode_shard(db, ENTRY, s), ctx.expand_rgsw(sd, br))
                     for s, sd, br in zip(shards, seeds, b_rows)])
    pick = np.arange(n) % k
    rows, out = inspire.PinnedBuffer((n, 6, PLEN), np.uint64), inspire.PinnedBuffer((n, 2, PLEN), np.uint64)
    rows.array[...] = b_rows[pick]
    for b, o in ((b_rows[pick], None), (rows.array, None), (b_rows[pick], out.array), (rows.array, out.array)):
        out.array[...] = 0
        got = inspire.respond_seeded_nopacking_batch(crs, edb, shards[pick], seeds[pick], b, o)
        assert np.array_equal(got, want[pick])
    del got, b, o
    rows.close()
    out.close()
