"""The bounded waits for a query's rows in the kernels of host-buffer calls, made
to run out at once: the call fails with the status of rows that did not come
(3) and not with that of copies still in flight (4), and the next call on the
same context is answered correctly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
PLEN = 2 * N
ENTRY = 4
DEFAULT = 1 << 20


@pytest.mark.parametrize("n", [1, 64, 65, 160])  # (in ordinary memory gathered or copied to the device)
@pytest.mark.parametrize("kind", ["nopacking", "respond"])
def test_row_wait_running_out(oracle_mod, kind, n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire
    from inspire import _native as nat

    rng = np.random.default_rng(n)
    ctx = oracle_mod.Ctx()
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16), bytes(32), ENTRY // 2, mode="crt_fixed")
    db = rng.integers(0, 256, size=2 * N * ENTRY, dtype=np.uint8)
    edb = inspire.EncodedDatabase(crs, db, ENTRY)
    pack = oracle_mod.Pack(ctx, ENTRY // 2, bytes(32), mode=oracle_mod.MODE_CRT_FIXED)
    client = oracle_mod.Client(ctx, seed=0, rng_seed=n)
    y_body, _ = client.packing_keys(pack)
    cid = crs.register_client(inspire.ClientPackingKeys(y_body=y_body))
    qs = [client.query_seeded(i) for i in (5, 2047)]
    pick = np.arange(n) % 2
    seeds = np.stack([s for s, _ in qs])[pick]
    rows = inspire.PinnedBuffer((n, 6, PLEN), np.uint64)
    rows.array[...] = np.stack([b.reshape(6, PLEN) for _, b in qs])[pick]
    shard = ctx.encode_shard(db, ENTRY, 1)
    if kind == "nopacking":
        want = np.stack([ctx.respond_nopacking(shard, ctx.expand_rgsw(s, b)) for s, b in qs])[pick]
    else:
        want = np.stack([ctx.respond_inspiring(shard, ctx.expand_rgsw(s, b), bytes(32), mode=oracle_mod.MODE_CRT_FIXED,
                                               pack=pack, y_body=y_body) for s, b in qs])[pick]
    out = inspire.PinnedBuffer((n, 2, PLEN), np.uint64)

    def call(b_rows, to):
        if kind == "nopacking":
            return inspire.respond_seeded_nopacking_batch(crs, edb, [1] * n, seeds, b_rows, to)
        return inspire.respond_seeded_batch(crs, edb, [1] * n, seeds, b_rows, [cid] * n, to)

    def expect_rows_missing(b_rows, to):
        with pytest.raises(inspire.PirError, match=r"kernel status 3 for query 0") as ei:
            call(b_rows, to)
        assert ei.value.status == nat.ERR_DEVICE_STATUS

    plain = rows.array.copy()
    assert crs.L.inspire_ctx_set_row_wait_iters(crs.h, 0) == 0
    expect_rows_missing(rows.array, out.array)
    if kind == "nopacking" or n <= 64:  # (larger Respond batches in ordinary memory read device rows without a wait)
        expect_rows_missing(plain, None)
    assert crs.L.inspire_ctx_set_row_wait_iters(crs.h, DEFAULT) == 0
    for b_rows, to in ((rows.array, out.array), (plain, None)):
        assert np.array_equal(call(b_rows, to), want)
    rows.close()
    out.close()
