"""A single seeded query with its keys inline whose rows and response are
page-locked (read and written in place), only partly so, unaligned or lying
over one another: the same response, the oracle's."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
PLEN = 2 * N


@pytest.mark.parametrize("threshold", [0, 76])  # one CTA per query, two
@pytest.mark.parametrize("gamma", [1, 4, 16])
def test_single_query_buffers(oracle_mod, gamma, threshold):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire
    from inspire import _native as nat

    rng = np.random.default_rng(gamma)
    ctx = oracle_mod.Ctx()
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16), bytes(32), gamma)
    crs.pair_threshold = threshold
    db = rng.integers(0, 256, size=2 * N * 2 * gamma, dtype=np.uint8)
    edb = inspire.EncodedDatabase(crs, db, 2 * gamma)
    pack = oracle_mod.Pack(ctx, gamma, bytes(32), mode=oracle_mod.MODE_CRT_FIXED)
    polys = lambda k: np.concatenate([rng.integers(0, q, size=(k, N), dtype=np.uint64) for q in (268369921, 249561089)], axis=1)  # noqa: E731
    seeds, b_rows, y_body = rng.integers(0, 256, size=(6, 32), dtype=np.uint8), polys(6), polys(3)
    want = ctx.respond_inspiring(ctx.encode_shard(db, 2 * gamma, 1), ctx.expand_rgsw(seeds, b_rows), bytes(32),
                                 mode=oracle_mod.MODE_CRT_FIXED, pack=pack, y_body=y_body).reshape(-1)

    def call(rows_at, out_at):
        q = nat.SeededQueryC(1, seeds.ctypes.data, rows_at, 1, y_body.ctypes.data, None)
        assert crs.L.inspire_respond_seeded_inspiring(crs.h, edb.h, C.byref(q), C.c_void_p(out_at)) == 0, \
            crs.L.inspire_last_error()

    size = b_rows.nbytes
    locked = inspire.PinnedBuffer((size + 16 + want.nbytes + 16,), np.uint8)
    base = locked.array.ctypes.data
    plain = np.zeros(PLEN * 2, np.uint64)
    for rows_off, out_off in ((0, size + 16), (8, size + 16), (0, size + 8), (0, size + 4), (0, 0), (0, 3 * 8 * PLEN),
                              (0, None)):
        for _ in range(2):
            locked.array[...] = 0
            locked.array[rows_off:rows_off + size] = b_rows.view(np.uint8).reshape(-1)
            call(base + rows_off, plain.ctypes.data if out_off is None else base + out_off)
            got = plain if out_off is None else locked.array[out_off:out_off + want.nbytes].copy().view(np.uint64)
            assert np.array_equal(got, want), (rows_off, out_off)
    locked.close()
