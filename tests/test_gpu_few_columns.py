"""Page-locked batches of more queries than SMs, of few columns (one SM to a
query, its whole rows staged at once) and of just more (two CTAs to an SM, rows
in chunks): bit-exact against the oracle, with moduli whose expansion takes the
general path, and with the wait for the rows made to run out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
MODULI = {"default": (268369921, 249561089), "half of the draws rejected": (134246401, 134250497)}


@pytest.mark.parametrize("gamma", [1, 2, 4, 8])
@pytest.mark.parametrize("mode", ["crt_fixed", "compat"])
@pytest.mark.parametrize("which", list(MODULI))
def test_page_locked_batches_of_few_columns(oracle_mod, which, mode, gamma):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    O, moduli, entry = oracle_mod, MODULI[which], 2 * gamma
    rng = np.random.default_rng(gamma)
    ctx = O.Ctx(moduli=moduli)
    omode = O.MODE_CRT_FIXED if mode == "crt_fixed" else O.MODE_COMPAT
    pack = O.Pack(ctx, gamma, bytes(32), mode=omode)
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16, crt_moduli=moduli), bytes(32), gamma, mode=mode)
    db = rng.integers(0, 256, size=(N + 700) * entry, dtype=np.uint8)
    edb = inspire.EncodedDatabase(crs, db, entry)
    polys = lambda k: np.concatenate([rng.integers(0, q, size=(k, N), dtype=np.uint64) for q in moduli], axis=1)  # noqa: E731
    k = 3
    b_rows = polys(6 * k).reshape(k, 6, 2 * N)
    b_rows[0] = np.repeat(np.array(moduli, np.uint64) - 1, N)  # the largest residues
    seeds = rng.integers(0, 256, size=(k, 6, 32), dtype=np.uint8)
    y_body = polys(3)
    shards = [ctx.encode_shard(db, entry, s) for s in range(2)]
    shard_ids = np.array([0, 1, 1])
    want = np.stack([ctx.respond_inspiring(shards[s], ctx.expand_rgsw(sd, br), bytes(32), mode=omode, pack=pack,
                                           y_body=y_body) for s, sd, br in zip(shard_ids, seeds, b_rows)])
    cid = crs.register_client(inspire.ClientPackingKeys(y_body=y_body))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in (sms, sms + 1, 2 * sms + 5):
        pick = np.arange(n) % k
        rows, out = inspire.PinnedBuffer((n, 6, 2 * N), np.uint64), inspire.PinnedBuffer((n, 2, 2 * N), np.uint64)
        rows.array[...] = b_rows[pick]
        out.array[...] = 0

        def call():
            inspire.respond_seeded_batch(crs, edb, shard_ids[pick], seeds[pick], rows.array, [cid] * n, out.array)

        assert crs.L.inspire_ctx_set_row_wait_iters(crs.h, 0) == 0
        with pytest.raises(inspire.PirError, match="kernel status 3 for query 0"):
            call()
        assert crs.L.inspire_ctx_set_row_wait_iters(crs.h, 1 << 20) == 0
        for _ in range(2):
            call()
            assert np.array_equal(out.array, want[pick]), n
        rows.close()
        out.close()
