"""Tree packing (src/inspiring/automorph_pack.rs:171-485) for every number of
columns, with CRT moduli at the ends of the transforms' lazy ranges and with
the rows read in place or copied, bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
MODULI = {"default": (268369921, 249561089), "half of the draws rejected": (134246401, 134250497),
          "just above 2^20": (1073153, 1093633)}


@pytest.mark.parametrize("gamma", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("which", list(MODULI))
def test_tree_shapes(oracle_mod, which, gamma):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    moduli = MODULI[which]
    rng = np.random.default_rng(gamma)
    ctx = oracle_mod.Ctx(moduli=moduli)
    polys = lambda k: np.concatenate([rng.integers(0, q, size=(k, N), dtype=np.uint64) for q in moduli], axis=1)  # noqa: E731
    keys = polys(11 * 6).reshape(11, 6, 2 * N)
    db = rng.integers(0, 256, size=(N + 700) * 2 * gamma, dtype=np.uint8)
    k = 3
    b_rows = polys(6 * k).reshape(k, 6, 2 * N)
    b_rows[0] = np.repeat(np.array(moduli, np.uint64) - 1, N)  # the largest residues
    seeds = rng.integers(0, 256, size=(k, 6, 32), dtype=np.uint8)
    shards = [0, 1, 1]
    rgsw = [ctx.expand_rgsw(sd, br) for sd, br in zip(seeds, b_rows)]
    for mode, omode in (("crt_fixed", oracle_mod.MODE_CRT_FIXED), ("compat", oracle_mod.MODE_COMPAT)):
        crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16, crt_moduli=moduli), bytes(32), gamma, mode=mode)
        crs.load_galois_keys(keys)
        edb = inspire.EncodedDatabase(crs, db, 2 * gamma)
        want = [ctx.respond_one_packing(ctx.encode_shard(db, 2 * gamma, s), rg, keys, mode=omode)
                for s, rg in zip(shards, rgsw)]
        for n in (1, 3, 40):
            pick = np.arange(n) % k
            sid, sd, br = np.array(shards)[pick], seeds[pick], np.ascontiguousarray(b_rows[pick])
            pinned = [inspire.PinnedBuffer(sh, np.uint64) for sh in (br.shape, (n, 2 * N), (n, 4 * N))]
            pinned[0].array[...] = br
            for args in ((br,), [b.array for b in pinned]):
                a, b = inspire.respond_seeded_packed_batch(crs, edb, sid, sd, *args)
                for i, p in enumerate(pick):
                    assert np.array_equal(a[i], want[p][0]) and np.array_equal(b[i], want[p][1])
            del a, b, args
            for b in pinned:
                b.close()
        full = inspire.respond_one_packing(crs, edb, inspire.ClientQuery(1, rgsw[2].reshape(6, 2, -1)))
        assert np.array_equal(full.ciphertext.a, want[2][0]) and np.array_equal(full.ciphertext.b, want[2][1])
        edb.close()
        crs.close()
