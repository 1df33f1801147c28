"""NoPacking's combined ciphertexts (src/pir/respond.rs:71-115, 408-415) by
every way the rows reach the kernel -- page-locked memory read in place,
ordinary memory gathered or copied -- at counts around its limits, and with CRT
moduli whose expansion takes the general path, bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
MODULI = {"default": (268369921, 249561089), "half of the draws rejected": (134246401, 134250497),
          "just above 2^20": (1073153, 1093633)}


@pytest.mark.parametrize("entry", [2, 32])
@pytest.mark.parametrize("which", list(MODULI))
def test_combined_paths(oracle_mod, which, entry):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    moduli = MODULI[which]
    rng = np.random.default_rng(entry)
    ctx = oracle_mod.Ctx(moduli=moduli)
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16, crt_moduli=moduli), bytes(32), entry // 2)
    db = rng.integers(0, 256, size=(N + 700) * entry, dtype=np.uint8)
    edb = inspire.EncodedDatabase(crs, db, entry)
    k = 3
    b_rows = np.concatenate([rng.integers(0, q, size=(k, 6, N), dtype=np.uint64) for q in moduli], axis=2)
    b_rows[0] = np.repeat(np.array(moduli, np.uint64) - 1, N)  # the largest residues
    seeds = rng.integers(0, 256, size=(k, 6, 32), dtype=np.uint8)
    shards = [0, 1, 1]
    want = np.stack([ctx.respond_nopacking(ctx.encode_shard(db, entry, s), ctx.expand_rgsw(sd, br))
                     for s, sd, br in zip(shards, seeds, b_rows)])
    for n in (1, 3, 64, 65, 153):
        pick = np.arange(n) % k
        sid, sd, br = np.array(shards)[pick], seeds[pick], np.ascontiguousarray(b_rows[pick])
        assert np.array_equal(inspire.respond_seeded_nopacking_batch(crs, edb, sid, sd, br), want[pick])
        rows, out = inspire.PinnedBuffer(br.shape, np.uint64), inspire.PinnedBuffer((n, 2, 2 * N), np.uint64)
        rows.array[...] = br
        out.array[...] = 0
        inspire.respond_seeded_nopacking_batch(crs, edb, sid, sd, rows.array, out.array)
        assert np.array_equal(out.array, want[pick])
        rows.close()
        out.close()
    full = inspire.respond(crs, edb, inspire.ClientQuery(1, ctx.expand_rgsw(seeds[2], b_rows[2]).reshape(6, 2, -1)),
                           with_columns=False)
    assert np.array_equal(np.stack([full.ciphertext.a, full.ciphertext.b]), want[2])
