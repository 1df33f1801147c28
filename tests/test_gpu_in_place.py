"""Batches whose page-locked buffers may not be read and written in place:
responses over the rows they answer, and responses that start off their
64-bit words.  Both are answered as from separate buffers, bit-exact against
the oracle, at counts either side of the gathered batches' limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
PLEN = 2 * N
ENTRY = 8


@pytest.fixture(scope="module")
def world(oracle_mod):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    rng = np.random.default_rng(31)
    ctx = oracle_mod.Ctx()
    w_seed = bytes(range(32))
    pack = oracle_mod.Pack(ctx, ENTRY // 2, w_seed, mode=oracle_mod.MODE_CRT_FIXED)
    client = oracle_mod.Client(ctx, seed=0, rng_seed=6)
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16), w_seed, ENTRY // 2, mode="crt_fixed")
    keys = np.concatenate([rng.integers(0, q, size=(11, 6, N), dtype=np.uint64) for q in (268369921, 249561089)], axis=2)
    crs.load_galois_keys(keys)
    y_body, _ = client.packing_keys(pack)
    cid = crs.register_client(inspire.ClientPackingKeys(y_body=y_body))
    db = rng.integers(0, 256, size=2 * N * ENTRY, dtype=np.uint8)
    edb = inspire.EncodedDatabase(crs, db, ENTRY)
    W = {"inspire": inspire, "crs": crs, "edb": edb, "cid": cid, "shards": [0, 1, 1]}
    qs = [client.query_seeded(i) for i in (3, 700, 2047)]
    W["seeds"] = np.stack([s for s, _ in qs])
    W["b_rows"] = np.stack([b.reshape(6, PLEN) for _, b in qs])
    sh = [ctx.encode_shard(db, ENTRY, s) for s in W["shards"]]
    rg = [ctx.expand_rgsw(s, b) for s, b in qs]
    W["nopacking"] = np.stack([ctx.respond_nopacking(h, g) for h, g in zip(sh, rg)])
    W["respond"] = np.stack([ctx.respond_inspiring(h, g, w_seed, mode=oracle_mod.MODE_CRT_FIXED, pack=pack, y_body=y_body)
                             for h, g in zip(sh, rg)])
    W["tree"] = [ctx.respond_one_packing(h, g, keys, mode=oracle_mod.MODE_CRT_FIXED) for h, g in zip(sh, rg)]
    return W


def call(W, kind, n, rows, out):
    pick = np.arange(n) % 3
    sid, sd = np.array(W["shards"])[pick], W["seeds"][pick]
    inspire = W["inspire"]
    if kind == "nopacking":
        inspire.respond_seeded_nopacking_batch(W["crs"], W["edb"], sid, sd, rows, out.reshape(n, 2, PLEN))
    else:
        inspire.respond_seeded_batch(W["crs"], W["edb"], sid, sd, rows, [W["cid"]] * n, out.reshape(n, 2, PLEN))


@pytest.mark.parametrize("n", [2, 64, 65, 153])
@pytest.mark.parametrize("kind", ["nopacking", "respond"])
def test_responses_over_the_rows(world, kind, n):
    W = world
    pick = np.arange(n) % 3
    buf = W["inspire"].PinnedBuffer((n, 6, PLEN), np.uint64)
    flat = buf.array.reshape(-1)
    for at in (0, flat.size - n * 2 * PLEN, 3 * PLEN):
        buf.array[...] = W["b_rows"][pick]
        out = flat[at:at + n * 2 * PLEN]
        call(W, kind, n, buf.array, out)
        assert np.array_equal(out.reshape(n, 2, PLEN), W[kind][pick]), at
    buf.close()


@pytest.mark.parametrize("n", [2, 65])
@pytest.mark.parametrize("kind", ["nopacking", "respond"])
def test_responses_off_their_words(world, kind, n):
    W = world
    pick = np.arange(n) % 3
    rows = W["inspire"].PinnedBuffer((n, 6, PLEN), np.uint64)
    rows.array[...] = W["b_rows"][pick]
    raw = W["inspire"].PinnedBuffer((8 * n * 2 * PLEN + 16,), np.uint8)
    for off in (4, 8):  # 8: words, but not the 16 bytes that some forms store
        raw.array[...] = 0
        out = np.frombuffer(raw.array.data, dtype=np.uint64, count=n * 2 * PLEN, offset=off)
        call(W, kind, n, rows.array, out)
        assert np.array_equal(out.reshape(n, 2, PLEN), W[kind][pick]), off
        assert not raw.array[:off].any() and not raw.array[off + 8 * n * 2 * PLEN:].any()
    del out
    rows.close()
    raw.close()


@pytest.mark.parametrize("n", [2, 33])
def test_tree_over_the_rows(world, n):
    W = world
    pick = np.arange(n) % 3
    buf = W["inspire"].PinnedBuffer((n, 6, PLEN), np.uint64)
    flat = buf.array.reshape(-1)
    for at in (0, flat.size - n * 3 * PLEN):
        buf.array[...] = W["b_rows"][pick]
        out_a = flat[at:at + n * PLEN].reshape(n, PLEN)
        out_b = flat[at + n * PLEN:at + 3 * n * PLEN].reshape(n, 2 * PLEN)
        a, b = W["inspire"].respond_seeded_packed_batch(W["crs"], W["edb"], np.array(W["shards"])[pick],
                                                        W["seeds"][pick], buf.array, out_a, out_b)
        for i in range(n):
            wa, wb = W["tree"][i % 3]
            assert np.array_equal(a[i], wa) and np.array_equal(b[i], np.asarray(wb)[:b.shape[1]]), (at, i)
    buf.close()
