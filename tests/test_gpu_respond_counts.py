"""Batches around the SM count, where the one-CTA Respond kernel changes its
form, with CRT moduli at the ends of the transforms' lazy ranges, bit-exact
against the oracle (src/pir/respond.rs:284-398)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
MODULI = {"default": (268369921, 249561089), "half of the draws rejected": (134246401, 134250497),
          "just above 2^20": (1073153, 1093633)}


@pytest.mark.parametrize("entry", [2, 32])
@pytest.mark.parametrize("mode", ["crt_fixed", "compat"])
@pytest.mark.parametrize("which", list(MODULI))
def test_respond_counts(oracle_mod, which, mode, entry):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    O, moduli = oracle_mod, MODULI[which]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(entry)
    ctx = O.Ctx(moduli=moduli)
    omode = O.MODE_CRT_FIXED if mode == "crt_fixed" else O.MODE_COMPAT
    pack = O.Pack(ctx, entry // 2, bytes(32), mode=omode)
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16, crt_moduli=moduli), bytes(32), entry // 2, mode=mode)
    db = rng.integers(0, 256, size=(N + 700) * entry, dtype=np.uint8)
    edb = inspire.EncodedDatabase(crs, db, entry)
    k = 3
    polys = lambda m: np.concatenate([rng.integers(0, q, size=(m, N), dtype=np.uint64) for q in moduli], axis=1)  # noqa: E731
    b_rows = polys(6 * k).reshape(k, 6, 2 * N)
    b_rows[0] = np.repeat(np.array(moduli, np.uint64) - 1, N)  # the largest residues
    y_body = polys(3)
    seeds = rng.integers(0, 256, size=(k, 6, 32), dtype=np.uint8)
    shards = [0, 1, 1]
    want = np.stack([ctx.respond_inspiring(ctx.encode_shard(db, entry, s), ctx.expand_rgsw(sd, br), bytes(32), mode=omode,
                                           pack=pack, y_body=y_body)
                     for s, sd, br in zip(shards, seeds, b_rows)])
    cid = crs.register_client(inspire.ClientPackingKeys(y_body=y_body))
    for n in (sms // 2 + 1, sms, sms + 1):
        pick = np.arange(n) % k
        sid, sd, br = np.array(shards)[pick], seeds[pick], np.ascontiguousarray(b_rows[pick])
        assert np.array_equal(inspire.respond_seeded_batch(crs, edb, sid, sd, br, [cid] * n), want[pick])
        rows, out = inspire.PinnedBuffer(br.shape, np.uint64), inspire.PinnedBuffer((n, 2, 2 * N), np.uint64)
        rows.array[...] = br
        inspire.respond_seeded_batch(crs, edb, sid, sd, rows.array, [cid] * n, out.array)
        assert np.array_equal(out.array, want[pick])
        rows.close()
        out.close()


@pytest.mark.parametrize("captured", [False, True])
def test_overlapping_batches(captured):
    """Device batches of one query per SM on two streams at once, and captured
    into a graph, where the kernel keeps the form that shares an SM: the same
    responses as alone."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    n = torch.cuda.get_device_properties(0).multi_processor_count // 2 + 1
    rng = np.random.default_rng(n)
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16), bytes(32), 16)
    q = crs.params.crt_moduli
    polys = lambda *s: np.concatenate([rng.integers(0, m, size=(*s, N), dtype=np.uint64) for m in q], axis=-1)  # noqa: E731
    edb = inspire.EncodedDatabase(crs, rng.integers(0, 256, size=N * 32, dtype=np.uint8), 32)
    cid = crs.register_client(inspire.ClientPackingKeys(y_body=polys(3)))
    d = [torch.from_numpy(a).cuda() for a in (np.zeros(n, np.int32),
                                              rng.integers(0, 256, size=(n, 3, 32), dtype=np.uint8),
                                              polys(n, 3).view(np.int64), np.full(n, cid, np.int32))]
    outs = [torch.zeros((n, 2, 2 * N), dtype=torch.int64, device="cuda") for _ in range(5)]
    status = torch.full((5, n), -1, dtype=torch.int32, device="cuda")

    def batch(k, stream):
        inspire.respond_seeded_batch_device(crs, edb, n, *[t.data_ptr() for t in d], outs[k].data_ptr(),
                                            status[k].data_ptr(), stream.cuda_stream)

    batch(0, torch.cuda.current_stream())
    torch.cuda.synchronize()
    if captured:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for k in range(1, 5):
                batch(k, torch.cuda.current_stream())
        g.replay()
    else:
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        for k in range(1, 5):
            batch(k, streams[k & 1])
    torch.cuda.synchronize()
    assert not status.cpu().numpy().any()
    for o in outs[1:]:
        assert torch.equal(o, outs[0])
