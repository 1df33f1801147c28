"""The two-CTA Respond kernel's bounded wait for the other CTA's coefficients,
made to run out at the first step: every query ends with that status (5) and
not with that of stores still in flight (6), through device batches, host calls
and the serving loop, and the next launches on the same context are answered
correctly.  One column has no step and no wait."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
PLEN = 2 * N
DEFAULT = 1 << 20


@pytest.mark.parametrize("mode", ["crt_fixed", "compat"])
@pytest.mark.parametrize("gamma", [1, 2, 4, 16])
def test_peer_wait_running_out(oracle_mod, gamma, mode):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    omode = oracle_mod.MODE_COMPAT if mode == "compat" else oracle_mod.MODE_CRT_FIXED
    rng = np.random.default_rng(gamma)
    ctx = oracle_mod.Ctx()
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16), bytes(32), gamma, mode=mode)
    db = rng.integers(0, 256, size=2 * N * 2 * gamma, dtype=np.uint8)
    edb = inspire.EncodedDatabase(crs, db, 2 * gamma)
    pack = oracle_mod.Pack(ctx, gamma, bytes(32), mode=omode)
    client = oracle_mod.Client(ctx, seed=0, rng_seed=gamma)
    y_body, _ = client.packing_keys(pack)
    cid = crs.register_client(inspire.ClientPackingKeys(y_body=y_body))
    n = 5
    seeds, b_rows = zip(*[client.query_seeded(i) for i in (0, 5, 700, 2046, 2047)])
    seeds, b_rows = np.stack(seeds), np.stack([b.reshape(6, PLEN) for b in b_rows])
    shard = ctx.encode_shard(db, 2 * gamma, 1)
    want = np.stack([ctx.respond_inspiring(shard, ctx.expand_rgsw(s, b), bytes(32), mode=omode, pack=pack,
                                           y_body=y_body) for s, b in zip(seeds, b_rows)])
    sid = torch.ones(n, dtype=torch.int32, device="cuda")
    sd = torch.from_numpy(np.ascontiguousarray(seeds[:, 3:])).cuda()
    br = torch.from_numpy(np.ascontiguousarray(b_rows[:, 3:]).view(np.int64)).cuda()
    cl = torch.full((n,), cid, dtype=torch.int32, device="cuda")
    srv = inspire.Server(crs, max_batch=8, max_inflight=2, capacity=16)

    def device_batch():
        out = torch.zeros((n, 2, PLEN), dtype=torch.int64, device="cuda")
        status = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        inspire.respond_seeded_batch_device(crs, edb, n, sid.data_ptr(), sd.data_ptr(), br.data_ptr(), cl.data_ptr(),
                                            out.data_ptr(), status.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return out.cpu().numpy().view(np.uint64), status.tolist()

    def submit():
        tickets, rc = srv.submit([edb] * n, [1] * n, seeds, b_rows, [cid] * n)
        assert rc == 0
        return tickets

    assert crs.L.inspire_ctx_set_peer_wait_iters(crs.h, 0) == 0
    out, status = device_batch()
    if gamma == 1:
        assert status == [0] * n and np.array_equal(out, want)
    else:
        assert status == [5] * n
        with pytest.raises(inspire.PirError, match="kernel status 5 for query 0"):
            inspire.respond_seeded_batch(crs, edb, [1] * n, seeds, b_rows, [cid] * n)
        for t in submit():
            with pytest.raises(inspire.PirError, match="kernel status 5"):
                srv.poll(int(t), np.zeros((2, PLEN), np.uint64))
    assert crs.L.inspire_ctx_set_peer_wait_iters(crs.h, DEFAULT) == 0
    for _ in range(2):
        out, status = device_batch()
        assert status == [0] * n and np.array_equal(out, want)
        assert np.array_equal(inspire.respond_seeded_batch(crs, edb, [1] * n, seeds, b_rows, [cid] * n), want)
        got = np.zeros((n, 2, PLEN), np.uint64)
        srv.poll_batch(submit(), got)
        assert np.array_equal(got, want)
    srv.close()
