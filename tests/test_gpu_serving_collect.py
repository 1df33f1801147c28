"""Collecting many tickets at once: every response lands in its place whatever
the number of finished tickets (around the number from which the copies are
shared with helper threads), with several collectors at a time; a ticket that
was collected already ends the collected prefix."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048
ENTRY = 8


@pytest.mark.parametrize("capacity", [7, 130])  # without and with helper threads
def test_collect_batches(capacity):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    rng = np.random.default_rng(capacity)
    q = (268369921, 249561089)
    polys = lambda *s: np.concatenate([rng.integers(0, m, size=(*s, N), dtype=np.uint64) for m in q], axis=-1)  # noqa: E731
    crs = inspire.ServerCrs(inspire.InspireParams(p=1 << 16), bytes(32), ENTRY // 2)
    db = inspire.EncodedDatabase(crs, rng.integers(0, 256, size=N * ENTRY, dtype=np.uint8), ENTRY)
    cid = crs.register_client(inspire.ClientPackingKeys(y_body=polys(3)))
    n = 130
    seeds = rng.integers(0, 256, size=(n, 6, 32), dtype=np.uint8)
    rows = polys(n, 6)
    want = inspire.respond_seeded_batch(crs, db, [0] * n, seeds, rows, [cid] * n)
    srv = inspire.Server(crs, max_batch=min(32, capacity), max_inflight=3, capacity=capacity)

    def submit(lo, hi):
        t, rc = srv.submit(db, [0] * (hi - lo), seeds[lo:hi], rows[lo:hi], [cid] * (hi - lo))
        assert rc == 0 and len(t) == hi - lo
        return t

    for k in [c for c in (1, 7, 8, 9, 130) if c <= capacity]:
        out = np.zeros((k, 2, 2 * N), dtype=np.uint64)
        done = srv.poll_batch(submit(0, k), out)
        assert len(done) == k and (done > 0).all() and np.array_equal(out, want[:k])
    # without a place for the responses: the tickets are collected all the same
    assert len(srv.poll_batch(submit(0, 7))) == 7
    # the fourth ticket was collected before
    t = submit(0, 7)
    srv.poll(int(t[3]))
    out = np.zeros((7, 2, 2 * N), dtype=np.uint64)
    with pytest.raises(inspire.PirError, match="ticket"):
        srv.poll_batch(t, out)
    assert np.array_equal(out[:3], want[:3]) and not out[3:].any()
    assert len(srv.poll_batch(t[4:], out[4:])) == 3 and np.array_equal(out[4:], want[4:7])
    if capacity >= n:
        out = np.zeros((n, 2, 2 * N), dtype=np.uint64)
        parts = [(0, 40), (40, 80), (80, 130)]
        th = [threading.Thread(target=lambda lo, hi: srv.poll_batch(submit(lo, hi), out[lo:hi]), args=p) for p in parts]
        [x.start() for x in th]
        [x.join() for x in th]
        assert np.array_equal(out, want)
    srv.close()
