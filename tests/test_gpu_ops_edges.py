"""The batched transforms and external products at the edges of their kernels'
tiles (two polynomials per CTA, odd counts) and with the largest residues,
bit-exact against the oracle (src/math/ntt.rs:223-325,
src/rgsw/external_product.rs:88-150)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048


@pytest.fixture(scope="module")
def env(oracle_mod):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    return torch, inspire, inspire.ServerCrs(inspire.InspireParams(p=1 << 16), bytes(32), 16), oracle_mod.Ctx()


def _polys(rng, k, moduli):
    out = np.stack([rng.integers(0, q, size=(k, N), dtype=np.uint64) for q in moduli], axis=1)
    out[0] = np.array(moduli, np.uint64)[:, None] - 1  # the largest residues
    if k > 1:
        out[1] = 0
    return out


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.uint32).view(np.int32)).cuda()


@pytest.mark.parametrize("n", [1, 2, 3, 305, 913])
def test_ntt_counts(env, n):
    torch, inspire, crs, ctx = env
    polys = _polys(np.random.default_rng(n), n, crs.params.crt_moduli)
    guard = np.full((1, 2, N), 12345, np.uint64)  # nothing past the last polynomial is written
    d = _dev(torch, np.concatenate([polys, guard]))
    st = torch.cuda.current_stream().cuda_stream
    inspire.ntt_forward_device(crs, d.data_ptr(), n, st)
    got = d.cpu().numpy().view(np.uint32).reshape(n + 1, 2, N)
    assert np.array_equal(got[:n].astype(np.uint64), ctx.ntt_forward(polys.reshape(n, -1)).reshape(n, 2, N))
    inspire.ntt_inverse_device(crs, d.data_ptr(), n, st)
    back = d.cpu().numpy().view(np.uint32).reshape(n + 1, 2, N)
    assert np.array_equal(back[:n], polys)
    assert np.array_equal(back[n], guard[0])


@pytest.mark.parametrize("n", [1, 5])
def test_external_product_largest_residues(env, n):
    torch, inspire, crs, ctx = env
    rng = np.random.default_rng(n)
    cts = _polys(rng, 2 * n, crs.params.crt_moduli).reshape(n, 2, 2, N)
    rgsw = _polys(rng, 12 * n, crs.params.crt_moduli).reshape(n, 6, 2, 2, N)
    rgsw[0] = np.array(crs.params.crt_moduli, np.uint64)[:, None] - 1
    want = np.stack([ctx.external_product(c.reshape(2, -1), g.reshape(12, -1)) for c, g in zip(cts, rgsw)])
    dct, drg = _dev(torch, cts), _dev(torch, rgsw)
    dout = torch.zeros(n * 4 * N, dtype=torch.int32, device="cuda")
    inspire.external_product_device(crs, dct.data_ptr(), drg.data_ptr(), dout.data_ptr(), n,
                                    torch.cuda.current_stream().cuda_stream)
    got = dout.cpu().numpy().view(np.uint32).reshape(n, 2, 2 * N)
    assert np.array_equal(got.astype(np.uint64), want.reshape(n, 2, 2 * N))
