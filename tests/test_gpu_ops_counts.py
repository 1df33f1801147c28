"""The batched transforms and external products at the counts where their
kernels change form (around the CTAs or SMs that the chip has), bit-exact
against the oracle (src/math/ntt.rs:223-325, src/rgsw/external_product.rs:88-150)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2048


@pytest.mark.parametrize("beyond", [0, 1])
def test_ops_counts(oracle_mod, beyond):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import inspire

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    crs, ctx = inspire.ServerCrs(inspire.InspireParams(p=1 << 16), bytes(32), 16), oracle_mod.Ctx()
    moduli = crs.params.crt_moduli
    rng = np.random.default_rng(beyond)
    polys = lambda *s: np.stack([rng.integers(0, q, size=(*s, N), dtype=np.uint64) for q in moduli], axis=-2)  # noqa: E731
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.uint32).view(np.int32)).cuda()  # noqa: E731
    st = torch.cuda.current_stream().cuda_stream
    n = 3 * sms + beyond
    a = polys(n)
    d = dev(a)
    inspire.ntt_forward_device(crs, d.data_ptr(), n, st)
    got = d.cpu().numpy().view(np.uint32).astype(np.uint64)
    assert np.array_equal(got, ctx.ntt_forward(a.reshape(n, -1)).reshape(n, 2, N))
    inspire.ntt_inverse_device(crs, d.data_ptr(), n, st)
    assert np.array_equal(d.cpu().numpy().view(np.uint32).astype(np.uint64), a)
    n, k = sms + beyond, 3
    ct, rgsw = polys(k, 2), polys(k, 6, 2)
    want = np.stack([ctx.external_product(c.reshape(2, -1), g.reshape(12, -1)) for c, g in zip(ct, rgsw)])
    pick = np.arange(n) % k
    out = torch.zeros(n * 4 * N, dtype=torch.int32, device="cuda")
    dct, drg = dev(ct[pick]), dev(rgsw[pick])
    inspire.external_product_device(crs, dct.data_ptr(), drg.data_ptr(), out.data_ptr(), n, st)
    got = out.cpu().numpy().view(np.uint32).astype(np.uint64).reshape(n, 2, 2 * N)
    assert np.array_equal(got, want[pick].reshape(n, 2, 2 * N))
