"""The general scan reads the caller's arrays and nothing beside them: with
NaN on both sides of x0, the maps and the vectors the states are those of the
scan with arrays of their own, at dimensions that are padded inside and with
one, two and three levels of chunks.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [1, 5, 8, 13, 16, 20, 33, 63])
@pytest.mark.parametrize("count", [10, 200, 5000])
def test_nothing_beside_the_inputs_is_read(pb, ns, count):
    import torch

    g = torch.Generator(device="cuda").manual_seed(69000 + ns)
    r = lambda *s: torch.randn(s, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    M = r(count, ns, ns) * (0.3 / ns ** 0.5) + 0.6 * torch.eye(ns, dtype=torch.float64, device="cuda")
    V, x0, X = r(count, ns), r(ns), torch.empty((count, ns), dtype=torch.float64, device="cuda")

    def framed(v):
        b = torch.full((v.numel() + 256,), float("nan"), dtype=torch.float64, device="cuda")
        b[128:128 + v.numel()] = v.reshape(-1)
        return b, b.data_ptr() + 8 * 128

    (fm, pm), (fv, pv), (fx, px) = framed(M), framed(V), framed(x0)
    torch.cuda.synchronize()
    pb.affine_scan_general(pm, pv, px, ns, count, X.data_ptr())
    x, m, v = x0.cpu().numpy(), M.cpu().numpy(), V.cpu().numpy()
    ref = np.empty((count, ns))
    for k in range(count):
        ref[k] = x
        x = m[k] @ x + v[k]
    got = X.cpu().numpy()
    assert np.all(np.isfinite(got))
    # stable maps (spectral radius about 0.9): errors stay at some hundred roundings of the largest state
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
