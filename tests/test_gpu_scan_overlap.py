"""The general scan with its states written over its own inputs: over the maps,
over the vectors at the same and at other offsets, and with x0 inside.  The
states are those of the scan with separate arrays, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,count", [(1, 9), (5, 16), (5, 700), (16, 20000), (24, 3000), (64, 300)])
def test_states_over_the_inputs(pb, ns, count):
    import torch

    g = torch.Generator(device="cuda").manual_seed(68000 + ns)
    r = lambda *s: torch.randn(s, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    M = r(count, ns, ns) * (0.3 / ns ** 0.5) + 0.6 * torch.eye(ns, dtype=torch.float64, device="cuda")
    V, x0 = r(count, ns), r(ns)
    nm, nv = count * ns * ns, count * ns
    sep = torch.empty_like(V)
    pb.affine_scan_general(M.data_ptr(), V.data_ptr(), x0.data_ptr(), ns, count, sep.data_ptr())
    torch.cuda.synchronize()

    # one buffer: room | x0 | M | V | room, and where X starts in it
    at_x0, at_m = nv, nv + 64
    at_v = at_m + nm
    starts = {"maps": at_m, "end of maps": at_m + nm - nv, "maps and vectors": at_v - ns * (count // 2 + 1), "vectors": at_v,
              "vectors, one step on": at_v + ns, "vectors, one step back": at_v - ns, "x0 first": at_x0,
              "x0 last": at_x0 + ns - nv, "vectors, one value on": at_v + 1}
    for name, at in starts.items():
        buf = torch.full((at_v + 2 * nv + 64,), float("nan"), dtype=torch.float64, device="cuda")
        buf[at_x0:at_x0 + ns], buf[at_m:at_v], buf[at_v:at_v + nv] = x0, M.reshape(-1), V.reshape(-1)
        torch.cuda.synchronize()
        p = lambda k: buf.data_ptr() + 8 * k  # noqa: E731
        pb.affine_scan_general(p(at_m), p(at_v), p(at_x0), ns, count, p(at))
        torch.cuda.synchronize()
        assert np.array_equal(buf[at:at + nv].cpu().numpy(), sep.reshape(-1).cpu().numpy()), name
