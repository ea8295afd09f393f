"""The chunked general scan (kernels_general.cu) against the sequential FP64
recurrence: scan dimensions around the multiples of 8 (one warp per chunk up
to 16, a CTA above), map counts around the chunk length and its powers (the
levels), maps not on a 16-byte boundary, absent V and x0, and X in place of V.

Tolerance 1e-12 per channel in both precision forms (the arithmetic is FP64 in
both): up to 4097 maps near the identity, each step rounding at 1e-16.
"""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _maps(ns, count, seed):
    rng = np.random.default_rng(seed)
    M = 0.01 / np.sqrt(ns) * rng.standard_normal((count, ns, ns))
    M[:, np.arange(ns), np.arange(ns)] += 0.99
    return M, rng.standard_normal((count, ns)), rng.standard_normal(ns)


def _recurrence(M, V, x0):
    X = np.empty((M.shape[0], M.shape[1]))
    x = np.zeros(M.shape[1]) if x0 is None else x0
    for k in range(len(M)):
        X[k] = x
        x = M[k] @ x + (0.0 if V is None else V[k])
    return X


def _scan(pb, M, V, x0, precision, shift=0, in_place=False):
    import torch

    count, ns = M.shape[:2]
    dev = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()
    buf = torch.zeros(M.size + 1, dtype=torch.float64, device="cuda")
    dM = buf[shift:shift + M.size]
    dM.copy_(dev(M).reshape(-1))
    dV, dx = dev(V), dev(x0)
    out = torch.full((count * ns + 16,), float("nan"), dtype=torch.float64, device="cuda")
    dX = dV if in_place else out[:count * ns]
    torch.cuda.synchronize()
    ptr = lambda t: 0 if t is None else t.data_ptr()
    pb.affine_scan_general(ptr(dM), ptr(dV), ptr(dx), ns, count, ptr(dX), precision)
    assert bool(torch.isnan(out[count * ns:]).all())
    return dX.cpu().numpy().reshape(count, ns)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ns,count", [(1, 1), (1, 17), (7, 16), (8, 257), (9, 15), (15, 33), (16, 4097), (17, 256), (24, 272),
                                      (25, 31), (33, 100), (40, 289), (41, 16), (48, 65), (56, 33), (57, 300), (63, 18),
                                      (64, 273)])
def test_scan_matches_recurrence(pb, ns, count, precision):
    M, V, x0 = _maps(ns, count, 100 * ns + count)
    assert oracle.rel_err(_scan(pb, M, V, x0, precision), _recurrence(M, V, x0)) <= TOL


@pytest.mark.parametrize("ns,count", [(8, 300), (16, 40), (20, 300), (64, 40)])
def test_absent_unaligned_and_in_place(pb, ns, count):
    M, V, x0 = _maps(ns, count, 7 * ns + count)
    assert oracle.rel_err(_scan(pb, M, None, x0, 0), _recurrence(M, None, x0)) <= TOL
    assert oracle.rel_err(_scan(pb, M, V, None, 0), _recurrence(M, V, None)) <= TOL
    ref = _recurrence(M, V, x0)
    assert oracle.rel_err(_scan(pb, M, V, x0, 0, shift=1), ref) <= TOL  # 8 bytes off a 16-byte boundary
    assert oracle.rel_err(_scan(pb, M, V, x0, 0, in_place=True), ref) <= TOL


def test_many_maps_use_longer_chunks(pb):
    """Enough maps for the 64-step chunks of the lowest level."""
    ns, count = 2, 1 << 18
    M, V, x0 = _maps(ns, count, 5)
    assert oracle.rel_err(_scan(pb, M, V, x0, 0), _recurrence(M, V, x0)) <= TOL
