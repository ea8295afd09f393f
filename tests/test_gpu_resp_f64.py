"""The FP64 outputs of the response leaf (kernels_resp_f64.cu) and the sample
recurrence, at their edges.

Outputs: many row slices (y = x with 64 states), one row, windows of odd and
even widths, block counts around the tiles of 8 and 16, an output buffer 8
bytes off a 16-byte boundary, a W too wide for shared memory (the tiled GEMM
takes it).  Gate: 1e-12 per channel against the oracle.

Samples: y = D u alone, so an error of a sample is an error of y.  A run of up
to 64 samples keeps each term within about 64 roundings (1e-14 of its
amplitude); with at most 6 terms on a peak of at least a tenth of their sum the
bound is 6e-13.  Nominal steps above 1 and arguments above 1e7 take the
rotation.
"""
import numpy as np
import pytest

from oracle import oracle
from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu

CASES = [  # solver, n, m, p, T, y = x
    (0, 64, 3, 64, 16 * 40 + 5, True), (0, 64, 8, 1, 16 * 8 * 148 + 9, False), (0, 10, 1, 7, 16 * 7, False), (0, 33, 5, 33, 16 * 9 - 1, True),
    (0, 64, 24, 24, 3000, False), (0, 8, 64, 8, 2000, False), (1, 16, 7, 5, 16 * 15 + 3, False), (1, 3, 1, 3, 16 * 16 + 4, True),
    (1, 16, 2, 9, 40_003, False),
]


@pytest.mark.parametrize("solver,n,m,p,T,state", CASES)
def test_outputs_match_oracle(pb, solver, n, m, p, T, state):
    import torch

    c = wl.small(23000 + n + T, solver, n, m, p, T, h=1e-3)
    u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi)
    Cm, D = (None, None) if state else (c.C, c.D)
    plan = pb.Plan(c.A, c.B, Cm, D, c.x0, u, c.t0, c.t_end, c.h, solver=solver, precision=pb.FP64)
    assert plan.path == pb.PATH_BLOCKED_RESPONSE
    ref = oracle.simulate_affine(oracle.System(c.A, c.B, Cm, D, c.x0), oracle.Input.sinusoid(c.u.a, c.u.f, c.u.phi), solver,
                                 c.t0, c.t_end, c.h)
    for offset in (0, 1):
        buf = torch.full((ref.size + 8,), float("nan"), dtype=torch.float64, device="cuda")
        plan.execute(buf[offset:].data_ptr())
        torch.cuda.synchronize()
        y = buf[offset:offset + ref.size].cpu().numpy().reshape(ref.shape)
        assert oracle.rel_err(y, ref) <= 1e-12, offset
        assert bool(torch.isnan(buf[offset + ref.size:]).all())
    plan.close()


@pytest.mark.parametrize("solver,T,h,t0,fmax,terms", [(0, 20_000, 1e-3, 0.0, 10.0, 3), (0, 70_001, 1e-4, 50.0, 10.0, 1),
                                                      (1, 5000, 1e-2, 0.0, 9.0, 4), (0, 3000, 0.1, 0.0, 12.0, 2),
                                                      (1, 2000, 1e-2, 3e6, 8.0, 3), (0, 100, 1e-3, -1.0, 5.0, 6)])
def test_samples_through_d(pb, solver, T, h, t0, fmax, terms):
    r = np.random.default_rng(T)
    m = 2
    a, f, phi = r.uniform(0.2, 1.0, (m, terms)), r.uniform(0.1, fmax, (m, terms)), r.uniform(0.0, 6.28, (m, terms))
    D, x0 = np.eye(m), np.ones(1)
    A = np.array([[-1.0]])
    t_end = t0 + (T - 0.5) * h
    u = pb.register_sinusoid(a, f, phi)
    plan = pb.Plan(A, None, None, D, x0, u, t0, t_end, h, solver=solver, precision=pb.FP64)
    plan.execute()
    _, y = plan.output()
    plan.close()
    ref = oracle.simulate_affine(oracle.System(A, None, None, D, x0), oracle.Input.sinusoid(a, f, phi), solver, t0, t_end, h)
    assert y.shape == ref.shape
    assert oracle.rel_err(y, ref) <= 6e-13
