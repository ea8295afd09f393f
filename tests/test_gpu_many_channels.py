"""Sampled solves whose output rows or response matrix do not fit the
block-response leaf, and the ones beside the line that do: every one of them
is solved (in-block sweeps or level by level past the line), to 1e-12 in FP64
and 1e-6 in the mixed form of the largest output, against the oracle: among
thousands of channels some nearly cancel, and their errors are those of the
products and not of the sums.
"""
import numpy as np
import pytest

from oracle import oracle
from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu

CASES = [  # solver, n, m, p, precision
    (0, 64, 1, 432, 0), (0, 64, 1, 440, 0), (0, 64, 1, 512, 0), (0, 64, 1, 512, 1), (0, 8, 1, 3500, 0), (0, 8, 1, 4000, 0),
    (0, 8, 1, 4000, 1), (1, 16, 2, 600, 0), (0, 20, 2, 1300, 0), (0, 64, 40, 600, 0), (0, 16, 2000, 2000, 0),
]


@pytest.mark.parametrize("kind", ["sin", "user"])
@pytest.mark.parametrize("solver,n,m,p,precision", CASES)
def test_many_channels_match_oracle(pb, solver, n, m, p, precision, kind):
    T = 300
    c = wl.small(70000 + n + p, solver, n, m, p, T, h=1e-3)
    if kind == "sin":
        u, inp = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi), oracle.Input.sinusoid(c.u.a, c.u.f, c.u.phi)
    else:
        u = pb.register_input("fType UFunc(fType t, int i) { return t * (fType)0.5 + (fType)(i % 7); }")
        inp = oracle.Input.callable(lambda t, i: 0.5 * t + i % 7)
    plan = pb.Plan(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, solver=solver, precision=precision)
    plan.execute()
    _, y = plan.output()
    plan.close()
    ref = oracle.simulate_affine(oracle.System(c.A, c.B, c.C, c.D, c.x0), inp, solver, c.t0, c.t_end, c.h)
    assert y.shape == ref.shape
    assert np.max(np.abs(y - ref)) <= (1e-12 if precision == 0 else 1e-6) * np.max(np.abs(ref))
