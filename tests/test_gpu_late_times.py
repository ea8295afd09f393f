"""Mixed solves with sinusoid inputs late on the time axis,
where rounded sample times and arguments differ from phases advanced by the
nominal step by more than the form's error.  They agree with the FP64 form,
which samples at the rounded times, to the mixed gate of 1e-6; before that
point the inputs enter as phases.
"""
import numpy as np
import pytest

from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t0,phase", [(0.0, 0.0), (1e6, 0.0), (1e9, 0.0), (-1e9, 0.0), (0.0, 3e9)])
@pytest.mark.parametrize("solver,n", [(0, 24), (1, 12), (0, 96)])
def test_mixed_batch_agrees_with_fp64(pb, solver, n, t0, phase):
    c = wl.small(74000 + n, solver, n, 3, 3, 3000, h=1e-3)
    u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi + phase)
    spec = dict(A=c.A, B=c.B, C=c.C, D=c.D, x0=c.x0, u=u, t0=t0, t_end=t0 + 2999.5e-3, h=c.h, solver=solver)
    y = []
    for precision in (0, 1):
        b = pb.Batch([spec] * 2, precision=precision)
        b.execute()
        y.append(b.output(1)[1])
        b.close()
    assert y[0].shape == y[1].shape
    assert np.max(np.max(np.abs(y[1] - y[0]), 0) / np.max(np.abs(y[0]), 0)) <= 1e-6


@pytest.mark.parametrize("t0", [0.0, 1e8, 1e9])
@pytest.mark.parametrize("solver,n,m,precision", [(0, 12, 3, 1), (0, 16, 1, 1), (0, 32, 4, 1), (0, 64, 8, 1), (1, 8, 2, 1), (0, 96, 4, 1),
                                                  (0, 24, 20, 1)])
def test_mixed_plan_agrees_with_fp64(pb, solver, n, m, precision, t0):
    c = wl.small(74500 + n, solver, n, m, 3, 3000, h=1e-3)
    u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi)
    y = []
    for form in (0, precision):
        plan = pb.Plan(c.A, c.B, c.C, c.D, c.x0, u, t0, t0 + 2999.5e-3, c.h, solver=solver, precision=form)
        plan.execute()
        y.append(plan.output()[1])
        plan.close()
    assert np.max(np.max(np.abs(y[1] - y[0]), 0) / np.max(np.abs(y[0]), 0)) <= 1e-6
