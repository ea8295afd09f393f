"""FP64 samples of sinusoid inputs at the ends of the single-precision range.

The run's recurrence corrects the rounding of the sample arguments in single
precision, so amplitudes that a float does not hold take another form.  The
solve starts late (t0 = 5e4), where the arguments' roundings are up to 4e-10 of
the amplitude, far above the gate of 1e-12 against the oracle.
"""
import numpy as np
import pytest

from oracle import oracle
from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 2.0 ** 140, 2.0 ** 66, 2.0 ** -66, 2.0 ** -140, 2.0 ** -170])
@pytest.mark.parametrize("solver,batch", [(0, False), (1, False), (0, True)])
def test_amplitudes_over_the_float_range(pb, solver, batch, scale):
    c = wl.small(66000, solver, 6, 2, 2, 2500, h=1e-3)
    a = c.u.a * scale
    a[0, 1] = 0.0
    u = pb.register_sinusoid(a, c.u.f, c.u.phi)
    x0, t0 = c.x0 * scale, 5e4
    t_end = t0 + (2500 - 0.5) * c.h
    if batch:
        b = pb.Batch([dict(A=c.A, B=c.B, C=c.C, D=c.D, x0=x0, u=u, t0=t0, t_end=t_end, h=c.h, solver=solver)] * 2,
                     precision=pb.FP64)
        b.execute()
        _, y = b.output(1)
        b.close()
    else:
        plan = pb.Plan(c.A, c.B, c.C, c.D, x0, u, t0, t_end, c.h, solver=solver, precision=pb.FP64)
        plan.execute()
        _, y = plan.output()
        plan.close()
    ref = oracle.simulate_affine(oracle.System(c.A, c.B, c.C, c.D, x0), oracle.Input.sinusoid(a, c.u.f, c.u.phi), solver,
                                 t0, t_end, c.h)
    assert y.shape == ref.shape and np.all(np.isfinite(y))
    # scaled by a power of two, which is exact
    assert oracle.rel_err(y / scale, ref / scale) <= 1e-12
