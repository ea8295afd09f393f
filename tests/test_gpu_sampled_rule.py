"""Solves with sampled inputs take the block-response leaf at every scan
dimension, any number of inputs, with short sample runs on short horizons, and
one-shot calls copy a long y out by ranges and a short one at once.

Gates: FP64 1e-12 and mixed 1e-6 per channel against the oracle; the one-shot
call equals the plan bit for bit.
"""
import numpy as np
import pytest

from oracle import oracle
from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu

SRC = ("fType UFunc(fType t, int i) {\n    fType x = t * (fType)0.0625;\n    x = x - floor(x);\n"
       "    return i % 2 ? (x < 0.5 ? (fType)1 : (fType)-1) : x;\n}\n")


def _user(t, i):
    x = t * 0.0625
    x -= np.floor(x)
    return (1.0 if x < 0.5 else -1.0) if i % 2 else x


CASES = [  # solver, n, m, p, T
    (0, 1, 1, 1, 1), (0, 1, 1, 1, 2), (0, 3, 2, 1, 9), (0, 8, 2, 2, 17), (0, 8, 1, 3, 4096), (0, 16, 3, 5, 1000), (0, 32, 2, 1, 4097),
    (0, 64, 16, 2, 3000), (0, 64, 40, 3, 700), (0, 57, 5, 8, 32768), (1, 1, 1, 1, 4), (1, 2, 3, 2, 1000), (1, 4, 1, 3, 33),
    (1, 16, 15, 3, 5000),
]


@pytest.mark.parametrize("solver,n,m,p,T", CASES)
def test_fp64_and_mixed_match_oracle(pb, solver, n, m, p, T):
    c = wl.small(21000 + n + T, solver, n, m, p, T, h=1e-3)
    u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi)
    uu = pb.register_input(SRC)
    sysd = oracle.System(c.A, c.B, c.C, c.D, c.x0)
    sin = oracle.simulate_affine(sysd, oracle.Input.sinusoid(c.u.a, c.u.f, c.u.phi), solver, c.t0, c.t_end, c.h)
    usr = oracle.simulate_affine(sysd, oracle.Input.callable(_user), solver, c.t0, c.t_end, c.h)
    dim = c.scan_dim
    for ui, ref, precision in ((u, sin, pb.FP64), (uu, usr, pb.FP64), (uu, usr, pb.MIXED)):
        plan = pb.Plan(c.A, c.B, c.C, c.D, c.x0, ui, c.t0, c.t_end, c.h, solver=solver, precision=precision)
        assert plan.path == pb.PATH_BLOCKED_RESPONSE
        assert plan.precision == (pb.MIXED if precision == pb.MIXED and dim > 8 else pb.FP64)
        plan.execute()
        _, y = plan.output()
        plan.close()
        assert oracle.rel_err(y, ref) <= (1e-12 if precision == pb.FP64 or dim <= 8 else 1e-6)
        _, y1 = pb.simulate(c.A, c.B, c.C, c.D, c.x0, ui, c.t0, c.t_end, c.h, solver=solver, precision=precision)
        assert np.array_equal(y, y1)


@pytest.mark.parametrize("solver,n,T,precision", [(0, 64, 300_001, 0), (0, 24, 300_001, 1), (1, 16, 300_003, 2)])
def test_long_outputs_by_ranges_equal_plan(pb, solver, n, T, precision):
    """y of 19 MB (9.6 MB as float): copied out by ranges."""
    c = wl.small(22000 + n, solver, n, 4, 8, T, h=1e-3)
    u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi) if precision != 1 else pb.register_input(SRC)
    plan = pb.Plan(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, solver=solver, precision=precision)
    plan.execute()
    _, y = plan.output()
    plan.close()
    _, y1 = pb.simulate(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, solver=solver, precision=precision)
    assert np.array_equal(y, y1)
    f = lambda a: np.asarray(a, dtype=np.float32).astype(np.float64)
    if precision != 1:  # the float call compiles a user input for float
        plan = pb.Plan(f(c.A), f(c.B), f(c.C), f(c.D), f(c.x0), u, c.t0, c.t_end, c.h, solver=solver, precision=precision)
        plan.execute()
        _, y = plan.output()
        plan.close()
        pb.set_option(pb.OPT_PRECISION, precision)
        try:
            _, y32, err = pb.simulate_f32(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, solver=solver)
        finally:
            pb.set_option(pb.OPT_PRECISION, pb.FP64)
        assert err == 0 and np.array_equal(y32, y.astype(np.float32))
