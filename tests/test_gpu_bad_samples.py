"""User input functions that turn NaN or infinite: the outputs before the first
step that reads such a sample are those of the same solve with a function that
stays finite, wherever the sample falls in its block and window.
"""
import numpy as np
import pytest

from oracle import oracle
from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu

H = 1e-3
GOOD = "fType UFunc(fType t, int i) { return sin(t * (fType)3 + i)%s; }"
KINDS = {"nan": " + (t > (fType)%r ? (fType)0 / (t - t) : (fType)0)", "inf": " + (t > (fType)%r ? (fType)1 / (t - t) : (fType)0)",
         "one": " + (fabs(t - (fType)%r) < (fType)3e-4 ? (fType)-1 / (t - t) : (fType)0)"}
CASES = [  # solver, n, m, p, precision
    (0, 8, 2, 2, 0), (0, 16, 1, 3, 0), (0, 30, 3, 2, 0), (0, 64, 2, 1, 0), (0, 64, 5, 8, 0), (1, 4, 2, 2, 0), (1, 16, 1, 2, 0),
    (0, 16, 1, 2, 1), (0, 32, 4, 4, 1), (0, 64, 3, 9, 1), (1, 8, 2, 2, 1), (1, 16, 1, 1, 1),
]


def _solve(pb, c, source, precision, T):
    plan = pb.Plan(c.A, c.B, c.C, c.D, c.x0, pb.register_input(source), c.t0, c.t_end, c.h, solver=c.solver, precision=precision)
    plan.execute()
    plan.execute()
    _, y = plan.output()
    plan.close()
    return y


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("solver,n,m,p,precision", CASES)
def test_outputs_before_a_bad_sample(pb, solver, n, m, p, precision, kind):
    T = 700
    c = wl.small(77000 + n, solver, n, m, p, T, h=H)
    ref = oracle.simulate_affine(oracle.System(c.A, c.B, c.C, c.D, c.x0), oracle.Input.callable(lambda t, i: np.sin(3.0 * t + i)),
                                 solver, c.t0, c.t_end, c.h)
    # first bad sample at half step 2 k - 1 or at step k: output k is the first that its state or its input spoils
    for k, half in ((9, 0), (320, 0), (320, 1), (321, 0), (335, 1), (336, 0), (343, 0), (640, 1)):
        t1 = (k - 0.5 * half) * H
        if kind == "one" and half and solver == 1:
            continue  # no sample there
        at = t1 if kind == "one" else t1 - 1e-4
        y = _solve(pb, c, GOOD % (KINDS[kind] % at), precision, T)
        d = np.max(np.abs(y[:k] - ref[:k])) / np.max(np.abs(ref))
        assert d <= (1e-12 if precision == 0 else 1e-6), (k, half, d)
        assert not np.all(np.isfinite(y[k])), (k, half)


def test_ranges_of_a_one_shot_solve(pb):
    T, p = 130_000, 9  # y long enough to be copied out range by range
    c = wl.small(77100, 0, 16, 2, p, T, h=H)
    for k in (3, 16 * 1015 + 1, 16 * 1016, 100_001):
        t, y = pb.simulate(c.A, c.B, c.C, c.D, c.x0, pb.register_input(GOOD % (KINDS["nan"] % (k * H - 1e-4))), c.t0, c.t_end, c.h)
        assert np.all(np.isfinite(y[:k])) and not np.all(np.isfinite(y[k]))


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("solver,n,m,p,precision", CASES[:3] + CASES[5:9] + CASES[10:11])
def test_without_B_only_its_own_step(pb, solver, n, m, p, precision, kind):
    """Without B a sample enters the output of its own step alone."""
    T, k = 700, 337
    c = wl.small(77200 + n, solver, n, m, p, T, h=H)
    ref = oracle.simulate_affine(oracle.System(c.A, None, c.C, c.D, c.x0), oracle.Input.callable(lambda t, i: np.sin(3.0 * t + i)),
                                 solver, c.t0, c.t_end, c.h)
    c.B = None
    y = _solve(pb, c, GOOD % (KINDS[kind] % (k * H if kind == "one" else k * H - 1e-4)), precision, T)
    good = np.arange(T) != k if kind == "one" else np.arange(T) < k
    d = np.max(np.abs(y[good] - ref[good])) / np.max(np.abs(ref))
    assert d <= (1e-12 if precision == 0 else 1e-6), d
    assert not np.any(np.isfinite(y[~good]))
