"""Set-up of a plan: small systems discretised on the host and larger ones on
the device (the line lies at 20 thousand multiply-adds), constants sent in one
copy or, past its block, one by one, the ABM start-up on the host (sinusoids, no
input).  FP64, gate 1e-12 against the oracle,
whatever the leaf.  Batches formed by several threads at once share the set-up
threads and give the bits they give alone.
"""
import threading

import numpy as np
import pytest

from oracle import oracle
from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu

CASES = [  # solver, n, input, path
    (0, 18, "sin", 0), (0, 19, "sin", 0), (0, 18, "sin", 1), (0, 19, "none", 0), (0, 190, "sin", 0), (1, 1, "sin", 0),
    (1, 16, "sin", 3), (1, 26, "sin", 0), (1, 27, "sin", 1), (1, 14, "none", 0), (1, 60, "sin", 0),
]


@pytest.mark.parametrize("solver,n,kind,path", CASES)
def test_plan_matches_oracle(pb, solver, n, kind, path):
    c = wl.small(61000 + n, solver, n, 2, 3, 500 + n, h=1e-3)
    on = kind == "sin"
    u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi) if on else 0
    pb.set_option(pb.OPT_PATH, path)
    try:
        plan = pb.Plan(c.A, c.B if on else None, c.C, c.D if on else None, c.x0, u, c.t0, c.t_end, c.h, solver=solver,
                       precision=pb.FP64)
    finally:
        pb.set_option(pb.OPT_PATH, 0)
    plan.execute()
    _, y = plan.output()
    plan.close()
    ref = oracle.simulate_affine(oracle.System(c.A, c.B if on else None, c.C, c.D if on else None, c.x0),
                                 oracle.Input.sinusoid(c.u.a, c.u.f, c.u.phi) if on else oracle.Input.zero(), solver, c.t0,
                                 c.t_end, c.h)
    assert y.shape == ref.shape
    assert oracle.rel_err(y, ref) <= 1e-12


def test_batches_formed_by_several_threads(pb):
    sets = []
    for k in range(4):
        cases = [wl.small(62000 + 10 * k + i, i % 2, 3 + 7 * i, 2, 2, 400 + 50 * i, h=1e-3) for i in range(6)]
        sets.append([dict(A=c.A, B=c.B, C=c.C, D=c.D, x0=c.x0, u=pb.register_sinusoid(c.u.a, c.u.f, c.u.phi), t0=c.t0,
                          t_end=c.t_end, h=c.h, solver=c.solver) for c in cases])

    def solve(specs):
        b = pb.Batch(specs, precision=pb.FP64)
        b.execute()
        out = [b.output(i)[1] for i in range(len(specs))]
        b.close()
        return out

    alone = [solve(s) for s in sets]
    got = [None] * 4

    def work(k):
        for _ in range(5):
            got[k] = solve(sets[k])

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for k in range(4):
        assert got[k] is not None
        for a, b in zip(alone[k], got[k]):
            assert np.array_equal(a, b)
