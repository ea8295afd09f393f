"""Batches whose scan levels mix the kernels: scan dimensions up to 64 (one
launch for all of them, on their own stream), above 64 in 64 x 64 tiles, in
32 x 32 tiles when a launch has few, and in 8-row CTAs when a level has few
columns.

Dimensions at the edges of the tiles (8 .. 64, 72, 96, 136, 512), lengths with
1, 2, 31 .. 33 and some thousand items.  Every form adds FP64 products over the
scan dimension, so an element carries at most about 600 roundings of a state's
peak; gate 1e-11 against the oracle.
"""
import pytest

from oracle import oracle
from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu

SETS = [  # (solver, n, m, p, T) of one batch
    [(0, 8, 1, 2, 700), (0, 17, 2, 3, 40), (0, 64, 3, 4, 1500), (0, 65, 2, 3, 33), (0, 96, 1, 9, 2500), (1, 5, 2, 3, 600)],
    [(1, 2, 1, 1, 900), (1, 16, 2, 4, 520), (1, 18, 1, 2, 1025), (1, 34, 3, 5, 517), (1, 128, 2, 3, 70)],
    [(0, 136, 2, 2, 16 * 33 + 1), (0, 72, 1, 72, 16 * 31)],
    [(0, 9, 2, 2, 3000), (1, 12, 1, 3, 5)],
]


@pytest.mark.parametrize("path", [0, 1])
@pytest.mark.parametrize("k", range(len(SETS)))
def test_levels_match_oracle(pb, k, path):
    cases = [wl.small(31000 + 100 * k + i, s, n, m, p, T, h=1e-3) for i, (s, n, m, p, T) in enumerate(SETS[k])]
    pb.set_option(pb.OPT_PATH, path)
    try:
        specs = [dict(A=c.A, B=c.B, C=c.C, D=c.D, x0=c.x0, u=pb.register_sinusoid(c.u.a, c.u.f, c.u.phi), solver=c.solver,
                      t0=c.t0, t_end=c.t_end, h=c.h) for c in cases]
        batch = pb.Batch(specs, precision=pb.FP64)
    finally:
        pb.set_option(pb.OPT_PATH, 0)
    for rep in range(3):  # launched twice, then replayed as a graph
        batch.execute()
        for i, c in enumerate(cases):
            _, y = batch.output(i)
            ref = oracle.simulate_affine(oracle.System(c.A, c.B, c.C, c.D, c.x0), oracle.Input.sinusoid(c.u.a, c.u.f, c.u.phi),
                                         c.solver, c.t0, c.t_end, c.h)
            assert y.shape == ref.shape
            assert oracle.rel_err(y, ref) <= 1e-11, (i, rep)
    batch.close()


def test_many_systems_in_one_launch(pb):
    """A batch whose levels are launches of thousands of tiles: entries found
    among several hundred, a row tile per warp in the narrow kernel, 32-row
    tiles where 64 would be padding.  Mixed form (the expansion, FP64 phases):
    gate 1e-10, as for its single plans."""
    cases = [wl.small(33000 + i, i % 2, 3 + (7 * i) % 60, 1 + i % 3, 2, 1500 + 37 * (i % 41), h=1e-3) for i in range(400)]
    specs = [dict(A=c.A, B=c.B, C=c.C, D=c.D, x0=c.x0, u=pb.register_sinusoid(c.u.a, c.u.f, c.u.phi), solver=c.solver,
                  t0=c.t0, t_end=c.t_end, h=c.h) for c in cases]
    batch = pb.Batch(specs, precision=pb.MIXED)
    batch.execute()
    for i in list(range(0, 400, 23)) + [1, 398, 399]:
        c = cases[i]
        _, y = batch.output(i)
        ref = oracle.simulate_affine(oracle.System(c.A, c.B, c.C, c.D, c.x0), oracle.Input.sinusoid(c.u.a, c.u.f, c.u.phi),
                                     c.solver, c.t0, c.t_end, c.h)
        assert y.shape == ref.shape
        assert oracle.rel_err(y, ref) <= 1e-10, i
    batch.close()
