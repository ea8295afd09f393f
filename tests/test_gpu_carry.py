"""The chunked carry of the blocks (kernels_carry.cu) at its edges: every padded
scan dimension, block counts around whole chunks (16 blocks), tiles (2 chunks),
whole CTAs (8 chunks) and the two-level top (256 blocks), and enough chunks that
a CTA of the upper levels takes several tiles.

An entry of the carry is a sum over the scan dimension at each of at most 16
steps a level: gate 1e-12 per channel against the oracle, and 1e-11 between the
blocked and the level-synchronous scan, which round in different orders.
"""
import pytest

from oracle import oracle
from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu

DIMS = [(0, 5), (0, 16), (0, 20), (1, 8), (0, 40), (1, 12), (0, 50), (0, 64)]  # scan dimensions 8, 16, .. 64


def _plan(pb, c):
    u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi)
    return pb.Plan(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, solver=c.solver, precision=pb.FP64)


@pytest.mark.parametrize("blocks", [1, 15, 16, 17, 33, 128, 129, 256, 257, 16 * 128 + 1])
@pytest.mark.parametrize("solver,n", DIMS)
def test_carry_matches_oracle(pb, solver, n, blocks):
    T = 16 * blocks - 3 + (3 if solver else 0)
    c = wl.small(41000 + 10 * n + blocks, solver, n, 2, 3, T, h=1e-3)
    plan = _plan(pb, c)
    assert plan.path == pb.PATH_BLOCKED_RESPONSE
    plan.execute()
    _, y = plan.output()
    plan.close()
    ref = oracle.simulate_affine(oracle.System(c.A, c.B, c.C, c.D, c.x0), oracle.Input.sinusoid(c.u.a, c.u.f, c.u.phi),
                                 solver, c.t0, c.t_end, c.h)
    assert y.shape == ref.shape
    assert oracle.rel_err(y, ref) <= 1e-12


@pytest.mark.parametrize("n", [30, 57])
def test_many_chunks_match_the_level_scan(pb, n):
    c = wl.small(42000 + n, 0, n, 1, 1, 16 * 16 * 32 * 148 + 16 * 300 + 5, h=1e-4)
    out = []
    for path in (0, 1):
        pb.set_option(pb.OPT_PATH, path)
        try:
            plan = _plan(pb, c)
        finally:
            pb.set_option(pb.OPT_PATH, 0)
        plan.execute()
        out.append(plan.output()[1])
        plan.close()
    assert oracle.rel_err(out[0], out[1]) <= 1e-11
