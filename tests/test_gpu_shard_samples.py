"""Time shards of solves with sinusoid inputs take the whole solve's samples:
runs of the same length, starting at the same samples of the horizon, so the
split equals the unsplit solve bit for bit, also where a shard's own samples
would be few enough for shorter runs and where it starts within a run.
"""
import numpy as np
import pytest

from parode_b200 import multi
from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu

CASES = [  # solver, n, m, p, T, shards, precision: runs of 8 to 64 in the whole, shards at odd multiples of a block
    (0, 8, 1, 1, 3000, 3, 0), (1, 4, 2, 2, 40000, 3, 0), (0, 16, 16, 2, 150000, 5, 0), (1, 8, 40, 2, 130000, 4, 0),
    (0, 32, 4, 4, 400000, 7, 0), (0, 16, 16, 2, 150000, 5, 1), (1, 8, 40, 2, 130000, 4, 1), (0, 64, 2, 2, 20000, 3, 1),
]


@pytest.mark.parametrize("terms", [3, 5])
@pytest.mark.parametrize("solver,n,m,p,T,shards,precision", CASES)
def test_split_is_the_whole_bit_for_bit(pb, solver, n, m, p, T, shards, precision, terms):
    r = np.random.RandomState(76000 + n)
    c = wl.small(76000 + n + T, solver, n, m, p, T, h=1e-3)
    u = pb.register_sinusoid(r.rand(m, terms), 0.1 + 5.0 * r.rand(m, terms), 6.0 * r.rand(m, terms))
    y, _ = multi.emulate_time_partition(pb, c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, shards, solver=solver,
                                        precision=precision)
    pb.set_option(pb.OPT_PATH, pb.PATH_BLOCKED_RESPONSE)
    try:
        whole = pb.Plan(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, solver=solver, precision=precision)
    finally:
        pb.set_option(pb.OPT_PATH, 0)
    whole.execute()
    _, y_whole = whole.output()
    whole.close()
    assert np.array_equal(y, y_whole)
