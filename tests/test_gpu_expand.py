"""The radix expansion (kernels_expand.cu) against the FP64 oracle: solves
without inputs (any form) and sinusoid inputs in the mixed and TF32 forms.

Sizes sit at the kernels' edges: scan dimensions around the multiples of 8,
block counts around 1, 16, 256 and 4096 (the levels), ragged last blocks, odd
output counts (ABM rows then start at an odd offset) and an output buffer
that is not 16-byte aligned, several terms per channel, and an input wider
than the system.

Tolerances: without inputs every operation is FP64, the plain gate 1e-12.
With sinusoids the arithmetic is FP64 too, but the phases advance by the
nominal step where the oracle rounds each sample's argument: at most
2 ulp(2 pi f t) <= 2e-12 of an input (f <= 10, t <= 100), times the ratio of
|D| |u| (or the response) to the output's peak, below 10 here: 1e-10.
"""
import numpy as np
import pytest

from oracle import oracle
from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu

TOL_FREE, TOL_PHASES = 1e-12, 1e-10


def _plan(pb, c, u, precision, B=True, Cm=True, D=True, x0=None):
    return pb.Plan(c.A, c.B if B else None, c.C if Cm else None, c.D if D else None, c.x0 if x0 is None else x0, u,
                   c.t0, c.t_end, c.h, solver=c.solver, precision=precision)


def _device_y(plan, offset):
    import torch

    n = plan.num_outputs * plan.channels
    buf = torch.full((n + 8,), float("nan"), dtype=torch.float64, device="cuda")
    y = buf[offset:offset + n]
    for _ in range(3):  # eager, captured, replayed
        y.fill_(float("nan"))
        plan.execute(y.data_ptr())
        torch.cuda.synchronize()
    assert bool(torch.isnan(buf[offset + n:]).all())  # nothing past the horizon
    return y.cpu().numpy().reshape(plan.num_outputs, plan.channels)


FREE = [  # solver, n, p (0: y = x), T
    (0, 1, 0, 1), (0, 1, 1, 16), (0, 8, 0, 17), (0, 9, 3, 257), (0, 24, 0, 4096), (0, 33, 5, 64 * 256 + 1),
    (0, 64, 0, 64 * 16 - 1), (0, 17, 2, 64 * 4096 + 65), (1, 1, 0, 5), (1, 2, 1, 4099), (1, 5, 3, 64 * 16 + 4),
    (1, 16, 0, 20011), (1, 16, 7, 64 * 17 + 3),
]


@pytest.mark.parametrize("solver,n,p,T", FREE)
def test_free_response(pb, solver, n, p, T):
    c = wl.small(11000 + n + T, solver, n, 1, max(p, 1), T, h=1e-3)
    plan = _plan(pb, c, 0, pb.FP64, B=False, Cm=p > 0, D=False)
    y = _device_y(plan, 1)
    plan.close()
    ref = oracle.simulate_affine(oracle.System(c.A, None, c.C if p else None, None, c.x0), oracle.Input.zero(), solver,
                                 c.t0, c.t_end, c.h)
    assert y.shape == ref.shape
    assert oracle.rel_err(y, ref) <= TOL_FREE


PHASES = [  # solver, n, m, p, T, terms, wider
    (0, 9, 1, 1, 3, 1, 0), (0, 16, 2, 3, 16 * 4 + 1, 3, 1), (0, 24, 3, 1, 4096, 2, 0), (0, 40, 1, 9, 64 * 17, 8, 0),
    (0, 64, 8, 8, 64 * 256 + 63, 3, 0), (0, 64, 12, 2, 5000, 4, 0), (0, 33, 4, 5, 100_000, 1, 2), (1, 3, 1, 1, 4, 1, 0),
    (1, 4, 2, 3, 64 * 16 + 3, 3, 0), (1, 10, 2, 5, 4101, 5, 0), (1, 16, 3, 7, 30_011, 3, 1),
]


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("solver,n,m,p,T,terms,wider", PHASES)
def test_sinusoid_phases(pb, solver, n, m, p, T, terms, wider, precision):
    c = wl.small(12000 + n + T, solver, n, m, p, T, h=1e-3)
    s = wl.sinusoid(wl.Rng(12500 + n), m + wider, terms)
    u = pb.register_sinusoid(s.a, s.f, s.phi)
    plan = _plan(pb, c, u, precision)
    assert plan.path == pb.PATH_BLOCKED_RESPONSE and plan.precision == precision
    assert plan.response_shape[1] == 2 * m * terms
    y = _device_y(plan, precision)
    plan.close()
    ref = oracle.simulate_affine(oracle.System(c.A, c.B, c.C, c.D, c.x0),
                                 oracle.Input.sinusoid(s.a[:m], s.f[:m], s.phi[:m]), solver, c.t0, c.t_end, c.h)
    assert oracle.rel_err(y, ref) <= TOL_PHASES


@pytest.mark.parametrize("solver", [0, 1])
def test_absent_matrices(pb, solver):
    """Only B, only D, y = x with inputs: against the oracle and the in-block sweep path."""
    c = wl.small(13000 + solver, solver, 12, 2, 3, 3000, h=1e-3)
    u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi)
    inp = oracle.Input.sinusoid(c.u.a, c.u.f, c.u.phi)
    for B, Cm, D in [(True, True, False), (False, True, True), (False, False, True), (True, False, False),
                     (True, False, True)]:
        plan = _plan(pb, c, u, pb.MIXED, B, Cm, D)
        y = _device_y(plan, 0)
        plan.close()
        ref = oracle.simulate_affine(oracle.System(c.A, c.B if B else None, c.C if Cm else None, c.D if D else None,
                                                   c.x0), inp, solver, c.t0, c.t_end, c.h)
        assert oracle.rel_err(y, ref) <= TOL_PHASES, (B, Cm, D)


def test_phases_match_the_sample_windows(pb):
    """The same mixed solve by the expansion and by the sample windows (a time
    shard of the whole horizon takes those) agree to the mixed gate."""
    from parode_b200 import multi

    c = wl.small(14000, 0, 48, 5, 6, 40_000, h=1e-3)
    u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi)
    plan = _plan(pb, c, u, pb.MIXED)
    y = _device_y(plan, 0)
    plan.close()
    yw, _ = multi.emulate_time_partition(pb, c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, 2, solver=0,
                                         precision=pb.MIXED)
    assert oracle.rel_err(y, yw) <= 1e-6


def test_one_shot_and_non_finite_state(pb):
    """The one-shot call equals the plan bit for bit, and a non-finite initial state spreads as in a sequential solve."""
    c = wl.small(15000, 0, 20, 2, 2, 9001, h=1e-3)
    u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi)
    plan = _plan(pb, c, u, pb.MIXED)
    y = _device_y(plan, 0)
    plan.close()
    _, y1 = pb.simulate(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, solver=0, precision=pb.MIXED)
    assert np.array_equal(y, y1)
    x0 = c.x0.copy()
    x0[3] = np.nan
    plan = _plan(pb, c, u, pb.MIXED, x0=x0)
    assert np.isnan(_device_y(plan, 0)).all()
    plan.close()


def test_input_with_too_few_channels_is_refused(pb):
    c = wl.small(16000, 0, 20, 3, 2, 3000, h=1e-3)
    u = pb.register_sinusoid(c.u.a[:2], c.u.f[:2], c.u.phi[:2])
    with pytest.raises(pb.ParODEError) as e:
        pb.simulate(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, solver=0, precision=pb.MIXED)
    assert e.value.code == -8


BATCH = [  # solver, n, m, p, T, terms, B, C, D (the batch's doublings; any scan dimension)
    (0, 1, 1, 1, 1, 1, True, True, True), (0, 8, 2, 3, 700, 3, True, True, True), (0, 65, 5, 4, 64 * 33, 3, True, True, True),
    (0, 96, 12, 12, 9001, 2, True, True, False), (0, 200, 3, 7, 2500, 5, True, False, True), (1, 1, 1, 1, 4, 1, True, True, True),
    (1, 17, 2, 2, 39_146, 3, True, True, True), (1, 40, 5, 5, 5003, 3, False, True, True), (1, 100, 2, 1, 1031, 4, True, True, True),
    (0, 30, 0, 30, 3333, 0, False, False, False), (0, 90, 0, 5, 20_000, 0, False, True, False),
    (1, 33, 0, 33, 4100, 0, False, False, False),
]


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_expansion(pb, precision):
    """Mixed: every system by the expansion; FP64: those without inputs."""
    specs, refs = [], []
    for k, (solver, n, m, p, T, terms, B, Cm, D) in enumerate(BATCH):
        if precision == 0 and m:
            continue
        c = wl.small(17000 + 31 * k, solver, n, max(m, 1), p, T, h=1e-3)
        s = wl.sinusoid(wl.Rng(17500 + k), max(m, 1), max(terms, 1))
        u = pb.register_sinusoid(s.a, s.f, s.phi)
        specs.append({"A": c.A, "B": c.B if B else None, "C": c.C if Cm else None, "D": c.D if D else None, "x0": c.x0,
                      "u": u, "t0": c.t0, "t_end": c.t_end, "h": c.h, "solver": solver})
        inp = oracle.Input.sinusoid(s.a, s.f, s.phi) if m else oracle.Input.zero()
        refs.append((m, oracle.simulate_affine(oracle.System(c.A, specs[-1]["B"], specs[-1]["C"], specs[-1]["D"], c.x0),
                                               inp, solver, c.t0, c.t_end, c.h)))
    b = pb.Batch(specs, precision=precision)
    for _ in range(3):  # eager, captured, replayed
        b.execute()
    for i, (m, ref) in enumerate(refs):
        _, y = b.output(i)
        assert y.shape == ref.shape
        err = oracle.rel_err(y, ref)
        assert err <= (TOL_PHASES if m else TOL_FREE), (i, specs[i]["solver"], specs[i]["A"].shape, err)
        assert b.path(i) == (3 if m else 2 if specs[i]["A"].shape[0] * (4 if specs[i]["solver"] else 1) <= 64 else 1)
    b.close()


@pytest.mark.parametrize("solver,n,m,T,terms", [(0, 72, 9, 100, 3), (1, 128, 16, 64 * 600 + 5, 3), (0, 520, 2, 1500, 3),
                                                (0, 64, 8, 9000, 7), (1, 16, 10, 3001, 40)])
def test_large_plan_runs_doublings(pb, solver, n, m, T, terms):
    """One system above scan dimension 64, or with more phases than the
    single-plan kernels take: few tiles a level, so most levels take the
    narrow kernel, the others the 64 x 64 tiles."""
    c = wl.small(18000 + n, solver, n, m, 3, T, h=5e-4)
    s = wl.sinusoid(wl.Rng(18500 + n), m, terms)
    u = pb.register_sinusoid(s.a, s.f, s.phi)
    plan = _plan(pb, c, u, pb.MIXED)
    assert plan.precision == pb.MIXED and plan.response_shape[1] == 2 * terms * m
    y = _device_y(plan, 0)
    plan.close()
    ref = oracle.simulate_affine(oracle.System(c.A, c.B, c.C, c.D, c.x0), oracle.Input.sinusoid(s.a, s.f, s.phi),
                                 solver, c.t0, c.t_end, c.h)
    assert oracle.rel_err(y, ref) <= TOL_PHASES


@pytest.mark.parametrize("n,p,T", [(24, 24, 64 * 16 * 9 + 1), (3, 1, 4100), (64, 5, 9000), (17, 33, 64 * 16 * 3), (40, 1, 70_000)])
def test_output_slices(pb, n, p, T):
    """Outputs in slices of the table by a cost model, row tiles dealt to the
    warps in parts that start and end inside a tile: many rows and few blocks,
    one row, ragged ends.  FP64 free response, gate 1e-12 as for the other forms."""
    c = wl.small(51000 + n + T, 0, n, 1, p, T, h=1e-3)
    plan = _plan(pb, c, 0, pb.FP64, B=False, D=False)
    ref = oracle.simulate_affine(oracle.System(c.A, None, c.C, None, c.x0), oracle.Input.zero(), 0, c.t0, c.t_end, c.h)
    for offset in (0, 1):
        assert oracle.rel_err(_device_y(plan, offset), ref) <= TOL_FREE, offset
    plan.close()
