"""What the block-length tuner times and which solves use it.

A class is tuned with the plan that it gets: in the mixed form sinusoid inputs
enter as phases (the expansion), user functions as samples, and the two leaves
keep entries of their own.  The tuned plan is no slower than the untuned one
and the reported times are those of the two plans.
"""
import pytest

from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _time(pb, torch, plans):
    """Median of 30 solves in ms, the plans in turn."""
    st = torch.cuda.Stream()
    ts = [[] for _ in plans]
    for it in range(34):
        for k, p in enumerate(plans):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(st)
            p.execute(0, st.cuda_stream)
            b.record(st)
            b.synchronize()
            if it >= 4:
                ts[k].append(a.elapsed_time(b))
    return [sorted(t)[len(t) // 2] for t in ts]


@pytest.mark.parametrize("solver,n,m,p,T,precision", [(0, 64, 8, 8, 1 << 19, 1), (0, 64, 8, 8, 1 << 18, 0), (0, 96, 8, 8, 1 << 16, 1)])
def test_tuned_plan_is_no_slower(pb, solver, n, m, p, T, precision):
    import torch

    pb.tune_clear()
    try:
        c = wl.small(67000 + n, solver, n, m, p, T, h=1e-3)
        u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi)
        plan = lambda: pb.Plan(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, solver=solver, precision=precision)  # noqa: E731
        untuned = plan()
        R, best, model = pb.tune_response_block(solver, n, m, p, T, precision)
        tuned = plan()
        assert tuned.response_shape[0] == 1 << R
        assert tuned.response_shape[1] == (6 * m if precision == 1 else tuned.response_shape[1])  # phases of three terms
        t_untuned, t_tuned = _time(pb, torch, [untuned, tuned])
        print(f"R={R} reported {best:.4f} / {model:.4f}, timed {t_tuned:.4f} / {t_untuned:.4f}")
        untuned.close()
        tuned.close()
        assert t_tuned <= 1.08 * t_untuned
        assert 0.8 * t_untuned <= model <= 1.25 * t_untuned
        assert 0.8 * t_tuned <= best <= 1.25 * t_tuned
    finally:
        pb.tune_clear()


def test_leaves_keep_their_own_entries(pb, tmp_path):
    out = tmp_path / "tune.txt"
    try:
        pb.tune_clear()
        R, _, _ = pb.tune_response_block(0, 32, 4, 4, 30000, 1)
        assert pb.tune_save(str(out)) == 2
        entries = {ln.split()[9]: int(ln.split()[7]) for ln in out.read_text().split("\n") if ln}
        assert set(entries) == {"0", "1"} and entries["1"] == R
        c = wl.small(67100, 0, 32, 4, 4, 30000, h=1e-3)
        sin = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi)
        fun = pb.register_input("fType UFunc(fType t, int i) { return sin(t + i); }")
        for u, want in ((sin, entries["1"]), (fun, entries["0"])):
            plan = pb.Plan(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, precision=1)
            assert plan.response_shape[0] == 1 << want
            plan.close()
    finally:
        pb.tune_clear()
