"""The launch count a plan reports is the number of kernels that one of its
executes runs, as the device's own activity record lists them.
"""
import pytest

from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu

CASES = [  # solver, n, m, p, T, precision, path, input
    (0, 8, 2, 2, 4096, 0, 5, "sin"), (1, 16, 2, 2, 70000, 0, 5, "sin"), (0, 8, 2, 2, 12, 0, 5, "sin"), (0, 12, 0, 12, 3000, 0, 5, "none"),
    (0, 64, 2, 2, 9000, 1, 5, "sin"), (0, 16, 2, 2, 20000, 0, 0, "sin"), (0, 32, 4, 4, 30000, 1, 0, "user"),
    (0, 32, 4, 4, 30000, 1, 3, "sin"), (0, 32, 4, 4, 30000, 1, 0, "sin"), (0, 24, 0, 24, 30000, 0, 0, "none"),
    (0, 16, 2, 2, 20000, 0, 4, "sin"), (0, 16, 2, 2, 20000, 0, 1, "sin"),
]


def _kernels(torch, f):
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    return sum(1 for e in p.events() if str(e.device_type).endswith("CUDA") and "Memcpy" not in e.name and "Memset" not in e.name)


@pytest.mark.parametrize("solver,n,m,p,T,precision,path,kind", CASES)
def test_launch_count_is_what_runs(pb, solver, n, m, p, T, precision, path, kind):
    import torch

    x = torch.zeros(8, device="cuda")
    if _kernels(torch, lambda: x.add_(1)) != 1:
        pytest.skip("the device's activity record is not available")
    c = wl.small(75000 + n, solver, n, max(m, 1), p, T, h=1e-3)
    u = 0
    if kind == "sin":
        u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi)
    elif kind == "user":
        u = pb.register_input("fType UFunc(fType t, int i) { return sin(t + i); }")
    pb.set_option(pb.OPT_PATH, path)
    try:
        plan = pb.Plan(c.A, c.B if m else None, c.C if m else None, c.D if m else None, c.x0, u, c.t0, c.t_end, c.h, solver=solver,
                       precision=precision)
    finally:
        pb.set_option(pb.OPT_PATH, 0)
    # two outputs in turn: the second execute launches kernel by kernel too
    y = [torch.empty((plan.num_outputs, plan.channels), dtype=torch.float64, device="cuda") for _ in range(2)]
    st = torch.cuda.Stream()
    plan.execute(y[0].data_ptr(), st.cuda_stream)
    seen = _kernels(torch, lambda: plan.execute(y[1].data_ptr(), st.cuda_stream))
    count = plan.launch_count
    plan.close()
    assert count == seen
