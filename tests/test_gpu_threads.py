"""Host threads that launch the same kernels with different amounts of shared
memory: plans executed side by side on streams of their own, and mixed batches
of very different phase counts formed by the server's set-up threads.  Every
solve gives the bits it gives alone (plans), or passes its gate (server).
"""
import threading

import numpy as np
import pytest

from oracle import oracle
from parode_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_plans_of_different_sizes_side_by_side(pb, precision):
    import torch

    # slices of W from a few KB to the whole of shared memory, in one kernel each (Kc 80 in the mixed form)
    shapes = [(64, 1, 1, 700), (64, 2, 64, 900), (64, 1, 9, 1500), (60, 2, 33, 800)]
    jobs = []
    for k, (n, m, p, T) in enumerate(shapes):
        c = wl.small(64000 + k, 0, n, m, p, T, h=1e-3)
        u = pb.register_sinusoid(c.u.a, c.u.f, c.u.phi)
        plan = pb.Plan(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, precision=precision)
        # two outputs in turn: every execute launches kernel by kernel
        y = [torch.empty((plan.num_outputs, plan.channels), dtype=torch.float64, device="cuda") for _ in range(2)]
        jobs.append((plan, y, torch.cuda.Stream()))
        plan.execute(y[0].data_ptr(), jobs[-1][2].cuda_stream)
    torch.cuda.synchronize()
    alone = [y[0].cpu().numpy() for _, y, _ in jobs]
    errors = []

    def work(k):
        plan, y, st = jobs[k]
        try:
            for it in range(300):
                plan.execute(y[(it + 1) % 2].data_ptr(), st.cuda_stream)
        except Exception as e:  # noqa: BLE001
            errors.append((k, e))

    th = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in th:
        t.start()
    for t in th:
        t.join()
    torch.cuda.synchronize()
    got = [[v.cpu().numpy() for v in y] for _, y, _ in jobs]
    for plan, _, _ in jobs:
        plan.close()
    assert not errors, errors
    for a, both in zip(alone, got):
        for v in both:
            assert np.array_equal(a, v)


def test_mixed_batches_formed_by_several_server_threads(pb):
    # one phase pair up to 240 (12 channels of 20 terms)
    r = np.random.RandomState(65)
    server = pb.Server(precision=1, hbm_budget_bytes=8e9, max_batch=2, max_inflight=4)
    ids = []
    for k in range(48):
        m, terms = (1, 1) if k % 2 else (12, 20)
        c = wl.small(65000 + k, 0, 12 + k % 5, m, 2, 300 + k, h=1e-3)
        a, f, phi = r.rand(m, terms) / terms, 0.1 + 2.0 * r.rand(m, terms), r.rand(m, terms)
        u = pb.register_sinusoid(a, f, phi)
        rid = server.submit(c.A, c.B, c.C, c.D, c.x0, u, c.t0, c.t_end, c.h, solver=c.solver)
        ids.append((rid, c, oracle.Input.sinusoid(a, f, phi)))
    for rid, c, inp in ids:
        _, y, _ = server.wait(rid, timeout_s=120)
        ref = oracle.simulate_affine(oracle.System(c.A, c.B, c.C, c.D, c.x0), inp, c.solver, c.t0, c.t_end, c.h)
        assert oracle.rel_err(y, ref) <= 1e-6
    assert server.stats()["failed"] == 0
    server.close()
