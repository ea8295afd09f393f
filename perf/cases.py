"""The solves this library is timed on, through its public entry points.

Each case is one thing a program does with the library:

  plan   a device-resident solve (Plan): made once, executed into a device
         buffer of the caller's; y stays on the device.  The mixed form's
         result, good to single precision, is kept as float32.
  batch  many systems set up once and executed together (Batch), their outputs
         gathered into one tensor.
  call   a one-shot solve with host arrays in and out: the float C ABI
         (simulate_f32) or the FP64 call (simulate).
  fresh  a batch of new systems: set up, executed, its outputs taken, closed
         (what a queue of solve requests does for every group of requests).
  scan   the affine scan over time-varying maps on device data.

A system is A = -d I + s G / sqrt(n) with G, B, C, D and x0 iid N(0, 1), so it
is stable, with d ~ 1 .. 2.  Inputs are sums of three sinusoids (the built-in
kind), a compiled input function (`user`), or none.
"""
import math

import numpy as np
import torch

import parode_b200 as pb

RK4, ABM = 0, 1
FP64, MIXED = 0, 1


def listed():
    plan = {"what": "plan", "input": "sin"}
    return [
        # the smallest solve in use: 8 states, 4096 steps; launches and latency
        dict(plan, name="plan_small", solver=RK4, n=8, m=2, p=2, T=4096, h=1e-3, precision=FP64),
        # one large RK4 solve, 64 states and 2^20 steps, in both precision forms
        dict(plan, name="plan_rk4_fp64", solver=RK4, n=64, m=8, p=8, T=1 << 20, h=1e-4, precision=FP64),
        dict(plan, name="plan_rk4_mixed", solver=RK4, n=64, m=8, p=8, T=1 << 20, h=1e-4, precision=MIXED),
        # an input function compiled from source, odd horizon
        dict(plan, name="plan_user_mixed", solver=RK4, n=32, m=4, p=4, T=300_001, h=1e-3, precision=MIXED, input="user"),
        # ABM (companion state 4 n): 16 states (scan dimension 64) and 128 (512)
        dict(plan, name="plan_abm_fp64", solver=ABM, n=16, m=4, p=4, T=200_003, h=1e-3, precision=FP64),
        dict(plan, name="plan_abm_mixed", solver=ABM, n=128, m=16, p=16, T=1 << 18, h=5e-4, precision=MIXED),
        # free response (no B, C, D: y is the state), odd size
        dict(plan, name="plan_free", solver=RK4, n=24, m=0, p=24, T=100_003, h=1e-3, precision=FP64, input="none"),
        # a thousand systems of uneven sizes: n in 4..96, T in 2^10..2^16, RK4 and ABM
        {"name": "batch_mixed", "what": "batch", "count": 1024, "n_lo": 4, "n_hi": 96, "T_lo": 1 << 10, "T_hi": 1 << 16, "h": 1e-3,
         "precision": MIXED},
        # a group of new requests: n in 8..256, T in 10^3..10^5
        {"name": "fresh_fp64", "what": "fresh", "count": 16, "n_lo": 8, "n_hi": 256, "T_lo": 1000, "T_hi": 100_000, "h": 1e-3,
         "precision": FP64},
        # the C ABI as a simulation script calls it: 16 states, 4 inputs and outputs, h = 0.1, 1.28e5 steps, float host arrays
        {"name": "call_f32", "what": "call", "solver": RK4, "n": 16, "m": 4, "p": 4, "T": 128_000, "h": 0.1, "input": "user", "float": True,
         "precision": FP64},
        # a short one-shot ABM solve in FP64
        {"name": "call_small", "what": "call", "solver": ABM, "n": 4, "m": 2, "p": 2, "T": 2000, "h": 1e-2, "input": "sin", "float": False,
         "precision": FP64},
        # time-varying maps: 16 states, 2^16 steps
        {"name": "scan_varying", "what": "scan", "n": 16, "T": 1 << 16, "precision": FP64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["plan", "plan", "plan", "plan", "plan", "batch", "fresh", "call", "call", "scan"])
    precision = rng.choice([FP64, MIXED])
    if what == "plan":
        solver = rng.choice([RK4, ABM])
        n = _log(rng, 4, 128)
        dim = n if solver == RK4 else 4 * n
        T = _log(rng, 1000, min(1 << 20, (1 << 26) // dim))
        kind = rng.choice(["sin", "sin", "sin", "user", "none"])
        m, p = (0, n) if kind == "none" else (rng.randint(1, max(1, n // 8) + 1), rng.randint(1, max(1, n // 8) + 1))
        return {"what": what, "solver": solver, "n": n, "m": m, "p": p, "T": T, "h": rng.choice([1e-4, 5e-4, 1e-3]), "precision": precision,
                "input": kind}
    if what == "batch":
        return {"what": what, "count": _log(rng, 32, 512), "n_lo": 4, "n_hi": rng.randint(32, 96), "T_lo": 1 << 10, "T_hi": _log(rng, 4096, 1 << 16),
                "h": 1e-3, "precision": precision}
    if what == "fresh":
        return {"what": what, "count": rng.randint(1, 16), "n_lo": 8, "n_hi": rng.randint(32, 256), "T_lo": 1000, "T_hi": _log(rng, 4000, 100_000),
                "h": 1e-3, "precision": precision}
    if what == "call":
        solver, n, T, flt = rng.choice([RK4, ABM]), _log(rng, 4, 64), _log(rng, 1000, 200_000), rng.random() < 0.5
        return {"what": what, "solver": solver, "n": n, "m": rng.randint(1, 4), "p": rng.randint(1, 4), "T": T,
                "h": rng.choice([1e-2, 0.1]) if solver == RK4 else 1e-2, "input": rng.choice(["sin", "user"]), "float": flt,
                "precision": FP64}
    return {"what": what, "n": rng.randint(4, 64), "T": _log(rng, 1000, 1 << 15), "precision": precision}


# ---- inputs ------------------------------------------------------------------


def _system(r, solver, n, m, p, T, h, diag=None):
    """One system as the package's calls take it (T: outputs)."""
    d = 1.0 + r.rand() if diag is None else diag
    A = 0.5 * r.standard_normal((n, n)) / math.sqrt(n)
    A[np.diag_indices(n)] -= d
    s = {"A": A, "B": None, "C": None, "D": None, "x0": r.standard_normal(n), "t0": 0.0, "t_end": (T - 0.5) * h, "h": h, "solver": solver}
    if m:
        s.update(B=r.standard_normal((n, m)), C=r.standard_normal((p, n)), D=r.standard_normal((p, m)))
        s["sin"] = (r.rand(m, 3), 0.1 + 9.9 * r.rand(m, 3), 2.0 * math.pi * r.rand(m, 3))
    return s


def _single(case, seed):
    r = np.random.RandomState(seed % (1 << 32))
    s = _system(r, case["solver"], case["n"], case["m"], case["p"], case["T"], case["h"], diag=1.5)
    s["wave"] = (r.rand(max(case["m"], 1)) + 0.25, r.rand(max(case["m"], 1)) + 0.5)
    return s


def _many(case, seed):
    r = np.random.RandomState(seed % (1 << 32))
    # sizes are the case's own (systems differ by the seed, not the work)
    z = np.random.RandomState(case["count"])
    out = []
    for i in range(case["count"]):
        n = int(round(math.exp(z.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        T = int(round(math.exp(z.uniform(math.log(case["T_lo"]), math.log(case["T_hi"])))))
        m = max(1, n // 8)
        out.append(_system(r, i % 2, n, m, m, T, case["h"]))
    return out


def _user_source(s):
    """A sawtooth (even channels) and a square wave (odd ones), period 16."""
    amp, level = s["wave"]
    rows = "".join("    if (nInputIndex == %d) return nInputIndex %% 2 ? (x < 0.5 ? (fType)%r : (fType)%r) : (fType)(%r * x);\n"
                   % (i, float(np.float32(level[i])), float(np.float32(-level[i])), float(np.float32(amp[i]))) for i in range(len(amp)))
    return "fType UFunc(fType t, int nInputIndex) {\n    fType x = t * (fType)0.0625;\n    x = x - floor(x);\n" + rows + "    return 0;\n}\n"


def _input(s, kind):
    if kind == "user":
        return pb.register_input(_user_source(s))
    return pb.register_sinusoid(*s["sin"]) if kind == "sin" else 0


_stream = []


def _library():
    """The library and the stream that all of the program's work is queued on."""
    if not _stream:
        pb.init()
        _stream.append(torch.cuda.Stream())
    return _stream[0]


class _Device:
    """A library-owned device buffer as torch.as_tensor takes it."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


def _outputs(b):
    return [torch.as_tensor(_Device(b.device_output(i), (b.num_outputs[i], b.channels[i])), device="cuda") for i in range(b.size)]


def prepare(case, seed):
    st = _library()
    what = case["what"]
    state = {"case": case, "stream": st}
    if what == "plan":
        s = _single(case, seed)
        plan = pb.Plan(s["A"], s["B"], s["C"], s["D"], s["x0"], _input(s, case["input"]), s["t0"], s["t_end"], s["h"], solver=s["solver"],
                       precision=case["precision"])
        state.update(plan=plan, y=torch.empty((plan.num_outputs, plan.channels), dtype=torch.float64, device="cuda"))
    elif what in ("batch", "fresh"):
        specs = _many(case, seed)
        for s in specs:
            s["u"] = _input(s, "sin")
        state["specs"] = specs
        if what == "batch":
            b = pb.Batch(specs, precision=case["precision"])
            y = _outputs(b)
            state.update(batch=b, y=[v.reshape(-1) for v in y],
                         out=torch.empty(sum(v.numel() for v in y), dtype=torch.float64, device="cuda"))
    elif what == "call":
        s = _single(case, seed)
        typ = np.float32 if case["float"] else np.float64
        T = pb.num_outputs(s["solver"], s["t0"], s["t_end"], s["h"])
        state.update(s={k: (v.astype(typ) if isinstance(v, np.ndarray) else v) for k, v in s.items()}, u=_input(s, case["input"]),
                     t=np.empty(T, typ), y=np.empty((T, case["p"]), typ))
    else:
        M, V, x0 = _maps(case, seed)
        state.update(M=M, V=V, x0=x0, X=torch.empty_like(V))
    torch.cuda.synchronize()
    return state


def run(state):
    case, st = state["case"], state["stream"]
    what = case["what"]
    if what == "plan":
        state["plan"].execute(state["y"].data_ptr(), st.cuda_stream)
        if case["precision"] == FP64:
            return state["y"]
        with torch.cuda.stream(st):
            return state["y"].to(torch.float32)
    if what == "batch":
        state["batch"].execute(st.cuda_stream)
        with torch.cuda.stream(st):
            y = torch.cat(state["y"], out=state["out"])
            return y if case["precision"] == FP64 else y.to(torch.float32)
    if what == "fresh":
        b = pb.Batch(state["specs"], precision=case["precision"])
        b.execute(st.cuda_stream)
        with torch.cuda.stream(st):
            y = [v.clone() if case["precision"] == FP64 else v.to(torch.float32) for v in _outputs(b)]
        b.close()
        return y
    if what == "call":
        s = state["s"]
        a = (s["A"], s["B"], s["C"], s["D"], s["x0"], state["u"], s["t0"], s["t_end"], s["h"])
        if case["float"]:
            t, y, err = pb.simulate_f32(*a, solver=s["solver"], t_out=state["t"], y_out=state["y"])
            if err:
                raise pb.ParODEError(err, "SimulateODE")
            return t, y
        return pb.simulate(*a, solver=s["solver"], precision=case["precision"], t_out=state["t"], y_out=state["y"])
    with torch.cuda.stream(st):
        pb.affine_scan_general(state["M"].data_ptr(), state["V"].data_ptr(), state["x0"].data_ptr(), case["n"], case["T"],
                               state["X"].data_ptr(), precision=case["precision"], stream=st.cuda_stream)
        return state["X"] if case["precision"] == FP64 else state["X"].to(torch.float32)


def _maps(case, seed):
    """M_k = a rotation-free contraction near the identity, different at every step."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, T = case["n"], case["T"]
    M = torch.randn((T, n, n), generator=g, dtype=torch.float64, device="cuda").mul_(0.01 / math.sqrt(n))
    M.diagonal(dim1=1, dim2=2).add_(0.985)
    V = torch.randn((T, n), generator=g, dtype=torch.float64, device="cuda")
    return M, V, torch.randn(n, generator=g, dtype=torch.float64, device="cuda")


# ---- what a pass cannot do without ---------------------------------------------


def _one(solver, n, m, p, T, size=8):
    """The system read once, y written once; the sequential recurrence's operations."""
    terms = 3 if solver == RK4 else 5
    dim = n if solver == RK4 else 4 * n
    system = n * n + (n * m + p * n + p * m if m else 0) + n
    out = 2 * p * (n + m) if m else 0
    return size * (system + T * p), T * (2 * n * dim + 2 * n * terms * m + out)


def work(case):
    what = case["what"]
    if what in ("plan", "call"):
        b, f = _one(case["solver"], case["n"], case["m"], case["p"], case["T"], 4 if case.get("float") else 8)
        if what == "call":
            b += case["T"] * (4 if case["float"] else 8)
        return {"bytes": b, "flops": f}
    if what in ("batch", "fresh"):
        both = [_one(s["solver"], s["A"].shape[0], s["B"].shape[1], s["C"].shape[0], int(s["t_end"] / s["h"]) + 1) for s in _many(case, 0)]
        return {"bytes": sum(b for b, _ in both), "flops": sum(f for _, f in both)}
    n, T = case["n"], case["T"]
    return {"bytes": 8 * T * (n * n + 2 * n), "flops": T * 2 * n * n}


# ---- the same in 64 bits ---------------------------------------------------------


def _u(s, kind, t, flt):
    """Inputs at times t (FP64), shape (len(t), m)."""
    if kind == "user":
        tt = t.to(torch.float32).to(torch.float64) if flt else t
        amp, level = (np.float32(v).astype(np.float64) for v in s["wave"])
        x = tt * 0.0625
        x = x - torch.floor(x)
        cols = [torch.where(x < 0.5, level[i], -level[i]) if i % 2 else amp[i] * x for i in range(len(amp))]
        return torch.stack([c.to(torch.float64) for c in cols], 1)
    a, f, phi = (torch.as_tensor(v, device=t.device) for v in s["sin"])
    out = torch.zeros((len(t), a.shape[0]), dtype=torch.float64, device=t.device)
    for k in range(a.shape[1]):
        out += a[:, k] * torch.sin((2.0 * math.pi * f[:, k])[None, :] * t[:, None] + phi[:, k])
    return out


def _recurrence(Phi, G, x):
    """x_0 .. x_{T-1} of x_{k+1} = Phi x_k + G_k, G (T, N): chunks side by side, twice (their ends, then from their starts)."""
    T, N = G.shape
    L = max(1, int(math.sqrt(T)))
    C = -(-T // L)
    Gp = torch.zeros((C * L, N), dtype=torch.float64, device=G.device)
    Gp[:T] = G
    Gp = Gp.reshape(C, L, N)
    P = Phi.T.contiguous()
    z = torch.zeros((C, N), dtype=torch.float64, device=G.device)
    for k in range(L):
        z = torch.addmm(Gp[:, k], z, P)
    PL = torch.linalg.matrix_power(Phi, L)
    starts = [x]
    for c in range(C - 1):
        starts.append(torch.addmv(z[c], PL, starts[-1]))
    z = torch.stack(starts)
    X = torch.empty((C, L, N), dtype=torch.float64, device=G.device)
    for k in range(L):
        X[:, k] = z
        z = torch.addmm(Gp[:, k], z, P)
    return X.reshape(C * L, N)[:T]


def _solve(s, kind, flt=False):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f = lambda v: None if v is None else torch.as_tensor((np.float32(v) if flt else v).astype(np.float64), device=dev)  # noqa: E731
    A, B, Cm, D, x = (f(s[k]) for k in ("A", "B", "C", "D", "x0"))
    h, n = s["h"], A.shape[0]
    T = int((s["t_end"] - (3 * h if s["solver"] == ABM else 0.0)) / h) + 1
    eye = torch.eye(n, dtype=torch.float64, device=dev)
    A2 = A @ A
    if s["solver"] == RK4:
        A3 = A2 @ A
        Phi = eye + h * A + h * h / 2 * A2 + h ** 3 / 6 * A3 + h ** 4 / 24 * (A3 @ A)
        G = torch.zeros((T, n), dtype=torch.float64, device=dev)
        if B is not None:
            U = _u(s, kind, s["t0"] + 0.5 * h * torch.arange(2 * T + 1, dtype=torch.float64, device=dev), flt)
            B0 = (h * B + h * h * (A @ B) + h ** 3 / 2 * (A2 @ B) + h ** 4 / 4 * (A3 @ B)) / 6
            B1 = (4 * h * B + 2 * h * h * (A @ B) + h ** 3 / 2 * (A2 @ B)) / 6
            G = U[0:-1:2] @ B0.T + U[1::2] @ B1.T + U[2::2] @ (h / 6 * B).T
        X = _recurrence(Phi, G, x)
        u = U[0:-1:2] if B is not None else None
        return X if Cm is None else X @ Cm.T + u @ D.T
    # ABM: three RK4 steps, then the AB4 predictor / AM4 corrector as one map of the last four states
    starts = [x]
    if B is not None:
        U9 = _u(s, kind, s["t0"] + 0.5 * h * torch.arange(9, dtype=torch.float64, device=dev), flt)
    for k in range(3):
        bu = [B @ U9[2 * k + j] for j in range(3)] if B is not None else [0.0] * 3
        x = starts[-1]
        k1 = A @ x + bu[0]
        k2 = A @ (x + 0.5 * h * k1) + bu[1]
        k3 = A @ (x + 0.5 * h * k2) + bu[1]
        k4 = A @ (x + h * k3) + bu[2]
        starts.append(x + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4))
    Phi = torch.zeros((4 * n, 4 * n), dtype=torch.float64, device=dev)
    Phi[:3 * n, n:] = torch.eye(3 * n, dtype=torch.float64, device=dev)
    q = h * h / 576
    Phi[3 * n:] = torch.cat([-81 * q * A2, h / 24 * A + 333 * q * A2, -5 * h / 24 * A - 531 * q * A2, eye + 28 * h / 24 * A + 495 * q * A2], 1)
    G = torch.zeros((T, 4 * n), dtype=torch.float64, device=dev)
    if B is not None:
        U = _u(s, kind, s["t0"] + h * torch.arange(T + 4, dtype=torch.float64, device=dev), flt)
        AB = A @ B
        taps = [-81 * q * AB, h / 24 * B + 333 * q * AB, -5 * h / 24 * B - 531 * q * AB, 19 * h / 24 * B + 495 * q * AB, 9 * h / 24 * B]
        for k, b in enumerate(taps):
            G[:, 3 * n:] += U[k:k + T] @ b.T
    X = torch.cat([torch.stack(starts[:3]), _recurrence(Phi, G, torch.cat(starts))[:, 3 * n:]])
    return X if Cm is None else X @ Cm.T + (U[:T + 3] @ D.T)


def _times(solver, T, h):
    """The time vector: the float of the time before plus the step, link by link (ABM: its first three times back from the fourth)."""
    t = np.empty(T)
    first = 3 if solver == ABM else 0
    ts = 3.0 * h if first else 0.0
    for i in range(first):
        t[i] = np.float32(ts - (first - i) * h)
    v = float(np.float32(ts))
    for i in range(first, T):
        t[i] = v
        v = float(np.float32(v + h))
    return t


def exact(case, seed):
    what = case["what"]
    if what == "plan":
        return _solve(_single(case, seed), case["input"])
    if what == "batch":
        return torch.cat([_solve(s, "sin").reshape(-1) for s in _many(case, seed)])
    if what == "fresh":
        return [_solve(s, "sin") for s in _many(case, seed)]
    if what == "call":
        y = _solve(_single(case, seed), case["input"], case["float"])
        return _times(case["solver"], case["T"], case["h"]), y
    M, V, x = _maps(case, seed)
    X = torch.empty_like(V)
    # the same chunks as _recurrence, each with its own maps
    T, n = V.shape
    L = max(1, int(math.sqrt(T)))
    C = -(-T // L)
    Mp = torch.eye(n, dtype=torch.float64, device=V.device).repeat(C * L, 1, 1)
    Vp = torch.zeros((C * L, n), dtype=torch.float64, device=V.device)
    Mp[:T], Vp[:T] = M, V
    Mp, Vp = Mp.reshape(C, L, n, n), Vp.reshape(C, L, n, 1)
    z = torch.zeros((C, n, 1), dtype=torch.float64, device=V.device)
    P = torch.eye(n, dtype=torch.float64, device=V.device).repeat(C, 1, 1)
    for k in range(L):
        z, P = torch.baddbmm(Vp[:, k], Mp[:, k], z), torch.bmm(Mp[:, k], P)
    starts = [x[:, None]]
    for c in range(C - 1):
        starts.append(P[c] @ starts[-1] + z[c])
    z = torch.stack(starts)
    X = torch.empty((C, L, n), dtype=torch.float64, device=V.device)
    for k in range(L):
        X[:, k] = z[:, :, 0]
        z = torch.baddbmm(Vp[:, k], Mp[:, k], z)
    return X.reshape(C * L, n)[:T]
