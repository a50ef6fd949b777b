"""The work that users of this framework have it do, as cases that can be timed.

A case is one call, or the calls of one time step, of the SGDLM filter through the
package's public entry points: the reference-style Python class with host arrays,
the fused device step, the batched step, the learned proposal and its network's
gradient, the multi-step forecast and the allocation-free log|det|.

The data are simulated from a true SGDLM: m series, each with three external
predictors (intercept, own lag, an iid covariate) and up to kmax simultaneous
parents with coefficients N(0, 0.1^2), rescaled to a spectral radius of at most
0.5.  A state's filter has run 40 steps of the decoupled filter from the vague
prior, so that it stands where a filter in use stands; it then cycles through the
16 steps that follow, one per pass.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from gpusgdlm_gb300 import SGDLM, Batch
from gpusgdlm_gb300 import _lib as L

N_EXT, BURN_IN, RING = 3, 40, 16
HIDDEN = 128  # width of the proposal network


def listed():
    return [
        # the smallest calls: one step of the decoupled filter (no simulation), host arrays
        {"name": "filter_m20", "kind": "filter", "m": 20, "kmax": 5},
        # the README's time step: m = 6, plain FP64, 10 000 draws, host arrays
        {"name": "readme_m6_fp64", "kind": "step", "m": 6, "kmax": 0, "n": 10000, "precision": "fp64"},
        # the same loop on a system of ordinary size in the default precision
        {"name": "step_m100", "kind": "step", "m": 100, "kmax": 10, "n": 10000, "precision": "mixed"},
        # the headline workload: the fused step on device-resident data, m = 400
        {"name": "device_m400", "kind": "device", "m": 400, "kmax": 17, "n": 10000, "precision": "mixed"},
        # a fused step of odd sizes
        {"name": "device_m133_odd", "kind": "device", "m": 133, "kmax": 8, "n": 4999, "precision": "mixed"},
        # the plain FP64 form (the reference's arithmetic) at an ordinary size and the headline's
        {"name": "device_m100_fp64", "kind": "device", "m": 100, "kmax": 10, "n": 10000, "precision": "fp64"},
        {"name": "device_m400_fp64", "kind": "device", "m": 400, "kmax": 17, "n": 10000, "precision": "fp64"},
        # forecasts 1..5 steps ahead, 10 000 samples each, into host arrays
        {"name": "forecast_k5_m400", "kind": "forecast", "m": 400, "kmax": 17, "n": 10000, "steps": 5,
         "evolution": False, "precision": "mixed"},
        # independent instances of mixed sizes advanced together by one graph launch
        {"name": "batch_16", "kind": "batch", "count": 16, "m_low": 20, "m_high": 400, "kmax": 17, "n": 10000},
        # one step with the learned importance proposal in use
        {"name": "learned_m200", "kind": "learned", "m": 200, "kmax": 12, "n": 10000},
        # a training batch of that proposal's network: forward, loss, every gradient
        {"name": "gradient_b4096", "kind": "gradient", "max_p": 15, "batch": 4096},
        # log|det| of a batch of draws without allocations, odd sizes
        {"name": "logdet_m333_odd", "kind": "logdet", "m": 333, "kmax": 11, "n": 1999},
    ]


def _between(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["filter", "step", "step", "device", "device", "forecast", "batch", "learned",
                       "gradient", "logdet"])
    if kind == "gradient":
        return {"kind": kind, "max_p": rng.randint(4, 24), "batch": _between(rng, 256, 8192)}
    if kind == "batch":
        low = rng.randint(20, 60)
        return {"kind": kind, "count": rng.randint(2, 12), "m_low": low, "m_high": rng.randint(low + 20, 400),
                "kmax": rng.randint(4, 17), "n": _between(rng, 1000, 10000)}
    m = _between(rng, 8, 400)
    c = {"kind": kind, "m": m, "kmax": rng.randint(1, min(17, m - 1))}
    if kind == "filter":
        return c
    if kind == "logdet":
        return dict(c, n=_between(rng, 200, 2000))
    if kind == "learned":
        return dict(c, m=min(m, 250), n=_between(rng, 1000, 10000))
    if kind == "forecast":
        return dict(c, n=_between(rng, 500, 10000), steps=rng.randint(1, 5), evolution=rng.random() < 0.3,
                    precision="mixed")
    fp64 = rng.random() < 0.35
    if kind == "step":  # up to the 50 000 draws of the precision configuration
        return dict(c, n=_between(rng, 500, 8000 if fp64 else 50000), precision="fp64" if fp64 else "mixed")
    return dict(c, n=_between(rng, 500, 10000), precision="fp64" if fp64 else "mixed")


# ------------------------------------------------------------------------- data
class Problem:
    """A true SGDLM's structure and data: p, sp (NaN: no simultaneous parent), y, predictors."""

    def __init__(self, m, kmax, seed, steps=BURN_IN + RING + 6):
        rng = np.random.default_rng(seed)
        if m == 6 and kmax == 0:  # the README's system
            ext = np.array([2, 1, 1, 3, 1, 2])
            parents = [[5], [0, 5, 3], [], [0, 1], [], [1, 3]]
        else:
            ext = np.full(m, N_EXT)
            parents = []
            for j in range(m):
                k = int(rng.integers(0, kmax + 1))
                q = rng.choice(m - 1, size=k, replace=False)
                parents.append([int(v) + (v >= j) for v in q])
        self.m, self.ext = m, ext
        self.p = ext + np.array([len(q) for q in parents])
        self.P = max(int(self.p.max()), 3 + kmax if kmax else 0)
        self.sp = np.full((self.P, m), np.nan)
        self.parent = np.full((self.P, m), -1)
        gamma = np.zeros((m, m))
        for j, q in enumerate(parents):
            for t, par in enumerate(q):
                self.sp[ext[j] + t, j] = j + m * par
                self.parent[ext[j] + t, j] = par
                gamma[j, par] = rng.normal(0, 0.1)
        power = gamma
        for _ in range(5):
            power = power @ power
        radius = np.linalg.norm(power) ** (1 / 32) if m > 1 else 0.0
        if radius > 0.5:
            gamma *= 0.5 / radius
        inverse = np.linalg.inv(np.eye(m) - gamma)
        phi = rng.normal(0, 0.3, size=(m, 3)) * (np.arange(3) < ext[:, None])
        lam = rng.gamma(5.0, 80.0, size=m)
        self.y = np.zeros((steps + 1, m))
        self.X = np.zeros((steps + 1, m, 3))
        for t in range(1, steps + 1):
            self.X[t] = np.stack([np.ones(m), self.y[t - 1], rng.normal(size=m)], axis=1)
            nu = (self.X[t] * phi).sum(1) + rng.normal(size=m) / np.sqrt(lam)
            self.y[t] = inverse @ nu

    def F(self, t, with_parents=True):
        """The predictors of step t (max_p x m); the parents' places are zero for a forecast."""
        F = np.zeros((self.P, self.m), order="F")
        for k in range(min(3, self.P)):
            F[k] = np.where(k < self.ext, self.X[t, :, k], 0.0)
        if with_parents:
            on = self.parent >= 0
            F[on] = self.y[t][self.parent[on]]
        return F

    def vague_prior(self):
        m, P = self.m, self.P
        R = np.asfortranarray(np.repeat((0.1 * np.eye(P))[:, :, None], m, axis=2))
        return np.zeros((P, m), order="F"), R, np.full(m, 2.0), np.full(m, 0.0025)


def _engine(pr, precision="mixed", compat=L.COMPAT_REFERENCE, seed=1):
    """The engine after the burn-in, in the prior state before step BURN_IN + 1."""
    s = SGDLM(1, strict=True, precision=precision, compat=compat)
    s.setSimultaneousParents(pr.p, pr.sp)
    s.setDiscountFactors(np.full(pr.m, 0.97), np.full((pr.P, pr.P, pr.m), 0.98))
    s.setPriorParameters(*pr.vague_prior())
    for t in range(1, BURN_IN + 1):
        s.computePosterior(pr.y[t], pr.F(t))
        s.computePrior()
    s.setRngState(seed, 0)
    return s


def _device(a, dtype=torch.float64):
    return torch.tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


def _staged(pr):
    """y, F and the next step's x of the ring's steps, as the device entry points read them."""
    ts = range(BURN_IN + 1, BURN_IN + RING + 1)
    return (_device(np.stack([pr.y[t] for t in ts])),
            _device(np.stack([pr.F(t).ravel(order="F") for t in ts])),
            _device(np.stack([pr.F(t + 1, False).ravel(order="F") for t in ts])))


def _draws(case, seed):
    """FP32 draws of a fitted model's coefficients (series-major) and the parental sets."""
    pr = Problem(case["m"], case["kmax"], seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    mean = 0.1 * torch.randn((pr.m, 1, pr.P), generator=g, device="cuda") / math.sqrt(1 + case["kmax"] / 4)
    theta = mean + 0.02 * torch.randn((pr.m, case["n"], pr.P), generator=g, device="cuda")
    return pr, theta.contiguous()


def _network(case, seed):
    """A training batch of the proposal network and its parameters."""
    P, B = case["max_p"], case["batch"]
    F, O = 2 * P + 5, 2 * P + 2
    rng = np.random.default_rng(seed)
    X = rng.normal(size=(B, F)).astype(np.float32)
    Y = (0.1 * rng.normal(size=(B, O))).astype(np.float32)
    mask = (rng.random((B, O)) < 0.8).astype(np.float32)
    w = np.concatenate([v.astype(np.float32).ravel() for v in (
        rng.normal(size=(HIDDEN, F)) / math.sqrt(F), 0.1 * rng.normal(size=HIDDEN),
        rng.normal(size=(HIDDEN, HIDDEN)) / math.sqrt(HIDDEN), 0.1 * rng.normal(size=HIDDEN),
        0.1 * rng.normal(size=(O, HIDDEN)), 0.1 * rng.normal(size=O))])
    return F, O, X, Y, mask, w


# ---------------------------------------------------------------------- prepare
class State:
    t = 0

    def step(self):
        """This pass's step of the ring: its index and its time."""
        i = self.t % RING
        self.t += 1
        return i, BURN_IN + 1 + i


def prepare(case, seed):
    st = State()
    st.case, kind = case, case["kind"]
    if kind == "gradient":
        F, O, st.X, st.Y, st.mask, w = _network(case, seed)
        st.s = SGDLM(1, strict=True)
        st.s.setSimultaneousParents(np.full(4, case["max_p"]), np.full((case["max_p"], 4), np.nan))
        st.s.setProposalParams(w)
        return st
    if kind == "logdet":
        pr, st.theta = _draws(case, seed)
        sp = np.where(np.isnan(pr.sp), 2147483648, np.nan_to_num(pr.sp)).astype(np.uint32)
        st.sp = torch.tensor(sp.view(np.int32).ravel(order="F"), device="cuda")
        st.P = pr.P
        st.logdet = torch.zeros(case["n"], dtype=torch.float64, device="cuda")
        st.flags = torch.zeros(case["n"], dtype=torch.int32, device="cuda")
        st.stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        return st
    if kind == "batch":
        ms = np.linspace(case["m_low"], case["m_high"], case["count"]).round()
        prs = [Problem(int(m), min(case["kmax"], int(m) - 1), seed + 1 + k) for k, m in enumerate(ms)]
        st.engines = [_engine(pr, seed=seed + k) for k, pr in enumerate(prs)]
        st.inputs, st.now, st.forecasts = [], [], []
        for s, pr in zip(st.engines, prs):
            s._ensure_sim(case["n"], case["n"])
            staged = torch.cat(_staged(pr), dim=1)
            st.inputs.append(staged)
            st.now.append(torch.zeros_like(staged[0]))
            st.forecasts.append(torch.zeros((case["n"], pr.m), dtype=torch.float64, device="cuda"))
        st.stats = [torch.zeros(8, dtype=torch.float64, device="cuda") for _ in prs]
        st.batch = Batch(st.engines)
        y = [v.data_ptr() for v in st.now]
        F = [v.data_ptr() + 8 * pr.m for v, pr in zip(st.now, prs)]
        x = [v.data_ptr() + 8 * pr.m * (1 + pr.P) for v, pr in zip(st.now, prs)]
        st.batch.record(y, F, x, case["n"] / 2, [f.data_ptr() for f in st.forecasts], None,
                        [v.data_ptr() for v in st.stats])
        torch.cuda.synchronize()
        return st
    pr = st.pr = Problem(case["m"], case["kmax"], seed)
    # forecasts several steps ahead take the corrected samplers: the reference's beta
    # sampler gives NaN for the shapes that are met here
    st.s = _engine(pr, case.get("precision", "mixed"),
                   L.COMPAT_NONE if kind == "forecast" else L.COMPAT_REFERENCE, seed)
    if kind == "device":
        n = case["n"]
        st.s._ensure_sim(n, n)
        st.y, st.F, st.x = _staged(pr)
        st.forecast = torch.zeros((n, pr.m), dtype=torch.float64, device="cuda")
        st.weights = torch.zeros(n, dtype=torch.float64, device="cuda")
        st.stats = torch.zeros(8, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return st
    ts = range(BURN_IN + 1, BURN_IN + RING + 1)
    st.F = [pr.F(t) for t in ts]
    if kind == "forecast":
        st.x = [np.asfortranarray(np.stack([pr.F(t + k, False) for k in range(case["steps"])], axis=2))
                for t in ts]
        if case["evolution"]:
            rng = np.random.default_rng(seed)
            st.G = np.asfortranarray(np.eye(pr.P)[:, :, None] * 0.98
                                     + 0.005 * rng.normal(size=(pr.P, pr.P, pr.m)))
        return st
    st.x = [pr.F(t + 1, False) for t in ts]
    if kind == "learned":  # a network trained earlier, its parameters set from the program's own copy
        rng = np.random.default_rng(seed)
        st.s.setProposal("learned", train_steps=0)
        _, F, O = st.s.proposalSizes()
        st.s.setProposalParams(np.concatenate([v.ravel() for v in (
            0.01 * rng.normal(size=(HIDDEN, F)) / math.sqrt(F), 0.01 * rng.normal(size=HIDDEN),
            rng.normal(size=(HIDDEN, HIDDEN)) / math.sqrt(HIDDEN), 0.01 * rng.normal(size=HIDDEN),
            0.001 * rng.normal(size=(O, HIDDEN)), 0.001 * rng.normal(size=O))]).astype(np.float32))
    return st


# -------------------------------------------------------------------------- run
def run(st):
    case, kind = st.case, st.case["kind"]
    if kind == "gradient":
        loss, grad = st.s.proposalLossAndGradient(st.X, st.Y, st.mask)
        return [loss, grad]
    if kind == "logdet":
        ok = L.lib().sgdlm_log_det_noalloc(case["m"], st.P, case["n"], ctypes.c_void_p(st.theta.data_ptr()),
                                           ctypes.c_void_p(st.sp.data_ptr()),
                                           ctypes.c_void_p(st.logdet.data_ptr()),
                                           ctypes.c_void_p(st.flags.data_ptr()), st.stream)
        if ok != L.OK:
            raise RuntimeError(L.STATUS[ok])
        return st.logdet
    i, t = st.step()
    if kind == "batch":
        torch.cuda.synchronize()  # the last step has read its inputs
        for now, staged in zip(st.now, st.inputs):
            now.copy_(staged[i])
        torch.cuda.synchronize()  # this step's inputs are there
        st.batch.step()
        return [st.forecasts, st.stats]
    s, pr = st.s, st.pr
    if kind == "device":
        s.filterStepDevice(st.y[i].data_ptr(), st.F[i].data_ptr(), st.x[i].data_ptr(), case["n"] / 2,
                           st.forecast.data_ptr(), st.weights.data_ptr(), st.stats.data_ptr())
        return [st.forecast, st.weights, st.stats]
    if kind == "forecast":
        n = case["n"]
        if case["evolution"]:
            return s.computeEvoForecast(n, n, st.x[i], st.G)
        return s.computeForecast(n, n, st.x[i])
    s.computePosterior(pr.y[t], st.F[i])
    if kind == "filter":
        s.computePrior()
        q = s.getParameters()
        return [q["m"], q["C"], q["n"], q["s"]]
    n = case["n"]
    vb = s.computeVBPosterior(n, n)
    w = vb["IS_weights"]
    if 1.0 / np.dot(w, w) > n / 2:
        s.setPosteriorParameters(vb["m"], vb["C"], vb["n"], vb["s"])
    s.computePrior()
    out = [vb["m"], vb["C"], vb["n"], vb["s"], w, vb["sum_det_weights"]]
    if kind == "step":
        out.append(s.computeForecast(n, n, st.x[i]))
    return out


# ------------------------------------------------------------------------- work
def work(case):
    """Each input read once, each output written once; for a simulation, per draw: the sampling
    (Philox, normals and gammas, U'z), the log|det| (the dense part that a sparse elimination of
    these systems leaves is about half of the series) and the weighted moments; a forecast
    solve as 40 products with the sparse matrix."""
    kind = case["kind"]
    if kind == "gradient":
        B, F, O = case["batch"], 2 * case["max_p"] + 5, 2 * case["max_p"] + 2
        weights = HIDDEN * (F + HIDDEN + O)
        return {"bytes": 4 * (B * (F + 2 * O) + 2 * weights), "flops": 2 * B * (3 * weights - HIDDEN * F)}
    if kind == "batch":
        m = (case["m_low"] + case["m_high"]) / 2
        one = work({"kind": "device", "m": m, "kmax": min(case["kmax"], m - 1), "n": case["n"]})
        return {k: case["count"] * v for k, v in one.items()}
    m, kmax = case["m"], case["kmax"]
    P = 5 if kmax == 0 else N_EXT + kmax
    p = 3.3 if kmax == 0 else N_EXT + kmax / 2
    nnz = m * (p - N_EXT if kmax else 4 / 3)
    core = m if m <= 32 else m / 2
    state = m * (P * P + P + 2)
    if kind == "filter":
        return {"bytes": 8 * (2 * state + m * (P * P + P + 2)), "flops": m * (5.0 * P * P + 10 * P)}
    n = case["n"]
    if kind == "logdet":
        return {"bytes": 4 * n * nnz + 8 * n, "flops": n * 2 / 3 * core ** 3}
    sample, logdet = m * (p * (p + 1) + 40 * p), 2 / 3 * core ** 3 + 20 * nnz
    moments, solve = m * (p * (p + 1) + 4 * p), 40 * 2 * nnz + m * 60
    out = 8 * n * m
    if kind == "forecast":
        K = case["steps"]
        return {"bytes": K * (out + 8 * m * P) + 8 * state, "flops": n * K * (sample + solve)}
    vb = {"bytes": 8 * (3 * state + m * (1 + P) + n), "flops": n * (sample + logdet + moments)}
    if kind == "learned":
        return {"bytes": vb["bytes"], "flops": vb["flops"] + n * m * 2 * p * (p + 1)}
    return {"bytes": vb["bytes"] + out + 8 * m * P, "flops": vb["flops"] + n * (sample + solve)}


# ------------------------------------------------------------------------ exact
def _exact_filter(case, seed):
    pr = Problem(case["m"], case["kmax"], seed)
    a, R, r, c = pr.vague_prior()
    for t in range(1, BURN_IN + 2):
        F, y = pr.F(t), pr.y[t]
        for j in range(pr.m):
            on = np.arange(pr.P) < pr.p[j]
            mean = np.where(on, a[:, j], 0)
            cov = np.where(on[:, None] | on[None, :], R[:, :, j], 0)
            A = cov @ F[:, j]
            Q = c[j] + F[:, j] @ A
            e = y[j] - F[:, j] @ mean
            A /= Q
            a[:, j] = mean + e * A
            cov = (cov - np.outer(A, A) * Q) * ((r[j] + e * e / Q) / (r[j] + 1))
            R[:, :, j] = np.where(on[:, None] & on[None, :], cov / 0.98, cov)
            c[j] *= (r[j] + e * e / Q) / (r[j] + 1)
            r[j] = (r[j] + 1) * 0.97
    return [a, R, r, c]


def _exact_logdet(case, seed):
    pr, theta = _draws(case, seed)
    m = pr.m
    j = np.nonzero(pr.parent.T >= 0)
    rows, ks = torch.tensor(j[0], device="cuda"), torch.tensor(j[1], device="cuda")
    cols = torch.tensor(pr.parent.T[j], device="cuda")
    out = []
    for i in range(0, case["n"], 250):
        block = theta[:, i:i + 250].double()
        A = torch.eye(m, dtype=torch.float64, device="cuda").repeat(block.shape[1], 1, 1)
        A[:, rows, cols] = -block[rows, :, ks].T
        out.append(torch.linalg.slogdet(A)[1])
    return torch.cat(out)


def _exact_gradient(case, seed):
    F, O, X, Y, mask, w = _network(case, seed)
    X, Y, mask = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (X, Y, mask))
    parts, at = [], 0
    for shape in ((HIDDEN, F), (HIDDEN,), (HIDDEN, HIDDEN), (HIDDEN,), (O, HIDDEN), (O,)):
        size = math.prod(shape)
        v = torch.tensor(w[at:at + size]).reshape(shape)
        v = v.bfloat16().double() if len(shape) == 2 else v.double()  # the network's weights are BF16
        parts.append(v.cuda().requires_grad_())
        at += size
    W1, b1, W2, b2, W3, b3 = parts
    gelu = torch.nn.functional.gelu
    out = gelu(gelu(X @ W1.T + b1) @ W2.T + b2) @ W3.T + b3
    loss = (mask * (out - Y) ** 2).sum() / mask.sum()
    loss.backward()
    return [loss.item(), torch.cat([v.grad.ravel() for v in parts])]


def exact(case, seed):
    """The other kinds return Monte-Carlo results of the framework's own random stream: no value
    but that stream's is theirs."""
    if case["kind"] == "filter":
        return _exact_filter(case, seed)
    if case["kind"] == "logdet":
        return _exact_logdet(case, seed)
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed)
    return None
