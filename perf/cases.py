"""Performance cases of the K2 evaluator: what its callers run, through the public entry points.

listed() gives the named cases, draw(rng) more of the same ranges.  prepare() makes what a program
holds before the call (the zero table on the GPU, the plan, the candidate arrays), run() is one
pass, work() the bytes and operations a pass cannot do without, and exact() the outputs of the same
inputs from FP64 matrix products and sines/cosines in torch.

The zero table is the same for every seed (the zeros of zeta are the same for every program);
candidates, offsets, grids and gradients come from the seed.  Every seed's state has its own
ZeroTable and plan.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

from mertens_bound_b200 import autograd, hit_polish, k2, path1, polish, score, synth

N_FULL = 2_325_572          # zeros below 1.3e6: the certificate's table
N_SEARCH = 466_659          # zeros below 3e5: the search scoring table
N_DRIVER = 600_000          # the search drivers' zeros_600k table
N_SCAN = 98_624             # zeros below 74,000: the peak re-optimisation's table
INF = math.inf


# ------------------------------------------------------------------ the cases


def listed():
    return [
        # one small batch through the plain FP64 evaluator (host arrays): latency of a single call
        dict(name="plain_small", kind="plain", P=64, n=10_000, k=3e-9),
        # a search loop that scores a few points at a time through a kept plan (host arrays)
        dict(name="plan_host_small", kind="plan", P=16, n=10_000, k=3e-9, host=True),
        # the search scoring step: 4,096 candidates over every zero below 3e5, on the device
        dict(name="plan_search", kind="plan", P=4096, n=N_SEARCH, k=3e-9, host=False),
        # batched scoring of uneven (k, T) groups over the full table
        dict(name="batched_uneven", kind="batched", P=16_384, n=N_FULL, groups=12, mix=0),
        # K2 as a differentiable function: forward and backward, an odd candidate count
        dict(name="grad_odd", kind="grad", P=1001, n=N_DRIVER, k=1e-9),
        # batched Newton polish of the offsets from the best point of a short grid
        dict(name="newton_polish", kind="newton", P=1024, n=N_SEARCH, k=3e-9, iters=8),
        # the certificate's interval: one point over the whole table
        dict(name="certified_full", kind="certified", P=1, n=N_FULL, k=1.5e-10, grad=False),
        # peak re-optimisation: the 25,001-point grid around one point
        dict(name="grid_scan", kind="grid", points=25_001, n=N_SCAN, k=3e-9, step=2e-5),
        # the enumerators' staged polish of their hits, all stages
        dict(name="hit_polish", kind="hits", P=256, n=N_DRIVER, k=3e-9),
        # the search drivers' step: candidates scored under the weight kernels, grid + Newton
        dict(name="driver_scoring", kind="scoring", P=256, n=N_DRIVER),
        # Taylor-moment polish of a candidate list, exact Newton on its top 25
        dict(name="taylor_polish", kind="taylor", P=1024, n=100_000),
        # the GPU enumerator's leaf screen on leaves it has just made on the device
        dict(name="screen_leaves", kind="screen", P=1 << 20, n=4096, k=3e-9),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plan", "plan", "batched", "grad", "newton", "certified", "grid", "hits", "scoring",
                       "taylor", "screen"])
    k = rng.choice([3e-9, 1e-9, 1.5e-10])
    if kind == "plain":
        n = _log_int(rng, 2_000, N_SEARCH)
        return dict(kind=kind, P=_log_int(rng, 1, min(4096, 400_000_000 // n)), n=n, k=k)
    if kind == "plan":
        n = _log_int(rng, 2_000, N_FULL)
        return dict(kind=kind, P=_log_int(rng, 1, min(16_384, 4_000_000_000 // n)), n=n, k=k, host=rng.random() < 0.4)
    if kind == "batched":
        return dict(kind=kind, P=_log_int(rng, 512, 8192), n=_log_int(rng, 100_000, N_FULL), groups=rng.randint(2, 12),
                    mix=rng.randint(1, 10**6))
    if kind == "grad":
        n = _log_int(rng, 10_000, N_FULL)
        return dict(kind=kind, P=_log_int(rng, 8, min(4096, 2_000_000_000 // n)), n=n, k=k)
    if kind == "newton":
        return dict(kind=kind, P=_log_int(rng, 16, 2048), n=_log_int(rng, 20_000, N_SEARCH), k=3e-9,
                    iters=rng.randint(2, 8))
    if kind == "certified":
        return dict(kind=kind, P=_log_int(rng, 1, 24), n=_log_int(rng, 50_000, N_FULL), k=k, grad=rng.random() < 0.5)
    if kind == "grid":
        return dict(kind=kind, points=2 * _log_int(rng, 200, 12_500) + 1, n=_log_int(rng, 5_000, N_SCAN), k=3e-9,
                    step=rng.choice([2e-5, 1e-5, 5e-6]))
    if kind == "hits":
        return dict(kind=kind, P=_log_int(rng, 4, 256), n=_log_int(rng, 16_000, N_DRIVER), k=3e-9)
    if kind == "scoring":
        return dict(kind=kind, P=_log_int(rng, 8, 256), n=_log_int(rng, 20_000, N_DRIVER))
    if kind == "taylor":
        return dict(kind=kind, P=_log_int(rng, 16, 1024), n=_log_int(rng, 10_000, 100_000))
    return dict(kind=kind, P=_log_int(rng, 5_000, 1 << 20), n=4096, k=3e-9)


# ------------------------------------------------------------------ inputs


@functools.lru_cache(maxsize=1)
def _full():
    return synth.make_table(N_FULL, seed=1)


def _table(n):
    """The first n zeros (one fixed table: make_table's first n zeros depend on n only through the
    random streams' lengths, so every case takes a prefix of the full one)."""
    return _full().truncate(n)


def _points(case, seed):
    """Candidates of a seed, with FP64 offsets as the drivers' lists carry them."""
    c = synth.make_candidates(case["P"], seed=seed)
    if case["kind"] in ("plan", "grad", "batched", "scoring"):
        c.delta[:] = np.random.default_rng(seed).uniform(-1e-4, 1e-4, c.n)
    return c


def _groups(case):
    """(counts, ks, Ts) of a batched case: its mix 0 is the twelve uneven (k, T) groups, any other
    mix random group sizes over the same cutoffs and Gaussian widths."""
    if case["mix"] == 0:
        return synth.batched_uneven_groups()
    r = random.Random(case["mix"])
    cuts = sorted(r.sample(range(1, case["P"]), case["groups"] - 1))
    counts = [b - a for a, b in zip([0] + cuts, cuts + [case["P"]])]
    return (counts, [r.choice([3e-9, 1e-9, 1.5e-10]) for _ in counts],
            [r.choice([1e5, 3e5, 6e5, 1.3e6]) for _ in counts])


WEIGHTS = ("jp", "g15", "g10", "raw", "10k")
GRID_STEP, GRID_HALF = 2.5e-5, 10            # Newton's starting grid: 21 points
SCREEN_SCALE = 1.75                          # coefficient scale: some leaves pass the first stages


def _data(case):
    d = _table(case["n"])
    if case["kind"] == "screen":
        d.c_re *= SCREEN_SCALE
        d.c_im *= SCREEN_SCALE
    return d


def _dev_u64(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64).copy()).cuda()


def _start_offsets(case, c):
    """Newton's starting offsets: each candidate's best |K2| on a short grid over the first 4,096
    zeros (the reference's polish scans that many)."""
    d = _table(min(4096, case["n"]))
    T = _Exact(d, np.exp(-case["k"] * d.gamma * d.gamma))
    grid = [(m * GRID_STEP) for m in range(-GRID_HALF, GRID_HALF + 1)]
    h = torch.stack([T.sums(_limbs(_shift(c, np.full(c.n, g))), first=True)[0].abs() for g in grid])
    return np.array(grid)[h.argmax(dim=0).cpu().numpy()]


def prepare(case, seed):
    kind = case["kind"]
    data = _data(case)
    s = dict(case=case, kind=kind, table=k2.ZeroTable.from_data(data))
    t = s["table"]
    if kind == "plain":
        s["cands"] = _points(case, seed)
    elif kind in ("plan", "batched"):
        s["cands"] = c = _points(case, seed)
        counts, ks, Ts = _groups(case) if kind == "batched" else ([case["P"]], [case["k"]], [INF])
        s["plan"] = k2.Plan(t, counts, ks, Ts)
        if not case.get("host"):
            s["vi"], s["vf"], s["delta"] = _dev_u64(c.v_int), _dev_u64(c.v_frac), torch.from_numpy(c.delta).cuda()
            s["out"] = torch.empty(3, c.n, dtype=torch.float64, device="cuda")
    elif kind == "grad":
        c = _points(case, seed)
        s["eval"] = autograd.K2Torch(t)
        s["vi"], s["vf"] = _dev_u64(c.v_int), _dev_u64(c.v_frac)
        s["delta"] = torch.from_numpy(c.delta).cuda().requires_grad_()
        s["k"] = torch.tensor(case["k"], dtype=torch.float64, device="cuda", requires_grad=True)
        s["g"] = torch.from_numpy(_upstream(case, seed)).cuda()
        s["eval"].plan(case["P"], float(case["k"]))
    elif kind == "newton":
        c = _points(case, seed)
        s["eval"] = autograd.K2Torch(t)
        s["vi"], s["vf"] = _dev_u64(c.v_int), _dev_u64(c.v_frac)
        s["start"] = torch.from_numpy(_start_offsets(case, c)).cuda()
        s["delta"] = s["start"].clone()
        s["eval"].plan(case["P"], float(case["k"]))
    elif kind == "certified":
        s["cands"] = _points(case, seed)
    elif kind == "grid":
        c = synth.make_candidates(1, seed=seed)
        s["y0"] = polish.from_fixed(int(c.v_int[0]), int(c.v_frac[0]), 25)
    elif kind == "hits":
        s["points"] = hit_polish.points_from_x(synth.leaves_x(case["P"], seed))
    elif kind == "scoring":
        s["cands"] = _points(case, seed)
        w = score.reference_weights(data.gamma)
        s["slots"] = score.register(t, {name: w[name] for name in WEIGHTS})
    elif kind == "taylor":
        s["cands"] = _points(case, seed)
        s["slot"] = t.add_weights(score.reference_weights(data.gamma)["jp"])
    elif kind == "screen":
        c = _points(case, seed)
        P = case["P"]
        s["vi"], s["vf"] = _dev_u64(c.v_int), _dev_u64(c.v_frac)
        s["hits"] = torch.empty(P, dtype=torch.int64, device="cuda")
        s["hit_scores"] = torch.empty(P, 3, dtype=torch.float32, device="cuda")
        s["count"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        s["scores"] = torch.empty(P, 3, dtype=torch.float32, device="cuda")
    return s


def _upstream(case, seed):
    return np.random.default_rng(seed + 1).standard_normal(case["P"])


# ------------------------------------------------------------------ one pass


def run(s):
    kind, case, t = s["kind"], s["case"], s["table"]
    if kind == "plain":
        return k2.k2_plain(t, s["cands"], case["k"])
    if kind in ("plan", "batched"):
        if case.get("host"):
            return s["plan"].run(s["cands"])
        o = s["out"]
        s["plan"].run_dev(s["vi"].data_ptr(), s["vf"].data_ptr(), s["delta"].data_ptr(), o[0].data_ptr(),
                          o[1].data_ptr(), o[2].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return [o[0], o[1], o[2]]
    if kind == "grad":
        val = s["eval"](s["vi"], s["vf"], s["delta"], s["k"])
        gd, gk = torch.autograd.grad(val, (s["delta"], s["k"]), s["g"])
        return [val.detach(), gd, gk]
    if kind == "newton":
        s["delta"].copy_(s["start"])            # the polish moves the offsets in place
        return [*s["eval"].newton(s["vi"], s["vf"], s["delta"], float(case["k"]), iters=case["iters"]), s["delta"]]
    if kind == "certified":
        if case["grad"]:
            return k2.k2_certified_grad(t, s["cands"], case["k"])
        return k2.k2_certified(t, s["cands"], case["k"])
    if kind == "grid":
        half = (case["points"] - 1) // 2
        return polish.grid(t, s["y0"], half * case["step"], case["step"], case["k"], INF)[1]
    if kind == "hits":
        r = hit_polish.polish_hits(t, s["points"], case["k"], thresholds=(None, None, None))
        return [r.h, r.dy, r.stage]
    if kind == "scoring":
        return score.score(t, s["cands"], s["slots"])
    if kind == "taylor":
        return path1.fast_polish_exact(t, s["cands"], s["slot"])
    hit_polish.screen_leaves_dev(t, s["vi"].data_ptr(), s["vf"].data_ptr(), case["P"], s["hits"].data_ptr(),
                                 s["hit_scores"].data_ptr(), s["count"].data_ptr(), case["P"], case["k"],
                                 d_scores=s["scores"].data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
    # the hit list comes in arbitrary order: the leaves' scores hold the same decisions in order
    return [s["scores"], s["count"]]


# ------------------------------------------------------------------ what a pass cannot do without

# per (point, zero): the phase product and its reduction (6), sine and cosine (2), the weighted
# value, dK2/ddelta and dK2/dk (6)
FLOPS_TERM = 14
ZERO_BYTES = 44             # G (20), gamma (8), c (16)


def work(case):
    kind, n = case["kind"], case["n"]
    P = case.get("P", 1)
    table = n * ZERO_BYTES
    if kind in ("plain", "plan", "grad"):
        return dict(bytes=table + 48 * P, flops=FLOPS_TERM * P * n)
    if kind == "batched":
        counts, _, Ts = _groups(case)
        n_T = [min(n, float(synth.zero_count(T))) for T in Ts]
        return dict(bytes=max(n_T) * ZERO_BYTES + 48 * P, flops=FLOPS_TERM * sum(c * m for c, m in zip(counts, n_T)))
    if kind == "newton":
        return dict(bytes=table + 64 * P, flops=FLOPS_TERM * P * n * (case["iters"] + 1))
    if kind == "certified":                       # every operation at both interval ends
        return dict(bytes=table + 40 * P, flops=2 * (FLOPS_TERM if case["grad"] else FLOPS_TERM - 4) * P * n)
    if kind == "grid":                            # a rotation and an addition per (point, zero)
        return dict(bytes=table + 8 * case["points"], flops=4 * case["points"] * n)
    if kind == "hits":
        per = sum(min(n, z or n) * (2 * m + 1) for z, m, *_ in hit_polish.STAGES)
        return dict(bytes=table + 40 * P, flops=4 * P * per)
    if kind == "scoring":
        # per weight vector: the 81-point grid over 4,096 zeros, at least one Newton step and h
        return dict(bytes=table + 8 * n * len(WEIGHTS) + 24 * P * len(WEIGHTS),
                    flops=len(WEIGHTS) * P * (4 * 81 * min(n, 4096) + 2 * FLOPS_TERM * n))
    if kind == "taylor":                          # 17 moments per term
        return dict(bytes=table + 8 * n + 48 * P, flops=(8 + 34) * P * n)
    return dict(bytes=256 * ZERO_BYTES + 28 * P, flops=(8 + 21) * P * 64)


# ------------------------------------------------------------------ the same in 64 bits
#
# frac(v G): with v = sum_i v_i 2^(22 i - 64) in 22-bit limbs and f_ij = frac(2^(22 i - 64) G_j) =
# h_ij 2^-28 + l_ij (h_ij a 28-bit integer), sum_i v_i h_ij < 2^53 is exact in a FP64 matrix
# product and sum_i v_i l_ij < 2^-3 is rounded at 2^-56.

LIMB = 22


def _limbs(points):
    """(P, 6) FP64 limbs of 64.64 points given as Python ints v 2^64 (mod 2^128)."""
    hi = np.array([p >> 64 for p in points], dtype=np.uint64)
    lo = np.array([p & (2**64 - 1) for p in points], dtype=np.uint64)
    out = np.empty((len(points), 6))
    m = np.uint64((1 << LIMB) - 1)
    for i in range(6):
        o = LIMB * i
        if o + LIMB <= 64:
            x = lo >> np.uint64(o)
        elif o < 64:
            x = (lo >> np.uint64(o)) | (hi << np.uint64(64 - o))
        else:
            x = hi >> np.uint64(o - 64)
        out[:, i] = (x & m).astype(np.float64)
    return torch.from_numpy(out).cuda()


def _fix(d):
    """round(d 2^64) of a double, exactly."""
    m, e = math.frexp(float(d))
    a, sh = int(m * 2.0**53), e + 11
    return a << sh if sh >= 0 else (a + (1 << (-sh - 1))) >> -sh


def _shift(c, delta):
    return [(((int(a) << 64) | int(b)) + _fix(x)) % 2**128 for a, b, x in zip(c.v_int, c.v_frac, delta)]


class _Exact:
    """A table's phases and sums in FP64 torch."""

    def __init__(self, d, w):
        gi, hi, lo = (np.ascontiguousarray(d.G3[:, i]) for i in range(3))
        fh, fl = np.empty((6, d.n)), np.empty((6, d.n))
        for i in range(6):
            sft = LIMB * i - 64
            if sft == -64:
                a, b = gi, hi
            elif sft < 0:
                r, l = np.uint64(-sft), np.uint64(64 + sft)
                a, b = (gi << l) | (hi >> r), (hi << l) | (lo >> r)
            elif sft == 0:
                a, b = hi, lo
            else:
                l, r = np.uint64(sft), np.uint64(64 - sft)
                a, b = (hi << l) | (lo >> r), lo << l
            fh[i] = (a >> np.uint64(36)).astype(np.float64)
            fl[i] = ((a & np.uint64(2**36 - 1)).astype(np.float64) * 2.0**-64 + b.astype(np.float64) * 2.0**-128)
        up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
        self.n, self.fh, self.fl = d.n, up(fh), up(fl)
        self.gamma, self.cr, self.ci = up(d.gamma), up(d.c_re), up(d.c_im)
        self.w = None if w is None else up(w)

    def cs(self, V, a, b):
        """cos and sin of gamma v for limbs V over the zeros [a, b)."""
        t = V @ self.fh[:, a:b]
        t *= 2.0**-28
        t -= torch.round(t)
        t += V @ self.fl[:, a:b]
        t *= 2.0 * math.pi
        s = torch.sin(t)
        return t.cos_(), s

    def sums(self, V, n=None, first=False, w=None):
        """K2, dK2/ddelta, dK2/dk (only K2 with first) of every row of V over the first n zeros."""
        n = self.n if n is None else n
        w = (self.w if w is None else w)[:n]
        P = V.shape[0]
        rows = max(1, min(P, 4096))
        out = torch.zeros(1 if first else 3, P, dtype=torch.float64, device="cuda")
        wr, wi, g = w * self.cr[:n], w * self.ci[:n], self.gamma[:n]
        for p in range(0, P, rows):
            step = max(1, (1 << 26) // min(rows, P - p))
            for a in range(0, n, step):
                b = min(n, a + step)
                c, s = self.cs(V[p:p + rows], a, b)
                q = slice(p, p + c.shape[0])
                if first:
                    out[0, q] += 2.0 * (c @ wr[a:b] - s @ wi[a:b])
                else:
                    X = torch.stack([wr[a:b], wr[a:b] * g[a:b], wr[a:b] * g[a:b]**2], 1)
                    Y = torch.stack([wi[a:b], wi[a:b] * g[a:b], wi[a:b] * g[a:b]**2], 1)
                    re, im = c @ X - s @ Y, s @ X + c @ Y
                    out[0, q] += 2.0 * re[:, 0]
                    out[1, q] -= 2.0 * im[:, 1]
                    out[2, q] -= 2.0 * re[:, 2]
        return out

    def matrices(self, V, n):
        """A, B = 2 Re, 2 Im of c e^{i gamma v}."""
        A = torch.empty(V.shape[0], n, dtype=torch.float64, device="cuda")
        B = torch.empty_like(A)
        step = max(1, (1 << 26) // V.shape[0])
        for a in range(0, n, step):
            b = min(n, a + step)
            c, s = self.cs(V, a, b)
            A[:, a:b] = 2.0 * (self.cr[a:b] * c - self.ci[a:b] * s)
            B[:, a:b] = 2.0 * (self.cr[a:b] * s + self.ci[a:b] * c)
        return A, B


def _h(A, B, g, w, ddy, deriv=False):
    """h (and h', h'') = sum w (A cos(g ddy) - B sin(g ddy)) for each row, in row chunks."""
    out = []
    rows = max(1, (1 << 26) // max(1, A.shape[1]))
    for p in range(0, A.shape[0], rows):
        t = ddy[p:p + rows, None] * g[None, :]
        c, s = torch.cos(t), t.sin_()
        v = A[p:p + rows] * c - B[p:p + rows] * s
        if deriv:
            d = -A[p:p + rows] * s - B[p:p + rows] * c
            out.append(torch.stack([v @ w, d @ (w * g), -(v @ (w * g * g))]))
        else:
            out.append((v @ w)[None])
    return torch.cat(out, 1)


def _newton(A, B, g, w, ddy, iters, clamp, tol):
    go = torch.ones_like(ddy, dtype=torch.bool)
    for _ in range(iters):
        _, fp, fpp = _h(A, B, g, w, ddy, True)
        go &= fpp.abs() > 1e-12
        step = torch.where(go, (fp / fpp).clamp(-clamp, clamp), torch.zeros_like(ddy))
        ddy = ddy - step
        go &= step.abs() >= tol
        if not bool(go.any()):
            break
    return ddy


def exact(case, seed):
    kind = case["kind"]
    d = _data(case)
    gauss = lambda k: np.exp(-k * d.gamma * d.gamma)  # noqa: E731
    if kind in ("plain", "plan", "grad"):
        c = _points(case, seed)
        o = _Exact(d, gauss(case["k"])).sums(_limbs(_shift(c, c.delta)))
        if kind == "grad":
            g = torch.from_numpy(_upstream(case, seed)).cuda()
            return [o[0], g * o[1], (g * o[2]).sum()]
        return [o[0], o[1], o[2]]
    if kind == "batched":
        c = _points(case, seed)
        V, T = _limbs(_shift(c, c.delta)), _Exact(d, None)
        out, p = [], 0
        for cnt, k, cut in zip(*_groups(case)):
            T.w = torch.from_numpy(gauss(k)).cuda()
            out.append(T.sums(V[p:p + cnt], n=int(np.searchsorted(d.gamma, cut))))
            p += cnt
        o = torch.cat(out, 1)
        return [o[0], o[1], o[2]]
    if kind == "newton":
        c = _points(case, seed)
        T = _Exact(d, gauss(case["k"]))
        start = _start_offsets(case, c)
        x, go = start.copy(), np.ones(c.n, dtype=bool)
        o = first = T.sums(_limbs(_shift(c, x)))
        for _ in range(case["iters"]):
            dd, dk = o[1].cpu().numpy(), o[2].cpu().numpy()
            go &= np.abs(dk) > 1e-12
            step = np.where(go, np.clip(dd / dk, -1e-4, 1e-4), 0.0)
            x = x - step
            go &= np.abs(step) >= 1e-13
            o = T.sums(_limbs(_shift(c, x)))
        keep = first[0].abs() > o[0].abs()
        o = torch.where(keep, first, o)
        xs = torch.where(keep, torch.from_numpy(start).cuda(), torch.from_numpy(x).cuda())
        return [first[0], o[0], o[1], o[2], xs]
    if kind == "certified":
        c = _points(case, seed)
        T = _Exact(d, gauss(case["k"]))
        o = T.sums(_limbs(_shift(c, c.delta)))
        if case["grad"]:
            return [o, o]
        a = 2.0 * (T.w * torch.hypot(T.cr, T.ci)).sum().expand(c.n)
        return [o[0], o[0], a]
    if kind == "grid":
        c = synth.make_candidates(1, seed=seed)
        vi, vf = polish.to_fixed(polish.from_fixed(int(c.v_int[0]), int(c.v_frac[0]), 25))
        half, sf = (case["points"] - 1) // 2, _fix_floor(case["step"])
        pts = [((vi << 64) + vf + m * sf) % 2**128 for m in range(-half, half + 1)]
        return _Exact(d, gauss(case["k"])).sums(_limbs(pts), first=True)[0]
    if kind == "hits":
        return _exact_hits(case, seed, d)
    if kind == "screen":
        return _exact_screen(case, seed, d)
    c = _points(case, seed)
    T = _Exact(d, None)
    A, B = T.matrices(_limbs(_shift(c, c.delta)), d.n)
    W = score.reference_weights(d.gamma)
    if kind == "taylor":
        return _exact_taylor(A, B, T.gamma, torch.from_numpy(W["jp"]).cuda())
    out = {}
    for name in WEIGHTS:
        w, m = torch.from_numpy(W[name]).cuda(), min(d.n, 4096)
        h0 = A @ w
        best, at = h0.abs(), torch.zeros_like(h0)
        for i in range(-40, 41):
            x = torch.full_like(h0, 2.5e-4 * i / 40)
            h = _h(A[:, :m], B[:, :m], T.gamma[:m], w[:m], x)[0].abs()
            at, best = torch.where(h > best, x, at), torch.maximum(h, best)
        x = _newton(A, B, T.gamma, w, at, 6, 1e-4, 1e-13)
        h = _h(A, B, T.gamma, w, x)[0]
        keep = h0.abs() > h.abs()
        out[name] = (h0, torch.where(keep, h0, h), torch.where(keep, torch.zeros_like(x), x))
    return out


def _fix_floor(step):
    m, e = math.frexp(step)
    a, sh = int(m * 2.0**53), e + 11
    return a << sh if sh >= 0 else a >> -sh


def _exact_hits(case, seed, d):
    T = _Exact(d, np.exp(-case["k"] * d.gamma * d.gamma))
    base = [x << 34 for x in synth.leaves_x(case["P"], seed)]
    centre = [0] * len(base)
    h_out = None
    for s, (zeros, m_half, step, recentre, _) in enumerate(hit_polish.STAGES):
        n, sf = min(d.n, zeros or d.n), _fix_floor(step)
        start = [b + (c if recentre else 0) for b, c in zip(base, centre)]
        pts = [(b + m * sf) % 2**128 for b in start for m in range(-m_half, m_half + 1)]
        h = T.sums(_limbs(pts), n=n, first=True)[0].reshape(len(base), -1)
        j = h.abs().argmax(dim=1)
        if s != 3:
            h_out = h.gather(1, j[:, None])[:, 0]
        centre = [(c if recentre else 0) + (int(i) - m_half) * sf for c, i in zip(centre, j.cpu())]
    dy = torch.tensor([c / 2.0**64 for c in centre], dtype=torch.float64)
    return [h_out, dy, None]


def _exact_taylor(A, B, g, w, top=25):
    u = g * 1e-4
    grid = torch.from_numpy(np.linspace(-3.0e-5, 3.0e-5, 121)).cuda()
    z = grid * 1e4
    h = torch.zeros(A.shape[0], grid.shape[0], dtype=torch.float64, device="cuda")
    for m in range(9):
        s = (-1.0)**m
        cm = A @ (w * u**(2 * m)) * (s / math.factorial(2 * m))
        if m == 0:
            h0 = cm
        h += cm[:, None] * z**(2 * m)
        if m < 8:
            h -= (B @ (w * u**(2 * m + 1)) * (s / math.factorial(2 * m + 1)))[:, None] * z**(2 * m + 1)
    j = h.abs().argmax(dim=1)
    hp, dp = h.gather(1, j[:, None])[:, 0].clone(), grid[j].clone()
    sel = torch.argsort(hp.abs(), descending=True, stable=True)[:top]
    x = _newton(A[sel], B[sel], g, w, dp[sel], 4, 1e-5, 1e-13)
    hx = _h(A[sel], B[sel], g, w, x)[0]
    better = hx.abs() > h0[sel].abs()
    hp[sel] = torch.where(better, hx, h0[sel])
    dp[sel] = torch.where(better, x, torch.zeros_like(x))
    return [h0, hp, dp]


def _exact_screen(case, seed, d):
    d = d.truncate(256)
    c = _points(case, seed)
    T = _Exact(d, np.exp(-case["k"] * d.gamma * d.gamma))
    sf = _fix_floor(hit_polish.SCREEN_STEP)
    V = _limbs(_shift(c, c.delta))
    step = _Exact(d, None).cs(_limbs([sf]), 0, d.n)
    D = torch.atan2(step[1], step[0])[0]
    wr, wi = 2.0 * T.w * T.cr, 2.0 * T.w * T.ci
    S = torch.zeros(case["P"], 7, dtype=torch.float64, device="cuda")
    out = torch.full((case["P"], 3), -1.0, dtype=torch.float64, device="cuda")
    alive = torch.ones(case["P"], dtype=torch.bool, device="cuda")
    a = 0
    for s, (b, thr) in enumerate(zip(*hit_polish.SCREEN_GPU)):
        co, si = T.cs(V, a, b)
        re, im = co * wr[a:b] - si * wi[a:b], si * wr[a:b] + co * wi[a:b]
        for m in range(-3, 4):
            S[:, m + 3] += re @ torch.cos(m * D[a:b]) - im @ torch.sin(m * D[a:b])
        best = S.abs().amax(dim=1)
        out[:, s] = torch.where(alive, best, out[:, s])
        alive &= best >= thr
        a = b
    return [out, None]
