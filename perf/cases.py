"""Performance cases: the solves that users of this library run, through its C ABI.

A case is one call (or one round trip of a server) with everything a program has in hand
before it: the problem's arrays on the GPU, the objective's handle, the batch or the server.
Every solve runs a fixed number of iterations (all tolerances 0, the iteration limit ends
it), so that a pass does the same work on every input.

The problems are the library's two objectives: the synthetic bounded grid problem that its
benchmark is quoted on, and dsscfg, the example objective of the library it replaces.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lbfgsb-gpu_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import lbfgsb_b200 as LB  # noqa: E402

_FORM = {"f64": 0, "f32": 0, "mixed": 1, "bf16": 2}


def _solve(name, objective, nx, ny, form, driver, bound, iterations, m=8, proj=False):
    c = {"kind": "solve", "objective": objective, "nx": nx, "ny": ny, "form": form,
         "driver": driver, "bound": bound, "iterations": iterations, "m": m, "proj": proj}
    return dict(c, name=name) if name else c


def _many(name, kind, count, lo, hi, form, iterations):
    c = {"kind": kind, "count": count, "lo": lo, "hi": hi, "form": form, "iterations": iterations}
    return dict(c, name=name) if name else c


def listed():
    return [
        # The smallest call: one projected-gradient norm, as a solver callback issues it.
        {"kind": "projgr", "n": 65536, "name": "projgr_64k"},
        # The example program at its smallest size, unbounded, with a host callback: latency.
        _solve("dsscfg_64_f64", "dsscfg", 64, 64, "f64", "host", 0.0, 40),
        # The example program at its published FP64 size, with its box 0 <= x <= 0.25.
        _solve("dsscfg_256_f64_box", "dsscfg", 256, 256, "f64", "host", 0.25, 30),
        # An odd, ragged grid with a short memory and the projected subspace step.
        _solve("synth_333_f64_m5_proj", "synth", 333, 333, "f64", "device", 0.01, 30, m=5, proj=True),
        # A medium FP32 solve whose objective stays on the device (one CUDA graph a round).
        _solve("synth_1024_f32_device", "synth", 1024, 1024, "f32", "device", 1.0, 16),
        # Tight bounds: the first Cauchy steps walk hundreds of thousands of breakpoints.
        _solve("walk_512_f64", "synth", 512, 512, "f64", "host", 3e-7, 5),
        # The mixed-precision form at the larger of the two published FP32 sizes' scale.
        _solve("synth_2048_mixed", "synth", 2048, 2048, "mixed", "host", 1.0, 14),
        # The same with bfloat16 history.
        _solve("synth_2048_bf16", "synth", 2048, 2048, "bf16", "device", 1.0, 14),
        # The largest ordinary solves: the headline problem in FP64 and in plain FP32.
        _solve("synth_4096_f64", "synth", 4096, 4096, "f64", "host", 1.0, 12),
        _solve("synth_4096_f32", "synth", 4096, 4096, "f32", "host", 1.0, 12),
        # Many independent solves of mixed sizes in one call.
        _many("batch_192_f32", "batch", 192, 32, 512, "f32", 12),
        # A burst of requests to the continuous-batching server.
        _many("serve_48_mixed", "serve", 48, 64, 768, "mixed", 12),
    ]


# iterations * n of a single solve: at most the largest listed case's
_MOST = 4096 * 4096 * 12


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    r = rng.random()
    if r < 0.06:
        return {"kind": "projgr", "n": _log_int(rng, 1000, 1 << 22)}
    if r < 0.16:
        return _many(None, "batch", _log_int(rng, 24, 192), _log_int(rng, 16, 48),
                     _log_int(rng, 200, 512), rng.choice(["f32", "f32", "f64", "mixed"]),
                     rng.randint(8, 12))
    if r < 0.24:
        return _many(None, "serve", _log_int(rng, 8, 48), _log_int(rng, 32, 96),
                     _log_int(rng, 256, 768), rng.choice(["mixed", "f32", "bf16"]),
                     rng.randint(6, 12))
    form = rng.choice(["f64", "f64", "f32", "f32", "mixed", "bf16"])
    driver = rng.choice(["host", "device"])
    m = rng.choice([8, 8, 8, 5, 3])
    # a float f stops resolving the decrease after a while: fewer iterations
    if rng.random() < 0.25:
        nx, ny = _log_int(rng, 24, 2048), _log_int(rng, 24, 2048)
        f64 = rng.random() < 0.75
        it = (40 if nx * ny < 70000 else 20) if f64 else 8
        return _solve(None, "dsscfg", nx, ny, "f64" if f64 else "f32", "host",
                      rng.choice([0.0, 0.0, 0.25, 0.1]), it, m)
    if rng.random() < 0.12:
        s = _log_int(rng, 64, 512)
        return _solve(None, "synth", s, s, "f64", driver, 0.08 / (s * s), 5, m)
    s = _log_int(rng, 24, 4000)
    it = (30 if s < 400 else 14) if form == "f64" else 12
    return _solve(None, "synth", s, s, form, driver, rng.choice([1.0, 1.0, 0.05, 0.0]),
                  min(it, _MOST // (s * s)), m, rng.random() < 0.2)


# ---- the problems ------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _problem(case, seed):
    """The arrays of one problem on the GPU: the start point, the bounds, and the fields."""
    n = case["nx"] * case["ny"]
    rt = torch.float64 if case["form"] == "f64" else torch.float32
    gen = _gen(seed)

    def u(lo, hi):
        return torch.rand(n, dtype=rt, device="cuda", generator=gen) * (hi - lo) + lo

    p = {"n": n, "rt": rt}
    b = case["bound"]
    if case["objective"] == "dsscfg":
        # the example's parameter is 1; its start point, moved a little
        p["lam"] = 0.5 + (int(seed) * 0.6180339887498949) % 1.0
        x = torch.empty(n, dtype=rt, device="cuda")
        k = torch.arange(n, device="cuda")
        i, j = (k % case["nx"]).to(rt), (k // case["nx"]).to(rt)
        d = torch.minimum(torch.minimum(i, case["nx"] - i) / (case["nx"] + 1),
                          torch.minimum(j, case["ny"] - j) / (case["ny"] + 1))
        x = p["lam"] / (p["lam"] + 1) * torch.sqrt(d) * u(0.99, 1.01)
        p["l"] = torch.zeros_like(x)
        p["u"] = torch.full_like(x, b)
        p["nbd"] = torch.full((n,), 2 if b > 0 else 0, dtype=torch.int32, device="cuda")
        p["x0"] = torch.minimum(x, p["u"]) if b > 0 else x
        return p
    p["kappa"], p["w"] = u(0.5, 2.0), u(0.0, 1.0)
    p["t"] = torch.randn(n, dtype=rt, device="cuda", generator=gen)
    p["b"] = torch.randn(n, dtype=rt, device="cuda", generator=gen) * 2
    p["l"] = torch.full((n,), -b if b > 0 else -1.0, dtype=rt, device="cuda")
    p["u"] = torch.full((n,), b if b > 0 else 1.0, dtype=rt, device="cuda")
    kind = torch.rand(n, device="cuda", generator=gen)
    p["nbd"] = torch.where(kind < 0.8, 2, torch.where(kind < 0.9, 1, 0)).to(torch.int32)
    if b == 0:
        p["nbd"].zero_()
    p["x0"] = torch.zeros(n, dtype=rt, device="cuda")
    # f(x0) subtracted from f, so that a float f resolves the decrease
    h2 = 1.0 / (case["nx"] + 1) ** 2
    p["f0"] = 0.0
    if rt == torch.float32:
        w, t = p["w"].double(), p["t"].double()
        p["f0"] = float(h2 * (w * torch.nn.functional.softplus(-t) + 0.05).sum())
    return p


def _option(case):
    o = LB.default_option(np.float64 if case["form"] == "f64" else np.float32)
    o.eps_f = o.eps_g = o.eps_x = 0.0
    o.max_iteration = case["iterations"]
    o.hessian_approximate_dimension = case.get("m", 8)
    return o


class _Solve:
    """One problem, its objective's handle and the call's arguments."""

    def __init__(self, case, seed):
        lib = LB.load()
        p = _problem(case, seed)
        self.is64 = case["form"] == "f64"
        sfx = "f64" if self.is64 else "f32"
        self.x0, self.x, self.keep = p["x0"], torch.empty_like(p["x0"]), p
        self.opt = _option(case)
        self.summ = LB.SummaryF64() if self.is64 else LB.SummaryF32()
        self.ext = LB.Ext(_FORM[case["form"]], 0, LB.TRACE_CB(), None, 1 if case["proj"] else 0)
        if case["objective"] == "dsscfg":
            self.obj = LB.DsscfgObjective(case["nx"], case["ny"], p["lam"])
            f = self.obj.f64 if self.is64 else self.obj.f32
        else:
            host = {k: p.pop(k).double().cpu().numpy() for k in ("kappa", "w", "t", "b")}
            self.obj = LB.SynthObjective(dict(host, s=case["nx"], f_offset=p["f0"]),
                                         single_precision_fields=not self.is64)
            self.obj._fields = None  # the handle keeps its own copy
            dev = case["driver"] == "device"
            f = ((self.obj.d64 if self.is64 else self.obj.d32) if dev
                 else (self.obj.f64 if self.is64 else self.obj.f32))
        a = (p["n"], self.x.data_ptr(), p["nbd"].data_ptr(), p["l"].data_ptr(), p["u"].data_ptr(),
             C.byref(self.opt), f)
        tail = (self.obj.handle, None, C.byref(self.ext), C.byref(self.summ))
        if case["driver"] == "device":
            self.fn, self.args = getattr(lib, "lbfgsb_b200_minimize_device_" + sfx), a + tail
        else:
            self.fn, self.args = getattr(lib, "lbfgsb_b200_minimize_ext_" + sfx), a + (None, None) + tail

    def run(self):
        self.x.copy_(self.x0)
        rc = self.fn(*self.args)
        s = self.summ
        real = np.float64 if self.is64 else np.float32
        # residual_f is left out: a difference of two nearly equal values of f
        return {"x": self.x, "residual_g": real(s.residual_g), "residual_x": real(s.residual_x),
                "iterations": int(s.num_iteration), "info": int(s.info), "status": int(rc)}

    def __del__(self):
        self.obj.close()


class _Many:
    """A batch of synthetic problems with log-uniform grid sides; for the server, the server."""

    def __init__(self, case, seed):
        rng = np.random.default_rng(int(seed))
        # the sides of a case are its own, the same for every seed, as is its work
        q = (np.arange(case["count"]) * 0.6180339887498949 + 0.11) % 1.0
        sides = np.rint(np.exp(np.log(case["lo"]) + q * np.log(case["hi"] / case["lo"]))).astype(int)
        seeds = rng.integers(1, 1 << 40, size=case["count"])
        self.case = case
        self.is64 = case["form"] == "f64"
        self.batch = LB.SynthBatch(sides, seeds, single_precision_fields=not self.is64,
                                   dtype=np.float64 if self.is64 else np.float32)
        self.flat = torch.zeros(sum(self.batch.n), device="cuda",
                                dtype=torch.float64 if self.is64 else torch.float32)
        self.xs = list(self.flat.split(self.batch.n))
        self.opt = _option(case)
        self.server = None
        if case["kind"] == "serve":
            self.server = LB.BatchServer(self.batch, self.opt, form=_FORM[case["form"]])

    def run(self):
        self.flat.zero_()
        if self.server is None:
            rc, stat, summ, _ = LB.solve_batch_device(self.batch, self.xs, self.opt,
                                                      form=_FORM[self.case["form"]])
            out = [(s, m) for s, m in zip(stat, summ)]
        else:
            torch.cuda.current_stream().synchronize()  # the server reads x on its own stream
            tickets = [self.server.submit(p, x)[1] for p, x in enumerate(self.xs)]
            out = [self.server.wait(t)[:2] for t in tickets]
        real = np.float64 if self.is64 else np.float32
        return {"x": self.flat,
                "residual_g": np.array([m.residual_g for _, m in out], dtype=real),
                "iterations": np.array([m.num_iteration for _, m in out]),
                "info": np.array([m.info for _, m in out]),
                "status": np.array([s for s, _ in out])}

    def __del__(self):
        if getattr(self, "server", None):
            self.server.close()
        if getattr(self, "batch", None):
            self.batch.close()


class _Projgr:
    def __init__(self, case, seed):
        n, gen = case["n"], _gen(seed)
        self.x = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
        self.g = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
        self.l, self.u = torch.full_like(self.x, -1.0), torch.full_like(self.x, 1.0)
        self.nbd = torch.randint(0, 4, (n,), dtype=torch.int32, device="cuda", generator=gen)
        self.out = torch.zeros(1, dtype=torch.float64, device="cuda")
        self.args = (n, self.x.data_ptr(), self.g.data_ptr(), self.nbd.data_ptr(), self.l.data_ptr(),
                     self.u.data_ptr(), self.out.data_ptr(), None)
        self.fn = LB.load().lbfgsb_b200_projgr_noalloc_f64

    def run(self):
        self.fn(*self.args)
        return self.out


def prepare(case, seed):
    return {"solve": _Solve, "batch": _Many, "serve": _Many, "projgr": _Projgr}[case["kind"]](case, seed)


def run(state):
    return state.run()


def work(case):
    """One solve: every iteration's evaluation reads x and the fields and writes g; the
    iteration reads x, g, the bounds and the previous x and g, writes the new x, the pair
    (s, y) and the codes, and reads the history twice (the direction needs the products with
    the pair that the evaluation has just given)."""
    if case["kind"] == "projgr":
        return {"bytes": case["n"] * 36.0, "flops": case["n"] * 3.0}
    R = 8 if case["form"] == "f64" else 4
    H = {"f64": 8, "f32": 4, "mixed": 4, "bf16": 2}[case["form"]]
    m = case.get("m", 8)
    k = case["iterations"] + 1
    cols = sum(min(i, m) for i in range(k)) / k
    if case["kind"] == "solve":
        n = float(case["nx"] * case["ny"])
        fields = 4 if case["objective"] == "synth" else 0
    else:
        q = (np.arange(case["count"]) * 0.6180339887498949 + 0.11) % 1.0
        sides = np.rint(np.exp(np.log(case["lo"]) + q * np.log(case["hi"] / case["lo"])))
        n, fields = float((sides * sides).sum()), 4
    vectors = R * (2 + fields) + R * 7 + 4 + 1 + 2 * H
    return {"bytes": n * k * (vectors + 2 * 2 * cols * H), "flops": n * k * (2 * 7 * 2 * cols + 40)}


# ---- the same in 64 bits, with plain torch -------------------------------------------------

def _objective(case, p):
    nx, ny = case["nx"], case["ny"]
    D = {k: v.double().view(ny, nx) for k, v in p.items() if k in ("kappa", "w", "t", "b")}
    if case["objective"] == "synth":
        h2 = 1.0 / (nx + 1) ** 2

        def fun(x):
            X = x.view(ny, nx)
            e = torch.nn.functional.pad(X, (0, 1, 0, 1))
            de, dn = e[:-1, 1:] - X, e[1:, :-1] - X
            z = X - D["t"]
            f = (0.5 * D["kappa"] * (de * de + dn * dn)).sum() + h2 * (
                D["w"] * torch.nn.functional.softplus(z, threshold=700) - D["b"] * X
                + 0.05 * torch.cos(3 * X)).sum() - p["f0"]
            g = -D["kappa"] * (de + dn) + h2 * (D["w"] * torch.sigmoid(z) - D["b"] - 0.15 * torch.sin(3 * X))
            g[:, 1:] += (D["kappa"] * de)[:, :-1]
            g[1:, :] += (D["kappa"] * dn)[:-1, :]
            return float(f), g.reshape(-1)
        return fun
    hx, hy, lam = 1.0 / (nx + 1), 1.0 / (ny + 1), p["lam"]
    if case["form"] != "f64":
        lam = float(np.float32(lam))
    area = 0.5 * hx * hy

    def fun(x):
        P = torch.nn.functional.pad(x.view(ny, nx), (1, 1, 1, 1))
        X = P[1:-1, 1:-1]
        dxl, dyl = (P[1:-1, 2:] - X) / hx, (P[2:, 1:-1] - X) / hy  # a node's lower triangle
        dxu, dyu = (X - P[1:-1, :-2]) / hx, (X - P[:-2, 1:-1]) / hy  # and its upper one
        i, j = torch.arange(nx, device=x.device), torch.arange(ny, device=x.device)[:, None]
        right, top, left, bottom = (v.to(x.dtype) for v in (i < nx - 1, j < ny - 1, i > 0, j > 0))
        corners = 2.0 + right + top + left + bottom
        E = torch.exp(X)
        f = area * (0.5 * (dxl * dxl + dyl * dyl + dxu * dxu + dyu * dyu).sum()
                    - lam / 3.0 * ((corners * E).sum() + 2.0 * (nx + ny)))
        g = -dxl / hx * (1 + right) + dxu / hx * (1 + left) - dyl / hy * (1 + top) \
            + dyu / hy * (1 + bottom) - corners * lam / 3.0 * E
        return float(f), (g * area).reshape(-1)
    return fun


def _dcstep(stx, fx, dx, sty, fy, dy, stp, fp, dp, brackt, lo, hi):
    sgn = dp * (dx / abs(dx))

    def cubic(a, fa, da, sign, clamp=False):
        th = 3 * (fa - fp) / (stp - a) + da + dp
        s = max(abs(th), abs(da), abs(dp))
        rad = (th / s) ** 2 - da / s * (dp / s)
        return th, sign * s * math.sqrt(max(0.0, rad) if clamp else rad)

    if fp > fx:
        th, ga = cubic(stx, fx, dx, -1 if stp < stx else 1)
        r = (ga - dx + th) / (ga - dx + ga + dp)
        c = stx + r * (stp - stx)
        q = stx + dx / ((fx - fp) / (stp - stx) + dx) / 2 * (stp - stx)
        new, brackt = (c if abs(c - stx) < abs(q - stx) else c + (q - c) / 2), True
    elif sgn < 0:
        th, ga = cubic(stx, fx, dx, -1 if stp > stx else 1)
        r = (ga - dp + th) / (ga - dp + ga + dx)
        c, q = stp + r * (stx - stp), stp + dp / (dp - dx) * (stx - stp)
        new, brackt = (c if abs(c - stp) > abs(q - stp) else q), True
    elif abs(dp) < abs(dx):
        th, ga = cubic(stx, fx, dx, -1 if stp > stx else 1, True)
        r = (ga - dp + th) / (ga + (dx - dp) + ga)
        c = stp + r * (stx - stp) if r < 0 and ga != 0 else (hi if stp > stx else lo)
        q = stp + dp / (dp - dx) * (stx - stp)
        if brackt:
            new = c if abs(c - stp) < abs(q - stp) else q
            lim = stp + 0.66 * (sty - stp)
            new = min(lim, new) if stp > stx else max(lim, new)
        else:
            new = max(lo, min(hi, c if abs(c - stp) > abs(q - stp) else q))
    elif brackt:
        th, ga = cubic(sty, fy, dy, -1 if stp > sty else 1)
        r = (ga - dp + th) / (ga - dp + ga + dy)
        new = stp + r * (sty - stp)
    else:
        new = hi if stp > stx else lo
    if fp > fx:
        sty, fy, dy = stp, fp, dp
    else:
        if sgn < 0:
            sty, fy, dy = stx, fx, dx
        stx, fx, dx = stp, fp, dp
    return stx, fx, dx, sty, fy, dy, new, brackt


def _search(phi, f0, g0, stp, stpmax):
    """More' and Thuente's line search (ftol 1e-3, gtol 0.9, xtol 0.1): the accepted step."""
    gt, brackt, stage1 = 1e-3 * g0, False, True
    width, width1 = stpmax, 2 * stpmax
    a, fa, da, b, fb, db = 0.0, f0, g0, 0.0, f0, g0
    lo, hi = 0.0, stp + 4 * stp
    for _ in range(20):
        f, g, extra = phi(stp)
        ft = f0 + stp * gt
        if stage1 and f <= ft and g >= 0:
            stage1 = False
        if ((brackt and (stp <= lo or stp >= hi or hi - lo <= 0.1 * hi)) or (stp == stpmax and f <= ft and g <= gt)
                or (stp == 0 and (f > ft or g >= gt)) or (f <= ft and abs(g) <= 0.9 * -g0)):
            return stp, f, g, extra
        mod = gt if stage1 and f <= fa and f > ft else 0.0
        a, fm, dm, b, fn, dn, stp, brackt = _dcstep(a, fa - a * mod, da - mod, b, fb - b * mod, db - mod, stp,
                                                    f - stp * mod, g - mod, brackt, lo, hi)
        fa, fb, da, db = fm + a * mod, fn + b * mod, dm + mod, dn + mod
        if brackt:
            if abs(b - a) >= 0.66 * width1:
                stp = a + 0.5 * (b - a)
            width1, width = width, abs(b - a)
            lo, hi = min(a, b), max(a, b)
        else:
            lo, hi = stp + 1.1 * (stp - a), stp + 4 * (stp - a)
        stp = min(max(stp, 0.0), stpmax)
        if brackt and (stp <= lo or stp >= hi or hi - lo <= 0.1 * hi):
            stp = a
    raise ArithmeticError("no step")


def _middle(S, Y, theta):
    SY, SS = S @ Y.T, S @ S.T
    D, L = torch.diag(torch.diag(SY)), torch.tril(SY, -1)
    return torch.linalg.inv(torch.cat([torch.cat([-D, L.T], 1), torch.cat([L, theta * SS], 1)], 0))


def _lbfgsb(fun, x, nbd, l, u, m, iterations, proj):
    """L-BFGS-B 2.1 (Byrd, Lu, Nocedal and Zhu, 1995) in dense compact form."""
    inf = float("inf")
    l = torch.where((nbd == 1) | (nbd == 2), l, torch.full_like(l, -inf))
    u = torch.where(nbd >= 2, u, torch.full_like(u, inf))
    bounded, boxed = bool((nbd > 0).any()), bool((nbd == 2).all())
    x = torch.minimum(torch.maximum(x, l), u)
    f, g = fun(x)
    n = x.numel()
    S = x.new_zeros((0, n))
    Y, theta, M = S, 1.0, None

    def pgnorm():
        return float((torch.minimum(torch.maximum(x - g, l), u) - x).abs().max())

    step = 0.0
    for it in range(iterations + 1):
        W = torch.cat([Y, theta * S], 0)  # 2k x n
        k2 = W.shape[0]
        t = torch.where(g < 0, (x - u) / g, torch.where(g > 0, (x - l) / g, torch.full_like(x, inf)))
        d = torch.where(t > 0, -g, torch.zeros_like(g))
        xc, free = x, torch.ones_like(x, dtype=torch.bool)
        c = x.new_zeros(k2)
        if bounded or k2 == 0:
            p = W @ d
            f1, f2o = -float(d @ d), theta * float(d @ d)
            f2 = f2o - (float(p @ (M @ p)) if k2 else 0.0)
            dt, told, last = -f1 / f2, 0.0, None
            moving = torch.nonzero((t > 0) & (t < inf) & (g != 0)).flatten()
            passed = moving.new_zeros(0)
            if moving.numel() and float(t[moving].min()) <= dt:
                order = moving[torch.argsort(t[moving], stable=True)]
                # the walk reads a bounded piece of the sorted breakpoints at a time
                pn, cn, Mn = p.cpu().numpy(), c.cpu().numpy(), M.cpu().numpy() if k2 else None
                done, pos, left = False, 0, order.numel()
                while not done and pos < order.numel():
                    part = order[pos:pos + 65536]
                    tb, gb = t[part].cpu().numpy().tolist(), g[part].cpu().numpy().tolist()
                    zb = (torch.where(g[part] < 0, u[part], l[part]) - x[part]).cpu().numpy().tolist()
                    Wb = W[:, part].T.contiguous().cpu().numpy()
                    for q in range(len(tb)):
                        dl = tb[q] - told
                        if dt < dl:
                            done = True
                            break
                        told, left, db = tb[q], left - 1, -gb[q]
                        pos += 1
                        if left == 0 and moving.numel() == n:
                            cn, done, dt = cn + dl * pn, True, 0.0
                            break
                        f1 += dl * f2 + db * db - theta * db * zb[q]
                        f2 -= theta * db * db
                        if k2:
                            cn = cn + dl * pn
                            v = Mn @ Wb[q]
                            f1 += db * float(v @ cn)
                            f2 += 2 * db * float(v @ pn) - db * db * float(v @ Wb[q])
                            pn = pn - db * Wb[q]
                        f2 = max(5e-16 * f2o, f2)
                        dt = -f1 / f2
                p, c = torch.from_numpy(np.array(pn)).to(x), torch.from_numpy(np.array(cn)).to(x)
                passed = order[:pos]
            dt = max(dt, 0.0)
            told += dt
            c = c + dt * p
            d = d.clone()
            d[passed] = 0
            xc = x + told * d
            xc[passed] = torch.where(g[passed] < 0, u[passed], l[passed])
            free = t > 0
            free[passed] = False
            free |= g == 0
            free &= l < u
        z = xc
        if k2 and bool(free.any()):
            Wf = W * free
            r = -g.clone() if not bounded else -theta * (xc - x) - g + W.T @ (M @ c)
            N = torch.eye(k2, dtype=x.dtype, device=x.device) - M @ (Wf @ Wf.T) / theta
            v = torch.linalg.solve(N, M @ (Wf @ r))
            dn = (r / theta + (W.T @ v) / theta ** 2) * free
            if proj and bounded:
                z = torch.minimum(torch.maximum(xc + dn, l), u)
            if not proj or not bounded or float((z - x) @ g) > 0:
                room = torch.where(dn < 0, (l - xc) / dn, torch.where(dn > 0, (u - xc) / dn, torch.full_like(x, inf)))
                al = min(1.0, float(room.min()))
                z = torch.minimum(torch.maximum(xc + al * dn, l), u)
        d = z - x
        g0 = float(d @ g)
        if g0 >= 0:
            return None  # the memory reset is the solver's own business
        smax = 1e10
        if bounded:
            room = torch.where(d < 0, (l - x) / d, torch.where(d > 0, (u - x) / d, torch.full_like(x, inf)))
            smax = 1.0 if it == 0 else min(1e10, float(room.min()))
        dd = float(d @ d)
        s0 = min(1.0 / math.sqrt(dd), smax) if it == 0 and not boxed else 1.0
        if s0 > smax:
            return None

        def phi(a):
            xn = z if a == 1.0 else a * d + x
            fn, gn = fun(xn)
            return fn, float(gn @ d), (xn, gn)

        a, fn, gd, (xn, gn) = _search(phi, f, g0, s0, smax)
        s, y = a * d, gn - g
        step = float((xn - x).norm())
        dr, dg = (gd - g0) * a, -g0 * a
        x, f, g = xn, fn, gn
        if dr > 5e-16 * dg:
            S = torch.cat([S, s[None]], 0)[-m:]
            Y = torch.cat([Y, y[None]], 0)[-m:]
            theta = float(y @ y) / dr
            M = _middle(S, Y, theta)
    return x, pgnorm(), step


def _exact_solve(case, p, n, m):
    d = {k: (v.double() if torch.is_tensor(v) and v.is_floating_point() else v) for k, v in p.items()}
    try:
        return _lbfgsb(_objective(case, d), d["x0"], d["nbd"], d["l"], d["u"], m, case["iterations"],
                       case.get("proj", False))
    except (ArithmeticError, ValueError):
        return None


def exact(case, seed):
    if case["kind"] == "projgr":
        s = _Projgr(case, seed)
        pg = torch.where((s.g < 0) & (s.nbd >= 2), torch.maximum(s.x - s.u, s.g), s.g)
        pg = torch.where((s.g >= 0) & ((s.nbd == 1) | (s.nbd == 2)), torch.minimum(s.x - s.l, s.g), pg)
        return pg.abs().max().reshape(1)
    if case["kind"] != "solve":
        return None  # hundreds of solves in turn: too long
    p = _problem(case, seed)
    if case["form"] != "f64" and p["n"] > 2_500_000:
        return None  # a float f resolves too little of an iteration's decrease: other steps
    r = _exact_solve(case, p, p["n"], case["m"])
    if r is None:
        return None
    return {"x": r[0], "residual_g": np.float64(r[1]), "residual_x": np.float64(r[2]), "iterations": None, "info": None, "status": None}
