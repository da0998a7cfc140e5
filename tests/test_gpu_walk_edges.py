"""Breakpoint walks whose lengths lie around the cooperative walk's block sizes: the
sub-batches of 128 keys its warps hand on, the pieces of 512 keys it sorts, the first chunk of
1024 and the doubled ones after it.  A bounded separable quadratic whose first `passed`
variables reach their tiny bounds within the first Cauchy step, the others unbounded (the walk
ends at the test) or absent (every variable ends at its bound).  FP64 must reproduce the
oracle's discrete trace with f within 1e-10 per iteration; the FP32 forms must reach its final
f within their tolerance, 1e-5.  One more run walks with the memory full (col > 0)."""
import numpy as np
import pytest

from cases import _quad, apply_options

pytestmark = pytest.mark.gpu

TRACE_KEYS = ["nint", "nbreak", "nfree", "nenter", "nleave", "col", "head", "iword",
              "free_hash", "at_lower", "at_upper", "nfgv", "ifun"]
LENGTHS = [1, 2, 127, 128, 129, 511, 512, 513, 1023, 1024, 1025, 3071, 3073, 9000]


@pytest.fixture(scope="module")
def LB():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import lbfgsb_b200
    lbfgsb_b200.load()
    return lbfgsb_b200


def _prob(passed, free):
    n = passed + free
    k = np.arange(n)
    a = 1.0 + 0.5 * ((k * 7) % 5) + 0.01 * (k % 97)
    c = 0.9 * np.sin(1.7 * k + 0.3)
    c = np.where(np.abs(c) < 0.05, 0.05, c)
    tight = k < passed
    b = 1e-7 * (1.0 + ((k * 7919) % 10007) / 10007.0)
    nbd = np.where(tight, 2, 0).astype(np.int32)
    return _quad(n, a, c, np.where(tight, -b, 0.0), np.where(tight, b, 0.0), nbd)


def _opt(mod, dt):
    return apply_options(mod.default_option(dt), {"eps_f": 1e-9, "eps_g": 1e-8, "eps_x": 1e-9,
                                                  "max_iteration": 8})


def _same(a, b):
    assert (a.info, a.num_iteration, len(a.trace)) == (b.info, b.num_iteration, len(b.trace))
    for ra, rb in zip(a.trace, b.trace):
        diff = {k: (ra[k], rb[k]) for k in TRACE_KEYS if ra[k] != rb[k]}
        assert not diff, (ra["iter"], diff)
        assert abs(ra["f"] - rb["f"]) <= 1e-10 * max(1.0, abs(ra["f"]))


@pytest.mark.parametrize("free", [0, 70])
@pytest.mark.parametrize("passed", LENGTHS)
def test_f64_walk_lengths(LB, passed, free):
    from oracle import binding as OB
    if passed + free < 8:
        pytest.skip("fewer variables than the memory holds pairs")
    p = _prob(passed, free)
    a = OB.run_cpu("oracle", p, np.float64, option=_opt(OB, np.float64), trace=True)
    b = LB.solve(p, np.float64, option=_opt(LB, np.float64), objective="host", trace=True)
    assert a.trace[0]["nint"] >= passed
    _same(a, b)


@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("passed", [127, 513, 3073])
def test_f32_walk_lengths(LB, passed, form):
    from oracle import binding as OB
    p = _prob(passed, 70)
    a = OB.run_cpu("oracle", p, np.float64, option=_opt(OB, np.float64), trace=True)
    b = LB.solve(p, np.float32, option=_opt(LB, np.float32), objective="host", form=form)
    fref = a.evals[-1][0]
    assert abs(b.evals[-1][0] - fref) <= 1e-5 * max(1.0, abs(fref))


@pytest.mark.parametrize("s", [48, 100])
def test_f64_walks_with_history(LB, s):
    """A tightly bounded grid problem, whose later iterations walk too (col > 0)."""
    import synth
    from oracle import binding as OB
    p = dict(synth.synth_problem(s, seed=0), kind="synth")
    p["l"] = p["l"] * (0.08 / s**2)
    p["u"] = p["u"] * (0.08 / s**2)

    def opt(mod):
        return apply_options(mod.default_option(np.float64), {"eps_f": 0.0, "eps_g": 0.0,
                                                              "eps_x": 0.0, "max_iteration": 8})
    r = OB.run_cpu("oracle", p, np.float64, option=opt(OB), trace=True, record=False)
    g = LB.solve(p, np.float64, option=opt(LB), objective="host", trace=True, record=False)
    assert sum(1 for t in r.trace if t["col"] > 0 and t["nint"] > 1) >= 2
    _same(r, g)
