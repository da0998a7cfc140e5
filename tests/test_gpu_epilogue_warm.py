"""The pass epilogues' code is warmed beside the streaming when every CTA has at least eight tiles
of 512 variables (n >= 8 * 512 * 148 on a 148-SM chip).  On both sides of that size, with enough
iterations to fill and shift the memory, FP64 must reproduce the oracle's discrete trace with f
within 1e-10 per iteration (the parity tests' bounds)."""
import numpy as np
import pytest

from cases import apply_options

pytestmark = pytest.mark.gpu

TRACE_KEYS = ["nint", "nbreak", "nfree", "nenter", "nleave", "col", "head", "iword",
              "free_hash", "at_lower", "at_upper", "nfgv", "ifun"]


@pytest.mark.parametrize("s", [778, 779])
def test_f64_trace_around_the_warmed_size(s):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import lbfgsb_b200 as LB
    import synth
    from oracle import binding as OB
    prob = dict(synth.synth_problem(s, seed=0), kind="synth")

    def opt(mod):
        return apply_options(mod.default_option(np.float64), {"eps_f": 0.0, "eps_g": 0.0,
                                                              "eps_x": 0.0, "max_iteration": 11})
    a = OB.run_cpu("oracle", prob, np.float64, option=opt(OB), trace=True, record=False)
    b = LB.solve(prob, np.float64, option=opt(LB), objective="host", trace=True, record=False)
    assert len(a.trace) == len(b.trace)
    for ra, rb in zip(a.trace, b.trace):
        diff = {k: (ra[k], rb[k]) for k in TRACE_KEYS if ra[k] != rb[k]}
        assert not diff, (ra["iter"], diff)
        assert abs(ra["f"] - rb["f"]) <= 1e-10 * max(1.0, abs(ra["f"]))
