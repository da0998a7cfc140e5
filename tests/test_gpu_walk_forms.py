"""What the breakpoint walk decides in the FP32 forms.  A separable quadratic whose first `passed`
variables have bounds of 1e-7 that the first Cauchy step reaches: the first iteration must pass
the breakpoints that the FP64 oracle passes, and each of these variables must end exactly at the
bound on the side of its centre (a walk that left them, or sent them to the other bound, would
change f by less than the forms' tolerance)."""
import numpy as np
import pytest

from cases import _quad, apply_options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("passed", [1, 127, 129, 513, 3073])
def test_walked_variables_end_at_their_bounds(passed, form):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import lbfgsb_b200 as LB
    from oracle import binding as OB
    n = passed + 70
    k = np.arange(n)
    a = 1.0 + 0.5 * ((k * 7) % 5) + 0.01 * (k % 97)
    c = 0.9 * np.sin(1.7 * k + 0.3)
    c = np.where(np.abs(c) < 0.05, 0.05, c)
    tight = k < passed
    b = (1e-7 * (1.0 + ((k * 7919) % 10007) / 10007.0)).astype(np.float32).astype(np.float64)
    nbd = np.where(tight, 2, 0).astype(np.int32)
    p = _quad(n, a, c, np.where(tight, -b, 0.0), np.where(tight, b, 0.0), nbd)

    def opt(mod, dt):
        return apply_options(mod.default_option(dt), {"eps_f": 1e-9, "eps_g": 1e-8, "eps_x": 1e-9,
                                                      "max_iteration": 8})
    ref = OB.run_cpu("oracle", p, np.float64, option=opt(OB, np.float64), trace=True)
    got = LB.solve(p, np.float32, option=opt(LB, np.float32), objective="host", form=form, trace=True)
    for key in ("nint", "nbreak", "at_lower", "at_upper"):
        assert got.trace[0][key] == ref.trace[0][key], key
    assert ref.trace[0]["nint"] >= passed
    np.testing.assert_array_equal(got.x[tight], (np.sign(c) * b)[tight].astype(np.float32))
