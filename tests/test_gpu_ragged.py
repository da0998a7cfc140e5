"""Sizes around the tile edge of the staged passes (512 variables): the partial last tile is
staged as whole 16-byte words plus a ragged end of plain loads, which differ by element size
(8, 4, 2 and 1 bytes, and the free-set bits).  Bounded separable quadratics whose variables
all differ, so that a wrong value in the tail changes the run: FP64 must reproduce the
oracle's whole discrete trace with f within 1e-10 per iteration, and every precision form
must reach the FP64 oracle's final f within the FP32 tolerance of the forms, 1e-5."""
import numpy as np
import pytest

from cases import _quad, apply_options

pytestmark = pytest.mark.gpu

TRACE_KEYS = ["nint", "nbreak", "nfree", "nenter", "nleave", "col", "head", "iword",
              "free_hash", "at_lower", "at_upper", "nfgv", "ifun"]
SIZES = [9, 15, 17, 31, 33, 511, 513, 519, 527, 529, 1000, 1023]


@pytest.fixture(scope="module")
def LB():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import lbfgsb_b200
    lbfgsb_b200.load()
    return lbfgsb_b200


def _prob(n):
    k = np.arange(n)
    a = 1.0 + 0.5 * ((k * 7) % 5) + 0.01 * (k % 97)
    c = 0.9 * np.sin(1.7 * k + 0.3)
    nbd = np.array([2, 1, 0, 3], np.int32)[k % 4]
    return _quad(n, a, c, np.full(n, -0.5), np.full(n, 0.4), nbd)


def _oracle(n):
    from oracle import binding as OB
    opt = apply_options(OB.default_option(np.float64), {"eps_f": 1e-8, "eps_g": 1e-8, "eps_x": 1e-8})
    return OB.run_cpu("oracle", _prob(n), np.float64, option=opt, trace=True)


def _gpu(LB, n, dtype, form=0, trace=False):
    opt = apply_options(LB.default_option(dtype), {"eps_f": 1e-8, "eps_g": 1e-8, "eps_x": 1e-8})
    return LB.solve(_prob(n), dtype, option=opt, objective="host", form=form, trace=trace)


@pytest.mark.parametrize("n", SIZES)
def test_f64_trace_at_tile_edges(LB, n):
    a, b = _oracle(n), _gpu(LB, n, np.float64, trace=True)
    assert (a.info, a.num_iteration, len(a.trace)) == (b.info, b.num_iteration, len(b.trace))
    for ra, rb in zip(a.trace, b.trace):
        diff = {k: (ra[k], rb[k]) for k in TRACE_KEYS if ra[k] != rb[k]}
        assert not diff, (ra["iter"], diff)
        assert abs(ra["f"] - rb["f"]) <= 1e-10 * max(1.0, abs(ra["f"]))


@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("n", [9, 513, 519, 1023])
def test_f32_forms_at_tile_edges(LB, n, form):
    a, b = _oracle(n), _gpu(LB, n, np.float32, form=form)
    fref = a.evals[-1][0]
    assert b.info in (1, 2, 4)
    assert abs(b.evals[-1][0] - fref) <= 1e-5 * max(1.0, abs(fref))
