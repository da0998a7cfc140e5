"""The pass epilogues on both sides of the size from which their code is warmed (n >= 8 * 512 * 148
on a 148-SM chip), in the forms and memories that the FP64 trace test does not run.  A one-rank
sharded solve runs every epilogue in a launch of its own, which never warms anything: the plain
solve must give its bits, over enough iterations to fill and shift the memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s", [778, 779])
@pytest.mark.parametrize("dtype,form,m", [(np.float64, 0, 5), (np.float32, 0, 8), (np.float32, 0, 5),
                                          (np.float32, 1, 8), (np.float32, 2, 3)])
def test_warmed_epilogues_give_the_same_bits(s, dtype, form, m):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import lbfgsb_b200 as LB
    import synth
    prob = dict(synth.synth_problem(s, seed=0), kind="synth")
    opt = LB.default_option(dtype)
    opt.eps_f = opt.eps_g = opt.eps_x = 0.0
    opt.max_iteration, opt.hessian_approximate_dimension = 11, m
    a = LB.solve_sharded(prob, 1, dtype, option=opt, form=form)
    b = LB.solve(prob, dtype, option=opt, objective="host", form=form, record=False)
    assert (a.info, a.num_iteration) == (b.info, b.num_iteration)
    assert a.residual_g == b.residual_g and a.residual_x == b.residual_x
    np.testing.assert_array_equal(a.x, b.x)
