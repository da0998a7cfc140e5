"""The history slots are not cleared when a solve starts: only slots that the solve has written may
be read.  Solves whose workspace comes from pool memory full of NaN bytes must give the bits of
solves on fresh memory, in every form, host- and device-driven, with a short memory and with one
that never fills; so must a batch whose history is overwritten at its first evaluation.

The pool is filled through a batched solve's segment: its objective sees x, the segment's first
buffer, and sets what follows it to 0xff (for the batch's own case the history alone).  The solve
then takes its buffers from the segment's start in the order X (3), G (2), dsub, S, Y.  Of the
segment X[0] and G[0] (1 and 4 of its vectors) stay finite; its size puts them before S and in Y
(`behind` = 6 of the solve's vectors a vector of the segment), or in S and behind Y (8)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _region(n, vectors):
    """Offset and bytes, in a batch segment of n FP32 variables, of what follows `vectors` of its
    seven vectors, up to the end of the two histories (nine slots each)."""
    ld = (n + 511) // 512 * 512
    return vectors * ld * 4, (7 - vectors + 18) * ld * 4


def _batch(LB, sides, eps_g, spoil, vectors=7):
    """A batched FP32 solve; spoil: the instances whose memory after `vectors` vectors is set to 0xff
    bytes at their first evaluation (before anything is written there)."""
    import torch
    lib = LB.load()
    cuda = C.CDLL("libcuda.so.1")
    cuda.cuMemsetD8Async.argtypes = [C.c_void_p, C.c_ubyte, C.c_size_t, C.c_void_p]
    cuda.cuStreamSynchronize.argtypes = [C.c_void_p]
    bt = LB.SynthBatch(sides, [11 + k for k in range(len(sides))])
    objective = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_int,
                            *[C.c_void_p] * 5)
    inner = objective(bt.objective)
    spoilt = []

    def call(user, count, ids, first, ctas, x, g, f, active, stream):
        if not spoilt:
            cuda.cuStreamSynchronize(stream)
            base = (C.c_void_p * count)()
            assert lib.lbfgsb_b200_copy(base, C.c_void_p(x), C.sizeof(base), 2) == 0
            for k in spoil:
                off, size = _region(sides[k] ** 2, vectors)
                assert cuda.cuMemsetD8Async(base[k] + off, 0xFF, size, stream) == 0
            spoilt.append(True)
        return inner(user, count, ids, first, ctas, x, g, f, active, stream)

    keep = objective(call)
    bt.objective = C.cast(keep, C.c_void_p).value
    xs = [torch.zeros(s * s, dtype=torch.float32, device="cuda") for s in sides]
    opt = LB.default_option(np.float32)
    opt.eps_f = opt.eps_x = 0.0
    opt.eps_g = eps_g
    opt.max_iteration = 14
    rc, stat, _, _ = LB.solve_batch_device(bt, xs, opt)
    assert rc == 0 and spoilt
    torch.cuda.synchronize()
    out = [x.cpu().numpy() for x in xs]
    bt.close()
    return out


@pytest.fixture(scope="module")
def LB():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import lbfgsb_b200
    lbfgsb_b200.load()
    return lbfgsb_b200


@pytest.mark.parametrize("dtype,form", [(np.float64, 0), (np.float32, 0), (np.float32, 1), (np.float32, 2)])
@pytest.mark.parametrize("behind", [6, 8])
@pytest.mark.parametrize("driven,m,iterations", [("host", 8, 5), ("host", 5, 14), ("device", 8, 14)])
def test_solve_on_nan_memory(LB, dtype, form, driven, m, iterations, behind):
    import synth
    prob = dict(synth.synth_problem(70, seed=3), kind="synth")
    opt = LB.default_option(dtype)
    opt.eps_f = opt.eps_g = opt.eps_x = 0.0
    opt.max_iteration, opt.hessian_approximate_dimension = iterations, m

    def solve():
        return LB.solve(prob, dtype, option=opt, objective="device", driven=driven, form=form, record=False)

    assert LB.load().lbfgsb_b200_trim_memory() == 0
    clean = solve()
    assert LB.load().lbfgsb_b200_trim_memory() == 0
    # the segment's solve ends at its start point; the pool holds nothing else then
    words = behind * np.dtype(dtype).itemsize // 4 * 5120  # 70^2 in whole tiles
    _batch(LB, [int(words ** 0.5)], 1e30, [0], vectors=1)
    got = solve()
    assert (clean.info, clean.num_iteration) == (got.info, got.num_iteration)
    assert clean.residual_g == got.residual_g and clean.residual_x == got.residual_x
    np.testing.assert_array_equal(clean.x, got.x)


def test_batch_on_nan_history(LB):
    sides = [17, 40, 64]
    clean = _batch(LB, sides, 0.0, [])
    got = _batch(LB, sides, 0.0, [0, 1, 2])
    for a, b in zip(clean, got):
        np.testing.assert_array_equal(a, b)
