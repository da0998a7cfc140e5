"""A wait that gives up in one instance of a batched solve fails the call; the instances before
it that had ended by then must have been delivered: status 0 only with x copied back.

The failure is the flag that the host reads after a wait's time limit, written by a memset node
beside the objective into the state of one instance (its place in the instance's segment is
worked out here as the library lays it out, and checked against the state's n and m)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDES, SEEDS = [40, 33, 36], [5, 6, 7]


def _state_offset(n, real=4, hist=4, slots=9):
    ld = (n + 511) // 512 * 512
    off = 0
    for size in [ld * real] * 7 + [ld * slots * hist] * 2 + [ld, (ld // 32 + 4) * 4]:
        off = (off + 255) // 256 * 256 + size
    return (off + 255) // 256 * 256


def _solve(mark=None):
    """Three solves of one iteration; mark: the instance whose device_error flag is set."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import lbfgsb_b200 as LB
    lib = LB.load()
    cuda = C.CDLL("libcuda.so.1")
    cuda.cuMemsetD32Async.argtypes = [C.c_void_p, C.c_uint, C.c_size_t, C.c_void_p]
    cuda.cuStreamSynchronize.argtypes = [C.c_void_p]
    bt = LB.SynthBatch(SIDES, SEEDS)
    objective = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_int,
                            *[C.c_void_p] * 5)
    inner = objective(bt.objective)
    calls = []

    def call(user, count, ids, first, ctas, x, g, f, active, stream):
        if mark is not None and not calls:  # at the start points: x is the segment's first buffer
            cuda.cuStreamSynchronize(stream)
            base = (C.c_void_p * count)()
            assert lib.lbfgsb_b200_copy(base, C.c_void_p(x), C.sizeof(base), 2) == 0
            n = SIDES[mark] ** 2
            st = base[mark] + _state_offset(n)
            head = (C.c_int * 26)()
            assert lib.lbfgsb_b200_copy(head, C.c_void_p(st), C.sizeof(head), 2) == 0
            assert (head[0], head[1], head[5], head[25]) == (n, 8, 1, 0)
            calls.append(st + 25 * 4)
        elif mark is not None:
            cuda.cuMemsetD32Async(calls[0], 1, 1, stream)
        return inner(user, count, ids, first, ctas, x, g, f, active, stream)

    keep = objective(call)
    bt.objective = C.cast(keep, C.c_void_p).value
    xs = [torch.full((s * s,), 0.25, dtype=torch.float32, device="cuda") for s in SIDES]
    opt = LB.default_option(np.float32)
    opt.eps_f = opt.eps_g = opt.eps_x = 0.0
    opt.max_iteration = 1
    rc, stat, _, _ = LB.solve_batch_device(bt, xs, opt)
    torch.cuda.synchronize()
    out = [x.cpu().numpy() for x in xs]
    bt.close()
    return rc, stat, out, mark is None or len(calls) == 1


@pytest.mark.parametrize("mark", [0, 1, 2])
def test_ended_instances_before_a_failure_are_delivered(mark):
    rc, stat, good, _ = _solve()
    assert rc == 0 and stat == [0, 0, 0]
    rc, stat, x, marked = _solve(mark)
    assert marked and rc != 0
    for k in range(3):
        if k < mark:
            assert stat[k] == 0
            np.testing.assert_array_equal(x[k], good[k])
        else:
            assert stat[k] != 0
            np.testing.assert_array_equal(x[k], np.float32(0.25))


def test_large_and_small_instances_come_back():
    """Instances on both sides of the size from which x is copied back on its own (2^21)."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import lbfgsb_b200 as LB
    sides = [1449, 40, 1448]  # 1448^2 < 2^21 < 1449^2
    opt = LB.default_option(np.float32)
    opt.eps_f = opt.eps_g = opt.eps_x = 0.0
    opt.max_iteration = 3

    def solve(ids):
        bt = LB.SynthBatch(sides, [3, 4, 5])
        xs = [torch.full((sides[p] ** 2,), 0.25, dtype=torch.float32, device="cuda") for p in ids]
        rc, stat, summ, _ = LB.solve_batch_device(bt, xs, opt, ids=ids)
        torch.cuda.synchronize()
        assert rc == 0 and stat == [0] * len(ids)
        bt.close()
        return xs, [(s.info, s.num_iteration, s.residual_g) for s in summ]

    mixed, summ = solve([0, 1, 2])
    for k in range(3):
        alone, s = solve([k])
        assert s[0] == summ[k] and not torch.equal(mixed[k], torch.full_like(mixed[k], 0.25))
        assert torch.equal(alone[0], mixed[k])
