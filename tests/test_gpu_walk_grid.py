"""A device-driven round launches the cooperative walk whether one is due or not.  Its grid must
leave SMs to other solves (half of them): a grid that needs every SM at once makes solves on
several threads wait for one another.  Several threads' solves must give what each gives alone."""
import json
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _need_gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _option(LB):
    opt = LB.default_option(np.float64)
    opt.eps_f = opt.eps_g = opt.eps_x = 0.0
    opt.max_iteration = 6
    return opt


def _solve(LB, prob):
    return LB.solve(prob, np.float64, option=_option(LB), objective="device", driven="device", record=False)


def _prob(k):
    import synth
    p = dict(synth.synth_problem(40 + 3 * k, seed=k), kind="synth")
    if k % 2:  # tight bounds: the first steps walk
        p["l"], p["u"] = p["l"] * 5e-5, p["u"] * 5e-5
    return p


def test_walk_grid_leaves_sms(tmp_path):
    torch = _need_gpu()
    import lbfgsb_b200 as LB
    from torch.profiler import ProfilerActivity, profile
    _solve(LB, _prob(0))
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        _solve(LB, _prob(0))
        torch.cuda.synchronize()
    p.export_chrome_trace(str(tmp_path / "trace.json"))
    with open(tmp_path / "trace.json") as f:
        events = json.load(f)["traceEvents"]
    kernels = [e for e in events if e.get("cat") == "kernel"]
    if not kernels:
        pytest.skip("no kernel records from the profiler")
    grids = {e["args"]["grid"][0] for e in kernels if "k_walk_coop" in e["name"]}
    assert grids and max(grids) <= torch.cuda.get_device_properties(0).multi_processor_count // 2, grids


def test_threads_solve_as_alone():
    _need_gpu()
    import lbfgsb_b200 as LB
    probs = [_prob(k) for k in range(6)]
    alone = [_solve(LB, p) for p in probs]
    got = [None] * len(probs)

    def work(k):
        got[k] = _solve(LB, probs[k])

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(probs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, got):
        assert (a.info, a.num_iteration) == (b.info, b.num_iteration)
        np.testing.assert_array_equal(a.x, b.x)
