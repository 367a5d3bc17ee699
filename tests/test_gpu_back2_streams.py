"""A 2D plan's back-projection of stacks on several streams, and in CUDA graphs (sgb_fbp_backproject on device
pointers keeps nothing of a call in the plan).  Slices go in fours through a workspace; results must be those of one
call at a time, in every bit."""
import numpy as np
import pytest

import sinograms as S
from sinograms import learned

pytestmark = pytest.mark.gpu


def _plan():
    rg = S.SinoFanFlat(nb=256, d=1.0, na=240, orbit=360.0, orbit_start=11.0, dsd=600.0, dod=200.0)
    plan = S.plan_fbp(rg, S.ImageGeom((160, 128), (0.7, 0.7)))
    plan.set_back_form("fours")
    return plan


def _rows(torch, slices, seed):
    return torch.as_tensor(np.random.default_rng(seed).standard_normal((slices, 240, 256)).cumsum(2).astype(np.float32),
                           device="cuda")


def test_two_streams(cuda):
    import torch
    plan = _plan()
    assert plan.back_form(8)["slices"] == 4
    a, b = _rows(torch, 8, 1), _rows(torch, 12, 2)
    ref_a, ref_b = learned.fbp_backproject(plan, a), learned.fbp_backproject(plan, b)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    out = []
    for _ in range(20):
        for st, x in zip(streams, (a, b)):
            with torch.cuda.stream(st):
                out.append(learned.fbp_backproject(plan, x, sync=False))
    torch.cuda.synchronize()
    for i, y in enumerate(out):
        assert torch.equal(y, ref_b if i % 2 else ref_a), i


def test_threads(cuda):
    import threading

    import torch
    plan = _plan()
    xs = [_rows(torch, 4 + 4 * i, 10 + i) for i in range(4)]
    torch.cuda.synchronize()
    refs = [learned.fbp_backproject(plan, x) for x in xs]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(10):
                y = learned.fbp_backproject(plan, xs[i])
                torch.cuda.current_stream().synchronize()
                if not torch.equal(y, refs[i]):
                    bad.append(i)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


def test_graph_replayed_after_larger_stacks(cuda):
    import torch
    plan = _plan()
    a, b = _rows(torch, 8, 3), _rows(torch, 24, 4)
    eager = learned.fbp_backproject(plan, a)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        learned.fbp_backproject(plan, a, sync=False)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        out = learned.fbp_backproject(plan, a, sync=False)
    ref_b = learned.fbp_backproject(plan, b)
    fill = torch.full((64 << 20,), float("nan"), device="cuda")  # what a freed block would be given to
    graph.replay()
    torch.cuda.synchronize()
    first = out.clone()
    # slices go one by one in a graph: another order of the same taps, to the bar of every FP32 test
    assert float((first - eager).norm() / eager.norm()) < 1e-5
    out.zero_()
    side = torch.cuda.Stream()
    for _ in range(5):  # the graph beside eager calls on another stream
        graph.replay()
        with torch.cuda.stream(side):
            y = learned.fbp_backproject(plan, b, sync=False)
    torch.cuda.synchronize()
    assert torch.equal(out, first) and torch.equal(y, ref_b)
    del fill
