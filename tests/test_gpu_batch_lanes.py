"""Batches of more widths than there are streams to spread them over: direct, replayed from a graph, captured by the
caller, on another stream, and with work queued before and after, each bit for bit as the circuits alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batch_widths_side_by_side():
    import torch
    from qsim_b200 import engine as E
    from qsim_b200 import workloads as W

    widths = np.array(list(range(2, 17)) + [15, 13, 2], dtype=np.int32)
    parts = [W.qv_ops(int(w), int(w), 50 + i) for i, w in enumerate(widths)]
    amps = np.int64(1) << widths.astype(np.int64)
    off = np.cumsum(amps) - amps
    want = []
    for w, ops in zip(widths, parts):
        want.append(E.Plan(int(w), ops).execute_from_zero(E.empty_state(int(w))))
    want = torch.cat(want)
    plan = E.BatchPlan(widths, np.cumsum([0] + [len(p) for p in parts]), np.concatenate(parts), off)
    states = plan.alloc_states()
    for _ in range(4):                       # direct, then captured and replayed
        states.fill_(3.0)
        plan.execute(states)
        got = states.clone()                 # queued behind the batch
        assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))
    side = torch.cuda.Stream()
    other = torch.empty_like(states)
    with torch.cuda.stream(side):
        other.fill_(5.0)
        plan.execute(other)
        got = other.clone()
    side.synchronize()
    assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.execute(states)
    for _ in range(2):
        states.zero_()
        graph.replay()
        assert torch.equal(torch.view_as_real(states), torch.view_as_real(want))
