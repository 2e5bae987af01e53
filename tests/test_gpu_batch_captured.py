"""A batch that the caller captures: the widths are branches of the caller's graph as they are of the plan's own, between
the work captured before and after them, and each replay leaves the states of the circuits alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _longest_chain(graph):
    """(kernel nodes on the longest path, kernel nodes) of a captured graph."""
    from cuda.bindings import runtime as rt

    g = rt.cudaGraph_t(init_value=graph.raw_cuda_graph())
    err, _, count = rt.cudaGraphGetNodes(g)
    err, nodes, count = rt.cudaGraphGetNodes(g, count)
    assert int(err) == 0
    kernel = {int(n): rt.cudaGraphNodeGetType(n)[1] == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel
              for n in nodes[:count]}
    out = rt.cudaGraphGetEdges(g)
    out = rt.cudaGraphGetEdges(g, out[-1])
    assert int(out[0]) == 0
    after = {n: [] for n in kernel}
    for a, b in zip(out[1][: out[-1]], out[2][: out[-1]]):
        after[int(a)].append(int(b))
    depth = {}

    def walk(n):
        if n not in depth:
            depth[n] = kernel[n] + max((walk(m) for m in after[n]), default=0)
        return depth[n]

    return max(walk(n) for n in kernel), sum(kernel.values())


def test_captured_widths_are_branches():
    import torch
    from qsim_b200 import engine as E
    from qsim_b200 import workloads as W

    widths = np.array([15, 16, 17, 18, 15, 9, 17], dtype=np.int32)
    parts = [W.qv_ops(int(w), int(w), 90 + i) for i, w in enumerate(widths)]
    amps = np.int64(1) << widths.astype(np.int64)
    off = np.cumsum(amps) - amps
    want = torch.cat([E.Plan(int(w), ops).execute_from_zero(E.empty_state(int(w))) for w, ops in zip(widths, parts)])

    def plan_of(sel):
        a = np.int64(1) << widths[sel].astype(np.int64)
        return E.BatchPlan(widths[sel], np.cumsum([0] + [len(parts[i]) for i in sel]),
                           np.concatenate([parts[i] for i in sel]), np.cumsum(a) - a)

    plan = plan_of(list(range(len(widths))))
    longest = max(plan_of([i for i, v in enumerate(widths) if v == w]).info["n_launches"] for w in set(widths.tolist()))
    states, copy = plan.alloc_states(), plan.alloc_states()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        states.fill_(7.0)                 # in front of every branch
        plan.execute(states)
        copy.copy_(states)                # behind every branch
    depth, kernels = _longest_chain(graph)
    assert kernels >= plan.info["n_launches"]
    assert depth <= longest + 2           # the fill and the copy, where they are kernels
    graph.instantiate()
    for _ in range(3):
        copy.zero_()
        graph.replay()
        assert torch.equal(torch.view_as_real(copy), torch.view_as_real(want))
    plan.execute(states)                  # uncaptured, on the same streams and events
    assert torch.equal(torch.view_as_real(states), torch.view_as_real(want))
