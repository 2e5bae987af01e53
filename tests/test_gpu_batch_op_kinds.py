"""Batches whose circuits of one width differ in the op kinds of their passes (rotations and tables only, or a Toffoli
among them): one launch per level while the launches are small, and every state as the circuit alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ops(n, depth, seed, toffoli):
    from qsim_b200.circuit import Circuit, lower

    rng = np.random.default_rng(seed)
    qc = Circuit(n)
    for d in range(depth):
        for q in range(n):
            qc.ry(float(rng.uniform(0, 6)), q)
            qc.rz(float(rng.uniform(0, 6)), q)
        for q in range(d % 2, n - 1, 2):
            qc.cz(q, q + 1)
        if toffoli:
            qc.ccx(0, n // 2, n - 1)
    return lower(qc)


def _plan(widths, kinds, depth):
    from qsim_b200 import engine as E

    parts = [_ops(w, depth, 10 + i, k) for i, (w, k) in enumerate(zip(widths, kinds))]
    amps = np.int64(1) << np.array(widths, dtype=np.int64)
    plan = E.BatchPlan(np.array(widths, np.int32), np.cumsum([0] + [len(p) for p in parts]), np.concatenate(parts),
                       np.cumsum(amps) - amps)
    return plan, parts


@pytest.mark.parametrize("widths,kinds", [([12] * 8, [0, 1] * 4), ([10, 12, 12, 10, 12], [0, 0, 1, 1, 0]),
                                          ([16, 16, 16], [1, 0, 0]), ([13, 13, 17, 17, 9, 9], [0, 1, 1, 0, 0, 1]),
                                          ([25, 25], [0, 1])])
def test_states_and_launches(widths, kinds):
    import torch
    from qsim_b200 import engine as E

    plan, parts = _plan(widths, kinds, 4)
    levels = {}
    for i, w in enumerate(widths):
        levels[w] = max(levels.get(w, 0), _plan([w], [kinds[i]], 4)[0].info["n_launches"])
    if max(widths) < 20:
        assert plan.info["n_launches"] == sum(levels.values())
    states = plan.alloc_states()
    for _ in range(3):                       # direct, then replayed
        states.fill_(2.0)
        plan.execute(states)
        at = 0
        for w, ops in zip(widths, parts):
            want = E.Plan(w, ops).execute_from_zero(E.empty_state(w))
            assert torch.equal(torch.view_as_real(states[at: at + (1 << w)]), torch.view_as_real(want))
            at += 1 << w
