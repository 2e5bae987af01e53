"""Passes of rotations and diagonals only (an op loop of their own) beside passes with other ops in one circuit, single
and batched, over register-block widths, against FP64 and bit for bit alone and in a batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _circuit(n, toffolis, rng):
    from qsim_b200.circuit import Circuit
    qc = Circuit(n)
    for layer in range(4):
        for q in range(n):
            qc.u(*(float(x) for x in rng.uniform(0, 6, 3)), q)
        for q in range(layer % 2, n - 1, 2):
            qc.cz(q, q + 1)
        qc.cp(float(rng.uniform(0, 6)), 0, n - 1)
        if toffolis and layer == 1:
            qc.ccx(*(int(x) for x in rng.permutation(n)[:3]))
    return qc


@pytest.mark.parametrize("n", [3, 5, 13, 14, 15, 17])
@pytest.mark.parametrize("block", [0, 2, 3, 5])
def test_rotation_passes(n, block):
    import torch
    import sv_oracle as O
    from qsim_b200 import engine as E
    from qsim_b200.circuit import lower

    rng = np.random.default_rng(n)
    ops = [lower(_circuit(n, t, rng)) for t in (False, True)]
    h = E._h(0)
    h.call("qs_set_block_bits", block)
    try:
        alone = [E.Plan(n, o).execute_from_zero(E.empty_state(n)) for o in ops]
        plan = E.BatchPlan(np.full(2, n), np.cumsum([0] + [len(o) for o in ops]), np.concatenate(ops),
                           np.arange(2, dtype=np.int64) << n)
        states = plan.execute(plan.alloc_states())
        torch.cuda.synchronize()
    finally:
        h.call("qs_set_block_bits", 0)
    for k, o in enumerate(ops):
        got = alone[k].cpu().numpy()
        assert np.array_equal(got, states[k << n: (k + 1) << n].cpu().numpy())
        # the repository's bound for planned circuits: FP32 chains against FP64
        ref = O.simulate(n, o)
        assert abs(1 - O.fidelity(got, ref)) <= 1e-6 and O.max_abs_err(got, ref) <= 1e-5
