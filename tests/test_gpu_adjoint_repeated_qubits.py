"""Ops of the C entry that list a qubit twice: controls and phase qubits count once, an X on one of its own controls
never acts, and energies and gradients are those of the op without the repetition."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 12, 14])
def test_repeated_qubits(n):
    from qsim_b200 import engine as E
    from qsim_b200._lib import OP_MCPHASE, OP_MCX
    from qsim_b200.circuit import Circuit, lower
    from qsim_b200.paulis import PauliSum

    def layers(entangle):
        parts = []
        for k in range(3):
            qc = Circuit(n)
            for q in range(n):
                qc.ry(0.0, q, param_index=(k * n + q) % 7)
                qc.rz(0.0, q, param_index=(k + q) % 7)
            parts += [lower(qc), entangle()]
        return np.concatenate(parts)

    def ops(kind, *lists):
        qc = Circuit(n)
        for _ in lists:
            qc.x(0)
        out = lower(qc)
        for r, qs in zip(out, lists):
            r["kind"], r["nq"] = kind, len(qs)
            r["q"][:] = list(qs) + [0] * (8 - len(qs))
            r["m"][:] = 0.0
            if kind == OP_MCPHASE:
                r["m"][0], r["m"][1] = np.cos(0.7), np.sin(0.7)
        return out

    top = n - 1
    twice = layers(lambda: np.concatenate([ops(OP_MCX, (0, 0, top), (top, top, 1), (1, 1), (top, 0, 0), (top, top)),
                                           ops(OP_MCPHASE, (1, 1), (top, 0, top), (0, 0, 0))]))
    once = layers(lambda: np.concatenate([ops(OP_MCX, (0, top), (top, 1)), ops(OP_MCPHASE, (1,), (top, 0), (0,))]))
    rng = np.random.default_rng(n)
    theta = rng.uniform(0, 6, (2, 7))
    ps = PauliSum([0, 3, 1 << top], [1, 1, 5], [0.5, -0.25, 1.0], n)
    (e0, g0), (e1, g1) = (E.adjoint_gradient(n, o, 7, theta, ps) for o in (once, twice))
    # FP32 states: each of a few hundred roundings of 2^-24 per unit norm, on gradients of order one
    assert np.abs(e0 - e1).max() <= 1e-5 and np.abs(g0 - g1).max() <= 3e-5
    assert np.abs(g0).max() > 1e-2
