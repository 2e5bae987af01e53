"""Chains of channels with the permutations and diagonals between them (one map in the kernel), every kind of gate on
and off the chain's qubits, against the channel-by-channel FP64 trajectory: the program on the host, and the kernel."""
import numpy as np
import pytest

import plan_emulator as PE
import sv_oracle as O
from qsim_b200.circuit import Circuit, lower


def _circuit(n, length, seed):
    rng = np.random.default_rng(seed)
    qc = Circuit(n)
    for q in range(n):
        qc.ry(float(rng.uniform(0, 3)), q)
    for _ in range(length):
        q = [int(x) for x in rng.permutation(n)]
        kind = rng.choice(["x", "y", "cx", "ccx", "mcx", "cz", "cp", "ccz", "rz", "t", "rzz", "swap", "cswap", "crz", "h",
                           "rxx"])
        if kind in ("x", "y", "t", "h"):
            getattr(qc, kind)(q[0])
        elif kind == "rz":
            qc.rz(float(rng.uniform(0, 6)), q[0])
        elif kind in ("cp", "rzz", "crz", "rxx") and n >= 2:
            getattr(qc, kind)(float(rng.uniform(0, 6)), *q[:2])
        elif kind in ("cx", "cz", "swap") and n >= 2:
            getattr(qc, kind)(*q[:2])
        elif kind in ("ccx", "ccz", "cswap") and n >= 3:
            getattr(qc, kind)(*q[:3])
        elif kind == "mcx" and n >= 5:
            qc.mcx(q[:4], q[4])
        for c in rng.permutation(3)[: int(rng.integers(0, 4))]:
            getattr(qc, ("depolarize", "amplitude_damp", "dephase")[c])(float(rng.uniform(0.02, 0.4)), q[int(rng.integers(0, min(n, 3)))])
    return lower(qc), qc


CASES = [(1, 30), (2, 40), (3, 60), (4, 80), (5, 80), (8, 90), (12, 60)]


@pytest.mark.parametrize("n,length", CASES)
def test_program(n, length):
    ops, _ = _circuit(n, length, 7 * n)
    blob = PE.noise_program(n, ops)
    psi0 = np.zeros(1 << n, complex)
    psi0[0] = 1
    for seed in range(6):
        br = []
        got = PE.run(n, blob, psi0, seed=seed, branches=br)
        ref, ref_br, margin = O.noise_trajectory(n, ops, seed)
        if margin < 1e-6:
            continue
        assert [b for _, b in sorted(br)] == list(ref_br)
        assert np.abs(got - ref).max() <= 2e-5


@pytest.mark.gpu
@pytest.mark.parametrize("n,length", CASES + [(14, 40)])
def test_kernel(n, length):
    from qsim_b200.noise import run_trajectories

    ops, qc = _circuit(n, length, 7 * n)
    states, branches = run_trajectories(qc, 12, seed=0)
    states = states.cpu().numpy()
    for seed in range(12):
        ref, ref_br, margin = O.noise_trajectory(n, ops, seed)
        if margin < 1e-6:
            continue
        assert np.array_equal(branches[seed], ref_br)
        # FP32 amplitudes of norm 1 after at most a few hundred blocks and maps of a few roundings each
        assert np.abs(states[seed] - ref).max() <= 2e-5
