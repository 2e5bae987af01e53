"""Gates in front of few channels: long runs of permutations and diagonals stay register blocks of a unitary segment
(no map without a channel), with the FP64 trajectory's state and branches."""
import numpy as np
import pytest

import plan_emulator as PE
import sv_oracle as O
from qsim_b200.circuit import Circuit, lower

KINDS = ["cp", "cx", "cx+rz", "swap+ccz"]


def _circuit(n, gates, kind, noisy=True):
    rng = np.random.default_rng(n + gates)
    qc = Circuit(n)
    for q in range(n):
        qc.h(q)
    for _ in range(gates):
        a, b, c = (int(x) for x in rng.permutation(n)[:3])
        if kind == "cp":
            qc.cp(float(rng.uniform(0, 6)), a, b)
        elif kind == "swap+ccz":
            qc.swap(a, b)
            qc.ccz(a, b, c)
        else:
            qc.cx(a, b)
            if kind == "cx+rz":
                qc.rz(float(rng.uniform(0, 6)), b)
    for q in range(n if noisy else 0):
        qc.amplitude_damp(0.1, q)
    return qc


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,gates", [(5, 40), (12, 30), (12, 300)])
def test_no_map_without_a_channel(kind, n, gates):
    blocks = maps = free = 0
    for _, recs, _, _ in PE.decode(PE.noise_program(n, lower(_circuit(n, gates, kind)))):
        b = 0
        while b < len(recs):
            behind = int(recs[b]["pos"][4]) if recs[b]["pos"][6] else 0
            if recs[b]["pos"][6]:
                inner = recs[b + 1: b + 1 + behind] if behind else recs[b: b + 1]
                maps += 1
                free += not any(r["pos"][6] and r["op_end"] > r["op_begin"] for r in inner)
            else:
                blocks += 1
            b += 1 + behind
    plain = PE.decode(PE.program(n, lower(_circuit(n, gates, kind, noisy=False)), tile_bits=13, block_bits=4))
    # channels on every qubit, four qubits to a map
    assert free == 0 and maps <= (n + 3) // 4 + 1
    assert blocks <= sum(len(recs) for _, recs, _, _ in plain) + 1


@pytest.mark.parametrize("kind", KINDS)
def test_states(kind):
    n = 6
    ops = lower(_circuit(n, 40, kind))
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
        assert np.abs(got - ref).max() <= 2e-5   # coefficients rounded to FP32, as the chain tests
