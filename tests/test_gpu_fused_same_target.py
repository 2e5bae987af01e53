"""apply_gates_fused with several device gates on one qubit: applied in their order, against FP64, and in no more time
than as many gates on different qubits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gates(rng, count):
    return np.linalg.qr(rng.standard_normal((count, 2, 2)) + 1j * rng.standard_normal((count, 2, 2)))[0].astype(np.complex64)


@pytest.mark.parametrize("n", [1, 4, 11, 12, 13, 17])
@pytest.mark.parametrize("pattern", ["one", "two", "rounds", "five"])
def test_order_on_a_qubit(n, pattern):
    import torch
    import blackwell_kernels as bk
    import sv_oracle as O
    from qsim_b200.circuit import Circuit, lower

    targets = {"one": [n - 1] * 25, "two": [0, n - 1] * 6, "rounds": [q % n for q in range(24)],
               "five": [(3 * q) % min(n, 5) for q in range(12)]}[pattern]
    rng = np.random.default_rng(n)
    gates = _gates(rng, len(targets))
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64)
    state = torch.from_numpy(psi).cuda()
    bk.apply_gates_fused(state, torch.from_numpy(gates).cuda(), torch.tensor(targets, dtype=torch.int32, device="cuda"))
    qc = Circuit(n)
    for g, t in zip(gates, targets):
        qc.unitary(g.astype(np.complex128), [t])
    ref = O.simulate(n, lower(qc), psi.astype(np.complex128))
    # four roundings per gate, each of at most u of the pair's norm
    assert np.linalg.norm(state.cpu().numpy() - ref) <= 4 * 2.0 ** -24 * len(targets) * 2


def test_time_of_gates_on_one_qubit():
    import torch
    import blackwell_kernels as bk
    from qsim_b200 import engine as E

    state = E.empty_state(16)
    state.zero_()
    gates = torch.from_numpy(_gates(np.random.default_rng(0), 12)).cuda()

    def time(targets):
        t = torch.tensor(targets, dtype=torch.int32, device="cuda")
        bk.apply_gates_fused(state, gates, t)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(50):
                bk.apply_gates_fused(state, gates, t)
        best = 1e9
        for _ in range(10):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        return best

    assert time([5] * 12) <= 1.3 * time(list(range(12)))
