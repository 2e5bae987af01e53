"""apply_gates_fused with device tensors where the tile kernel begins, over target sets with and without qubit 0 and a
single and many tiles per CTA, against FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,targets", [
    (11, [0, 3, 10, 3]), (12, [11]), (12, list(range(12))), (13, list(range(1, 13))), (13, [0, 0, 0, 12, 0]),
    (16, [15, 1, 14, 2, 13, 3, 12, 4, 11, 5, 10, 6]), (20, list(range(8, 20))), (20, [19, 0, 19, 7, 0, 7, 7, 3]),
    (22, [21, 20, 5, 4, 21, 13, 2, 1]), (23, list(range(11, 23)) + [0, 22, 5]),
])
def test_fused_tiles(n, targets):
    import torch
    import blackwell_kernels as bk
    import sv_oracle as O
    from qsim_b200.circuit import Circuit, lower

    rng = np.random.default_rng(n + len(targets))
    gates = np.linalg.qr(rng.standard_normal((len(targets), 2, 2)) + 1j * rng.standard_normal((len(targets), 2, 2)))[0]
    gates = gates.astype(np.complex64)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64)
    state = torch.from_numpy(psi).cuda()
    bk.apply_gates_fused(state, torch.from_numpy(gates).cuda(), torch.tensor(targets, dtype=torch.int32, device="cuda"))
    qc = Circuit(n)
    for g, t in zip(gates, targets):
        qc.unitary(g.astype(np.complex128), [t])
    ref = O.simulate(n, lower(qc), psi.astype(np.complex128))
    # a gate's FMA chain rounds four times: at most 4 u of the pair's norm per gate
    assert np.linalg.norm(state.cpu().numpy() - ref) <= 4 * 2.0 ** -24 * len(targets) * 2
