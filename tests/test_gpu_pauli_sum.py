"""Pauli-sum expectation values and products over the widths where the kernels change their amplitudes per thread, and
over tables of every kind of term, against FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sum(n, m, rng):
    lim = 1 << n
    x = rng.integers(0, lim, m)
    x[: m // 3] = 1 << rng.integers(0, n, m // 3)          # one flipped qubit, masks shared
    x[m // 3: m // 2] = x[: m // 2 - m // 3]
    x[-(m // 8 + 1):] = 0
    z = rng.integers(0, lim, m)
    z[:: 3] &= ~np.int64(0xC1)                             # no sign inside a thread's amplitudes
    return x, z, rng.standard_normal(m)


@pytest.mark.parametrize("n,m", [(1, 3), (2, 9), (5, 1), (6, 20), (7, 40), (8, 300), (12, 1024), (17, 40), (18, 30),
                                 (19, 30), (20, 24), (21, 12)])
def test_pauli_sum_expectation_and_product(n, m):
    import torch
    from qsim_b200 import engine as E
    from qsim_b200.paulis import PauliSum

    rng = np.random.default_rng(n)
    x, z, c = _sum(n, m, rng)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64)
    state = torch.from_numpy(psi).cuda()
    ps = PauliSum(x, z, c, n)
    energy = E.expect_pauli_sum(state, ps)
    prod = E.apply_pauli_sum(state, ps).cpu().numpy()
    assert np.array_equal(state.cpu().numpy(), psi)

    p = psi.astype(np.complex128)
    j = np.arange(1 << n, dtype=np.uint64)
    want = np.zeros(1 << n, dtype=np.complex128)
    for xm, zm, cf in zip(x, z, c):
        src = j ^ np.uint64(xm)
        sign = 1.0 - 2.0 * (np.bitwise_count(src & np.uint64(zm)) & 1)
        want += cf * 1j ** (bin(int(xm) & int(zm)).count("1") % 4) * sign * p[src.astype(np.int64)]
    size = float(np.abs(c).sum())
    # FP64 sums: (m + 60) roundings of terms that add up to sum |c|; the product is then rounded to FP32 once
    assert abs(energy - np.vdot(p, want).real) <= (m + 60) * 2.0 ** -53 * size
    assert np.all(np.abs(prod - want) <= 2.0 ** -24 * np.abs(want) + (m + 4) * 2.0 ** -53 * size * np.abs(p).max() + 1e-45)
