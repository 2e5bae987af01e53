"""Matrix-free Chebyshev evolution over the widths where the kernel changes its
amplitudes per thread and thread groups, against a Taylor series in FP64."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _h_times(n, x, z, c, psi):
    j = np.arange(1 << n, dtype=np.uint64)
    out = np.zeros_like(psi)
    for xm, zm, cf in zip(x, z, c):
        src = j ^ np.uint64(xm)
        sign = 1.0 - 2.0 * (np.bitwise_count(src & np.uint64(zm)) & 1)
        out += cf * 1j ** (bin(int(xm) & int(zm)).count("1") % 4) * sign * psi[src.astype(np.int64)]
    return out


@pytest.mark.parametrize("n", [1, 2, 5, 6, 7, 12, 15, 16, 18, 19])
@pytest.mark.parametrize("diagonal", [False, True])
def test_pauli_evolution_widths(n, diagonal):
    import torch
    from blackwell_backend.chebyshev import chebyshev_coefficients, chebyshev_evolve_pauli
    from qsim_b200.paulis import PauliSum

    rng = np.random.default_rng(100 + n)
    m, lim = 22, 1 << n
    x = rng.integers(0, lim, m)
    x[: m // 2] = 1 << rng.integers(0, n, m // 2)        # single flips, repeated masks among them
    x[m // 2: m // 2 + 4] = x[:4]                         # shared masks: pairs of real and imaginary weights
    z = rng.integers(0, lim, m)
    if not diagonal:
        x[x == 0] = 1
    else:
        x[-3:] = 0
    ps = PauliSum(x, z, rng.uniform(-1, 1, m), n)
    t = 0.3
    psi = rng.standard_normal(lim) + 1j * rng.standard_normal(lim)
    psi = (psi / np.linalg.norm(psi)).astype(np.complex64)
    got, _ = chebyshev_evolve_pauli(torch.from_numpy(psi).cuda(), ps, t, precision=1e-8)

    term = psi.astype(np.complex128)
    want = term.copy()
    for k in range(1, 60):
        term = _h_times(n, x, z, ps.coefs.real, term) * (-1j * t / k)
        want += term
        if np.linalg.norm(term) < 1e-13:
            break
    # a degree's row sum of m weighted amplitudes rounds to (m + 3) u of
    # sum |c| / bound = 1, doubled by the recurrence, which carries an error on
    # at most linearly in the degree; the series is cut at 1e-8
    coeffs, _, _ = chebyshev_coefficients(t, ps.spectral_bound(), 1e-8)
    tol = 2 * (m + 3) * 2.0 ** -24 * float(np.sum(np.arange(len(coeffs)) * np.abs(coeffs)) + 1) + 1e-7
    assert math.isfinite(tol) and np.linalg.norm(got.cpu().numpy() - want) < tol
