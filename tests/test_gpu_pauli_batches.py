"""H psi of many vectors at once (through the gradient of a batch): widths and counts around the choice between two and
eight amplitudes per thread, partly filled CTAs and the vectors' strides, against FP64."""
import numpy as np
import pytest

import sv_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nb", [(7, 2048), (8, 1024), (8, 1023), (9, 512), (10, 300), (11, 128), (11, 127), (12, 70),
                                  (16, 4), (17, 2), (1, 9), (3, 4000)])
def test_energies_and_gradients(n, nb):
    from qsim_b200 import engine as E
    from qsim_b200.circuit import Circuit, lower
    from qsim_b200.paulis import PauliSum

    rng = np.random.default_rng(100 * n + nb)
    qc = Circuit(n)
    for q in range(n):
        qc.ry(0.0, q, param_index=q % 4)
        qc.rz(0.0, q, param_index=(q + 1) % 4)
    for q in range(n - 1):
        qc.cx(q, q + 1)
    for q in range(n):
        qc.rx(0.0, q, param_index=3)
    ops = lower(qc)
    theta = rng.uniform(0, 6, (nb, 4))
    terms = 40
    xs, zs = (rng.integers(0, 1 << n, terms).astype(np.uint64) for _ in range(2))
    xs[:8] = 0
    cs = rng.standard_normal(terms)
    e, g = E.adjoint_gradient(n, ops, 4, theta, PauliSum(xs, zs, cs, n))

    def energy(th):
        bound = ops.copy()
        for r in bound:
            if r["param"] >= 0:
                r["m"][0] = th[r["param"]]
                r["param"] = -1
        psi = O.simulate(n, bound)
        idx = np.arange(1 << n, dtype=np.uint64)
        total = 0.0
        for x, z, c in zip(xs, zs, cs):
            j = idx ^ x
            sign = 1 - 2 * (np.bitwise_count(j & z) & 1).astype(np.int64)
            total += c * np.real(1j ** int(np.bitwise_count(x & z)) * np.vdot(psi, sign * psi[j]))
        return total

    h = 1e-4
    # FP32 states: tens of roundings of 2^-24 against coefficients whose absolute sum is `size`; the central
    # difference adds h^2 / 6 of a third derivative, which is at most (2 n)^3 / 8 of the energy's size
    size = np.abs(cs).sum()
    for b in sorted({0, 1 % nb, nb // 2, nb - 1}):
        assert abs(e[b] - energy(theta[b])) <= 3e-6 * size
        for p in (0, 3):
            d = np.zeros(4)
            d[p] = h
            want = (energy(theta[b] + d) - energy(theta[b] - d)) / (2 * h)
            assert abs(g[b, p] - want) <= (6e-6 * n + h * h * n ** 3 / 6) * size


def _kernel_time(n, nb, terms):
    import torch
    from torch.profiler import ProfilerActivity, profile
    from qsim_b200 import engine as E
    from qsim_b200 import workloads as W
    from qsim_b200.circuit import Circuit, lower

    qc = Circuit(n)
    qc.ry(0.0, 0, param_index=0)
    ops, theta, ps = lower(qc), np.zeros((nb, 1)), W.random_pauli_observable(n, terms, seed=1)
    E.adjoint_gradient(n, ops, 1, theta, ps)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        for _ in range(10):
            E.adjoint_gradient(n, ops, 1, theta, ps)
        torch.cuda.synchronize()
    return sum(e.device_time_total / e.count for e in prof.key_averages() if "pauli_apply" in e.key)


# As many amplitudes in many short vectors as in few long ones, and a little less of them than where a kernel of its
# own begins: the same work, which may not take twice the time.
@pytest.mark.parametrize("a,b,terms", [((8, 1024), (11, 128), 64), ((8, 1000), (8, 1100), 8), ((12, 63), (12, 70), 8)])
def test_time_follows_the_amplitudes(a, b, terms):
    assert _kernel_time(*a, terms) <= 1.6 * _kernel_time(*b, terms)
