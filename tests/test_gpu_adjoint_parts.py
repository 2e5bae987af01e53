"""Gradients whose partial sums do not fit at once (1.5 GiB): the reverse passes run in parts, or are cut where one alone
has too many sums; the same gradients as in batches that fit, and no launch per gate."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gradient(n, ops, npar, theta, ps):
    from qsim_b200 import engine as E

    before = E.launch_count()
    e, g = E.adjoint_gradient(n, ops, npar, theta, ps)
    return e, g, E.launch_count() - before


# 4096 tiles; runs of one rotation are three sums of 8 bytes per vector and tile
@pytest.mark.parametrize("shared", [False, True])
def test_many_tiles(shared):
    from qsim_b200.circuit import Circuit, lower
    from qsim_b200.paulis import PauliSum

    n, layers, nb = 24, 90, 8                      # 2160 runs x 3 x 8 bytes x 8 x 4096 = 1.6 GiB
    qc = Circuit(n)
    for k in range(layers):
        for q in range(n):
            qc.ry(0.0, q, param_index=k % 7 if shared else k * n + q)
        for q in range(k % 2, n - 1, 2):
            qc.cx(q, q + 1)
    ops, npar = lower(qc), 7 if shared else n * layers
    theta = np.random.default_rng(1).uniform(0, 6, (nb, npar))
    ps = PauliSum([0, 3, 1 << 20], [1, 0, 5], [1.0, 0.5, -0.25], n)
    e, g, launches = _gradient(n, ops, npar, theta, ps)
    assert launches < len(ops) // 4
    for b in (0, nb - 1):
        e1, g1, _ = _gradient(n, ops, npar, theta[b: b + 1], ps)
        # the same FP64 sums; a shared parameter's are added in two parts
        assert abs(e[b] - e1[0]) <= 1e-12 and np.abs(g[b] - g1[0]).max() <= 1e-12


def test_one_pass_of_too_many_sums():
    from qsim_b200.circuit import Circuit, lower
    from qsim_b200.paulis import PauliSum

    n, layers, nb = 12, 90, 60000                  # one tile: 1080 runs x 3 x 8 bytes x 60000 = 1.45 GiB; limit 1118 gates
    qc = Circuit(n)
    for k in range(layers):
        for q in range(n):
            qc.rx(0.0, q, param_index=(k + q) % 5)
            if q % 3 == 0:
                qc.rz(0.0, q, param_index=q % 5)
        qc.cx(k % n, (k + 5) % n)
    ops = lower(qc)
    theta = np.random.default_rng(2).uniform(0, 6, (nb, 5))
    ps = PauliSum([0, 3], [1, 4], [1.0, 0.5], n)
    e, g, launches = _gradient(n, ops, 5, theta, ps)
    assert launches < len(ops) // 4
    e1, g1, _ = _gradient(n, ops, 5, theta[-40:], ps)
    assert np.abs(e[-40:] - e1).max() <= 1e-5
    # the cut changes where gates are fused: FP32 states after some hundreds of blocks, gradients of sums of 1440 gates
    assert np.abs(g[-40:] - g1).max() <= 2e-3
