"""Runs of gates that sweep the tile (Toffolis, phases, dense pairs) with rotations, X and CNOTs between them, so that
some sweeps find the addresses of the one before and some do not: energies and gradients against an FP64 sweep."""
import numpy as np
import pytest

import test_gpu_adjoint_passes as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,between", [(3, 4), (5, 2), (8, 3), (12, 5), (13, 3), (15, 6)])
def test_runs_of_sweeps(n, between):
    import torch
    from qsim_b200 import workloads as W
    from qsim_b200.autograd import expectation
    from qsim_b200.circuit import Circuit, lower

    rng = np.random.default_rng(n)
    gates = [("ry", [q], None, q) for q in range(n)]
    for k in range(60):
        q = [int(x) for x in rng.permutation(n)]
        kind = str(rng.choice(["mcx", "cz", "cp", "u2"]))
        if kind == "mcx":
            gates.append((kind, q[:3], None, -1))
        elif kind == "u2":
            gates.append((kind, q[:2], np.linalg.qr(rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4)))[0], -1))
        else:
            gates.append((kind, q[:2], float(rng.uniform(0, 6)), -1))
        if k % between == 0:
            gates.append([("cx", q[1:3], None, -1), ("x", q[:1], None, -1), ("rx", q[:1], None, k % n),
                          ("cx", [n - 1, 0], None, -1)][k // between % 4])
    gates.append(("rz", [0], None, 0))
    gates.append(("rx", [n - 1], None, 1))
    qc = Circuit(n)
    for kind, q, m, p in gates:
        if kind in P._G:
            getattr(qc, kind)(0.0, q[0], param_index=p)
        elif kind == "u2":
            qc.unitary(m, q)
        elif kind in ("x", "cx", "mcx"):
            qc.mcx(q[:-1], q[-1])
        else:
            qc.cz(*q) if kind == "cz" else qc.cp(m, *q)
    obs = W.random_pauli_observable(n, 10, seed=n, wmax=min(4, n))
    theta = rng.uniform(0, 2 * np.pi, (2, n))
    th = torch.tensor(theta, requires_grad=True)
    energy = expectation(th, n, lower(qc), obs)
    energy.sum().backward()

    j = np.arange(1 << n, dtype=np.uint64)
    # as the other passes: a gate rounds an amplitude to at most 8 u of its pair, twice that for each of two states
    tol = 4 * 8 * len(gates) * 2.0 ** -24 * float(np.abs(obs.coefs).sum())
    for b in range(2):
        psi = np.zeros(1 << n, complex)
        psi[0] = 1
        for g in gates:
            psi = P._step(psi, n, g, theta[b], False)
        lam = np.zeros_like(psi)
        for x, z, c in zip(obs.x, obs.z, obs.coefs.real):
            src = j ^ x
            sign = 1.0 - 2.0 * (np.bitwise_count(src & z) & 1)
            lam += c * 1j ** (bin(int(x & z)).count("1") % 4) * sign * psi[src.astype(np.int64)]
        assert abs(float(energy[b].detach()) - np.vdot(psi, lam).real) <= tol
        grad = np.zeros(n)
        for g in reversed(gates):
            if g[3] >= 0:
                grad[g[3]] += np.vdot(lam, P._apply(psi, g[1][0], P._G[g[0]])).imag
            psi, lam = P._step(psi, n, g, theta[b], True), P._step(lam, n, g, theta[b], True)
        assert np.abs(th.grad[b].numpy() - grad).max() <= tol
