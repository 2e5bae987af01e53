"""The tile passes of the adjoint gradient over widths and circuits that reach every kind of step, against an FP64 sweep."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(v, q):
    return v.reshape(-1, 2, 1 << q)


def _apply(v, q, u):
    p = _pairs(v, q)
    return np.stack([u[0, 0] * p[:, 0] + u[0, 1] * p[:, 1], u[1, 0] * p[:, 0] + u[1, 1] * p[:, 1]], 1).reshape(-1)


def _apply2(v, n, q0, q1, u):
    t = v.reshape((2,) * n)
    t = np.moveaxis(t, (n - 1 - q1, n - 1 - q0), (0, 1)).reshape(4, -1)
    t = (u @ t).reshape((2, 2) + (2,) * (n - 2))
    return np.moveaxis(t, (0, 1), (n - 1 - q1, n - 1 - q0)).reshape(-1)


_G = {"rx": np.array([[0, 1], [1, 0]], complex), "ry": np.array([[0, -1j], [1j, 0]]), "rz": np.diag([1.0 + 0j, -1.0])}


def _circuit(n, depth, rng):
    """(kind, qubits, matrix or phase, parameter): rotations in runs, CNOTs in both directions, Toffolis, phases, dense pairs."""
    out, npar = [], 0
    for _ in range(depth):
        q = [int(x) for x in rng.permutation(n)]
        kind = rng.choice(["rot", "rot", "rot", "u1", "cx", "cx", "x", "mcx", "cz", "cp", "u2"])
        if kind == "rot":
            out.append((str(rng.choice(["rx", "ry", "rz"])), q[:1], None, npar if rng.random() < 0.8 else -1))
            npar += out[-1][3] >= 0
        elif kind in ("u1", "u2"):
            k = 2 if kind == "u1" else 4
            if n < 2 and k == 4:
                continue
            m = np.linalg.qr(rng.standard_normal((k, k)) + 1j * rng.standard_normal((k, k)))[0]
            out.append((kind, q[: k // 2], m, -1))
        elif kind == "x":
            out.append((kind, q[:1], None, -1))
        elif kind == "mcx":
            if n >= 3:
                out.append((kind, q[: min(n, 4)], None, -1))
        elif n >= 2:
            out.append((kind, q[:2], float(rng.uniform(0, 6)), -1))
    out.append(("ry", [0], None, npar))
    return out, npar + 1


def _step(v, n, g, theta, inverse):
    kind, q, m, p = g
    if kind in _G:
        t = (theta[p] if p >= 0 else 0.7) * (-1 if inverse else 1)
        return _apply(v, q[0], np.cos(t / 2) * np.eye(2) - 1j * np.sin(t / 2) * _G[kind])
    if kind == "u1":
        return _apply(v, q[0], m.conj().T if inverse else m)
    if kind == "u2":
        return _apply2(v, n, q[0], q[1], m.conj().T if inverse else m)
    j = np.arange(1 << n)
    if kind in ("x", "cx", "mcx"):
        ctl = sum(1 << c for c in q[:-1])
        return v[np.where((j & ctl) == ctl, j ^ (1 << q[-1]), j)]
    mask = (1 << q[0]) | (1 << q[1])
    ph = -1 if kind == "cz" else np.exp(1j * m * (-1 if inverse else 1))
    return np.where((j & mask) == mask, ph * v, v)


@pytest.mark.parametrize("n,depth,batch,low", [(1, 6, 2, 1), (2, 12, 3, 1), (3, 20, 1, 1), (4, 30, 2, 1), (5, 40, 2, 1),
                                               (11, 60, 2, 1), (12, 120, 3, 1), (13, 80, 2, 0), (16, 90, 2, 0),
                                               (17, 60, 1, 1)])
def test_adjoint_passes_every_step_kind(n, depth, batch, low):
    import torch
    from qsim_b200 import workloads as W
    from qsim_b200.autograd import expectation
    from qsim_b200.circuit import Circuit, lower

    rng = np.random.default_rng(10 * n + depth)
    gates, npar = _circuit(n, depth, rng)
    if not low:      # many controls above the tile
        gates += [("cx", [c, t], None, -1) for c, t in zip(range(n - 1, 3, -1), list(range(n)) * 2) if c != t]
        gates += [("ry", [q], None, npar + q) for q in range(n)]
        npar += n
    qc = Circuit(n)
    for kind, q, m, p in gates:
        if kind in _G:
            getattr(qc, kind)(0.7, q[0], param_index=p)
        elif kind in ("u1", "u2"):
            qc.unitary(m, q)
        elif kind == "x":
            qc.mcx([], q[0])
        elif kind in ("cx", "mcx"):
            qc.mcx(q[:-1], q[-1])
        else:
            qc.cz(*q) if kind == "cz" else qc.cp(m, *q)
    obs = W.random_pauli_observable(n, 12, seed=n, wmax=min(4, n))
    theta = rng.uniform(0, 2 * np.pi, (batch, npar))
    th = torch.tensor(theta, requires_grad=True)
    energy = expectation(th, n, lower(qc), obs)
    energy.sum().backward()
    energy = energy.detach()

    j = np.arange(1 << n, dtype=np.uint64)
    size = float(np.abs(obs.coefs).sum())
    # FP32 states: a gate rounds an amplitude to at most 8 u of its pair, so
    # after g gates the states are off by 8 g u, and an energy or gradient
    # (bounded by sum |c|) by twice that for each of the two states
    tol = 4 * 8 * len(gates) * 2.0 ** -24 * size
    for b in range(batch):
        psi = np.zeros(1 << n, complex)
        psi[0] = 1
        for g in gates:
            psi = _step(psi, n, g, theta[b], False)
        lam = np.zeros_like(psi)
        for x, z, c in zip(obs.x, obs.z, obs.coefs.real):
            src = j ^ x
            sign = 1.0 - 2.0 * (np.bitwise_count(src & z) & 1)
            lam += c * 1j ** (bin(int(x & z)).count("1") % 4) * sign * psi[src.astype(np.int64)]
        assert abs(float(energy[b]) - np.vdot(psi, lam).real) <= tol
        grad = np.zeros(npar)
        for g in reversed(gates):
            if g[3] >= 0:
                grad[g[3]] += np.vdot(lam, _apply(psi, g[1][0], _G[g[0]])).imag
            psi, lam = _step(psi, n, g, theta[b], True), _step(lam, n, g, theta[b], True)
        assert np.abs(th.grad[b].numpy() - grad).max() <= tol
