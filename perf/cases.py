"""Workloads for timing the simulator through its public entry points.

Each case is a dict of plain values whose "kind" names one way the library is
used; `prepare` makes what a caller holds before the call (inputs from the
seed, a plan, a Hamiltonian, a simulator), `run` is one pass, `exact` the same
outputs in 64 bits with plain torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "qiskit-blackwell_b200", "python"))

DEV = "cuda:0"


def listed():
    return [
        # A program that applies gates one call at a time to a small state, as
        # scripts written against the kernel API do: launches and call overhead.
        {"name": "gates_10q", "kind": "gates", "n": 10, "gates": 24},
        # The same program on a state larger than L2: each call is one sweep of HBM.
        {"name": "gates_24q", "kind": "gates", "n": 24, "gates": 24},
        # One Quantum-Volume circuit through the simulator, statevector on the
        # host: the latency of a small job.
        {"name": "circuit_qv_12q", "kind": "circuit", "family": "qv", "n": 12, "depth": 12, "host": True},
        # Rotations, CZ brickwork and Toffolis at a width where the state still
        # fits L2, result kept on the device.
        {"name": "circuit_layers_22q", "kind": "circuit", "family": "layers", "n": 22, "depth": 20, "host": False},
        # A large one-off circuit from a plan: run before a specialised kernel
        # would pay for its compile.
        {"name": "plan_layers_28q", "kind": "plan", "n": 28, "depth": 20},
        # Many Quantum-Volume circuits of mixed widths, one plan run repeatedly.
        {"name": "batch_qv_256", "kind": "batch", "circuits": 256, "lo": 10, "hi": 16},
        # Variational steps: energy and full gradient of an EfficientSU2 ansatz,
        # small (latency) and at 20 qubits with 256 terms.
        {"name": "gradient_12q", "kind": "gradient", "n": 12, "batch": 16, "terms": 64},
        {"name": "gradient_20q", "kind": "gradient", "n": 20, "batch": 8, "terms": 256},
        # Time evolution with a CSR Hamiltonian larger than L2, and matrix-free
        # at the largest width of the evolution requests.
        {"name": "evolve_csr_20q", "kind": "csr", "n": 20, "t": 2.0},
        {"name": "evolve_pauli_22q", "kind": "pauli", "n": 22, "t": 10.0},
        # Noise trajectories of a brickwork circuit with three channels after
        # every gate.
        {"name": "noise_12q", "kind": "noise", "n": 12, "depth": 8, "trajectories": 1024},
        # Reading a resident state out: shots, an observable, all probabilities.
        {"name": "readout_24q", "kind": "readout", "n": 24, "shots": 1024, "terms": 64},
    ]


def draw(rng):
    kind = rng.choice(["gates", "circuit", "plan", "batch", "gradient", "csr", "pauli", "noise", "readout"])
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    if kind == "gates":
        return {"kind": kind, "n": rng.randint(4, 24), "gates": rng.randint(12, 48)}
    if kind == "circuit":
        family = rng.choice(["qv", "layers", "qft"])
        n = rng.randint(4, 22)
        depth = {"qv": min(n, 18), "layers": rng.randint(1, 20), "qft": 1}[family]
        return {"kind": kind, "family": family, "n": n, "depth": depth, "host": n <= 16 and rng.random() < 0.5}
    if kind == "plan":
        return {"kind": kind, "n": rng.randint(24, 27), "depth": rng.randint(3, 20)}
    if kind == "batch":
        lo = rng.randint(4, 10)
        return {"kind": kind, "circuits": log(8, 256), "lo": lo, "hi": rng.randint(lo, 16)}
    if kind == "gradient":
        return {"kind": kind, "n": rng.randint(6, 20), "batch": rng.randint(1, 8), "terms": log(8, 256)}
    if kind == "csr":
        return {"kind": kind, "n": rng.randint(8, 20), "t": round(rng.uniform(0.2, 2.0), 3)}
    if kind == "pauli":
        return {"kind": kind, "n": rng.randint(8, 22), "t": round(rng.uniform(0.5, 10.0), 3)}
    if kind == "noise":
        return {"kind": kind, "n": rng.randint(4, 13), "depth": rng.randint(2, 8), "trajectories": log(16, 1024)}
    return {"kind": kind, "n": rng.randint(12, 26), "shots": log(100, 8192), "terms": log(4, 96)}


# ------------------------------------------------------------------ inputs
def _haar(rng, k, count):
    z = rng.standard_normal((count, k, k)) + 1j * rng.standard_normal((count, k, k))
    q, r = np.linalg.qr(z)
    d = np.diagonal(r, axis1=1, axis2=2)
    return q * (d / np.abs(d))[:, None, :]


def _qv(rng, n, depth):
    out = []
    for _ in range(depth):
        p, u = rng.permutation(n), _haar(rng, 4, n // 2)
        out += [("u", (int(p[2 * j]), int(p[2 * j + 1])), (), u[j]) for j in range(n // 2)]
    return out


def _layers(rng, n, depth):
    out = []
    for d in range(depth):
        u = _haar(rng, 2, n)
        out += [("u", (q,), (), u[q]) for q in range(n)]
        out += [("cz", (a, a + 1), (), None) for a in range(d % 2, n - 1, 2)]
        if (d + 1) % 5 == 0:
            a, b, c = (int(q) for q in rng.choice(n, 3, replace=False))
            out.append(("ccx", (a, b, c), (), None))
    return out


def _qft(rng, n):
    out = [("u", (q,), (), u) for q, u in enumerate(_haar(rng, 2, n))]   # the state that is transformed
    h = np.array([[1, 1], [1, -1]]) / math.sqrt(2)
    for q in reversed(range(n)):
        out.append(("u", (q,), (), h))
        out += [("cp", (c, q), (), math.pi / 2 ** (q - c)) for c in reversed(range(q))]
    return out + [("swap", (q, n - 1 - q), (), None) for q in range(n // 2)]


def _gates(case, rng):
    """(what, qubits, controls, matrix) in the kernel API's terms: a 4x4's index bit 0 is its lower qubit."""
    n, out = case["n"], []
    for k in range(case["gates"]):
        what = ("1q", "2q", "diag", "phase", "mcx", "1q", "diag2", "fused", "mcu")[k % 9]
        q = [int(x) for x in rng.permutation(n)]
        ph = np.exp(1j * rng.uniform(0, 2 * math.pi, 4))
        if what == "1q":
            out.append((what, (q[0],), (), _haar(rng, 2, 1)[0]))
        elif what == "2q":
            out.append((what, tuple(sorted(q[:2])), (), _haar(rng, 4, 1)[0]))
        elif what == "diag":
            out.append((what, (q[0],), (), np.diag(ph[:2])))
        elif what == "phase":
            out.append((what, (q[0],), (), np.diag([1.0, ph[0]])))
        elif what == "diag2":
            out.append((what, tuple(sorted(q[:2])), (), np.diag(ph)))
        elif what == "mcx":
            out.append((what, (q[0],), tuple(q[1:2]), np.array([[0, 1], [1, 0]], complex)))
        elif what == "mcu":
            out.append((what, (q[0],), tuple(q[1:3]), _haar(rng, 2, 1)[0]))
        else:
            out.append((what, tuple(q[: min(n, 10)]), (), _haar(rng, 2, min(n, 10))))
    return out


def _circuit_list(case, rng):
    if case["kind"] == "plan" or case["family"] == "layers":
        return _layers(rng, case["n"], case["depth"])
    return _qv(rng, case["n"], case["depth"]) if case["family"] == "qv" else _qft(rng, case["n"])


def _terms(n, count, rng):
    """Random Pauli strings of weight 1-4 with normal coefficients: x masks, z masks, coefficients."""
    xs, zs = np.zeros(count, np.int64), np.zeros(count, np.int64)
    for k in range(count):
        w = int(rng.integers(1, min(4, n) + 1))
        for q, p in zip(rng.choice(n, w, replace=False), rng.integers(1, 4, w)):
            xs[k] |= int(p in (1, 2)) << int(q)
            zs[k] |= int(p in (2, 3)) << int(q)
    return xs, zs, rng.standard_normal(count)


def _spin_terms(n, rng, pairs=20):
    """Ising ring, transverse fields, and XX + YY on random pairs."""
    xs, zs, cs = [], [], []
    for i in range(n):
        xs.append(0), zs.append((1 << i) | (1 << (i + 1) % n)), cs.append(rng.uniform(-1, 1))
        xs.append(1 << i), zs.append(0), cs.append(rng.uniform(-1, 1))
    for _ in range(pairs):
        a, b = rng.choice(n, 2, replace=False)
        m, k = (1 << int(a)) | (1 << int(b)), rng.uniform(-0.5, 0.5)
        xs += [m, m]
        zs += [0, m]
        cs += [k, k]
    return np.array(xs), np.array(zs), np.array(cs)


def _random_state(n, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    s = torch.randn(1 << n, 2, device=DEV, generator=g)
    return torch.view_as_complex(s / s.double().square().sum().sqrt().float())


def _parity(x):
    for s in (16, 8, 4, 2, 1):
        x = x ^ (x >> s)
    return x & 1


def _by_mask(n, xs, zs, cs):
    """{x mask: complex128 [2^n] entries H[r, r ^ x]} of a Pauli sum."""
    r = torch.arange(1 << n, device=DEV)
    rows = {}
    for x, z, c in zip(xs.tolist(), zs.tolist(), cs.tolist()):
        w = c * 1j ** (bin(x & z).count("1") % 4)
        sign = 1.0 - 2.0 * _parity((r ^ x) & z).double()
        rows[x] = rows.get(x, 0) + w * sign
    return rows


def _csr(n, xs, zs, cs):
    """int32 row pointers and columns, complex64 values; columns ascending, zeros dropped."""
    rows = _by_mask(n, xs, zs, cs)
    r = torch.arange(1 << n, device=DEV, dtype=torch.int32)
    cols, order = torch.stack([r ^ x for x in rows], 1).sort(1)
    vals = torch.stack([v.to(torch.complex64) for v in rows.values()], 1).gather(1, order)
    keep = vals != 0
    ptr = torch.zeros((1 << n) + 1, dtype=torch.int32, device=DEV)
    ptr[1:] = keep.sum(1).cumsum(0)
    return ptr, cols[keep].contiguous(), vals[keep].contiguous()


def _ansatz(n, reps=4):
    """EfficientSU2: (gate, qubits, parameter index)."""
    out = []
    for r in range(reps + 1):
        out += [("ry", (q,), 2 * n * r + q) for q in range(n)]
        out += [("rz", (q,), 2 * n * r + n + q) for q in range(n)]
        if r < reps:
            out += [("cx", (q, q + 1), -1) for q in range(n - 1)]
    return out, 2 * n * (reps + 1)


def _brickwork(case, rng):
    """RY and RZ on every qubit, CX on alternating neighbours: (gate, qubits, angle)."""
    out = []
    for d in range(case["depth"]):
        for q in range(case["n"]):
            out += [("ry", (q,), float(rng.uniform(0, 2 * math.pi))), ("rz", (q,), float(rng.uniform(0, 2 * math.pi)))]
        out += [("cx", (q, q + 1), 0.0) for q in range(d % 2, case["n"] - 1, 2)]
    return out


# ------------------------------------------------------------- the program
def prepare(case, seed):
    from qsim_b200 import engine as E
    from qsim_b200.circuit import Circuit, lower
    from qsim_b200.paulis import PauliSum
    kind, rng, n = case["kind"], np.random.default_rng(seed), case.get("n")
    s = {"kind": kind, "case": case}
    if kind == "gates":
        s["program"] = []
        for what, q, ctrl, m in _gates(case, rng):
            if what in ("diag", "diag2"):
                m = np.diagonal(m)
            t = complex(m[1, 1]) if what == "phase" else torch.tensor(np.array(m), dtype=torch.complex64, device=DEV)
            if what == "fused":
                q = torch.tensor(q, dtype=torch.int32, device=DEV)
            s["program"].append((what, q, list(ctrl), t))
    elif kind in ("circuit", "plan"):
        qc = Circuit(n)
        for what, q, _, m in _circuit_list(case, rng):
            if what == "u":
                qc.unitary(m, q)
            elif what == "cp":
                qc.cp(m, *q)
            else:
                getattr(qc, what)(*q)
        if kind == "plan":
            E.set_jit(0)
            s["plan"], s["state"] = E.Plan(n, lower(qc)), E.empty_state(n, DEV)
        else:
            from blackwell_backend import BlackwellSimulator
            s["sim"], s["qc"] = BlackwellSimulator(DEV), qc
    elif kind == "batch":
        widths, per = _batch(case, rng)
        parts = []
        for w, gates in zip(widths, per):
            qc = Circuit(w)
            for _, q, _, m in gates:
                qc.unitary(m, q)
            parts.append(lower(qc))
        amps = np.array([1 << w for w in widths], np.int64)
        s["plan"] = E.BatchPlan(widths, np.cumsum([0] + [len(p) for p in parts]), np.concatenate(parts),
                                np.cumsum(amps) - amps)
        s["states"] = s["plan"].alloc_states()
    elif kind == "gradient":
        gates, count = _ansatz(n)
        qc = Circuit(n)
        for what, q, p in gates:
            qc.cx(*q) if what == "cx" else getattr(qc, what)(0.0, q[0], param_index=p)
        s["ops"], s["obs"] = lower(qc), PauliSum(*_terms(n, case["terms"], rng), n)
        s["theta"] = torch.tensor(rng.uniform(0, 2 * math.pi, (case["batch"], count)), dtype=torch.float32,
                                  device=DEV, requires_grad=True)
    elif kind in ("csr", "pauli"):
        xs, zs, cs = _spin_terms(n, rng)
        s["psi"], s["obs"] = _random_state(n, seed), PauliSum(xs, zs, cs, n)
        if kind == "csr":
            from blackwell_backend.hamiltonian import HamiltonianCSR
            s["h"] = HamiltonianCSR(*_csr(n, xs, zs, cs), n, s["obs"].spectral_bound())
    elif kind == "noise":
        from qsim_b200.noise import add_noise
        qc = Circuit(n)
        for what, q, a in _brickwork(case, rng):
            qc.cx(*q) if what == "cx" else getattr(qc, what)(a, q[0])
        s["qc"], s["seed"] = add_noise(qc, depolarizing=1e-3, amplitude_damping=1e-3, dephasing=1e-3), 1000003 * seed
    else:
        s["psi"], s["obs"] = _random_state(n, seed), PauliSum(*_terms(n, case["terms"], rng), n)
        s["generator"] = torch.Generator(device=DEV).manual_seed(seed)
    return s


def _widths(case):
    """The widths of a batch, the same for every seed."""
    rng = np.random.default_rng(case["circuits"])
    return [int(w) for w in rng.integers(case["lo"], case["hi"] + 1, case["circuits"])]


def _batch(case, rng):
    widths = _widths(case)
    return widths, [_qv(rng, w, w) for w in widths]


def _run_gates(s):
    import blackwell_kernels as bk
    state = bk.state_init(s["case"]["n"])
    for what, q, ctrl, m in s["program"]:
        if what == "1q":
            bk.apply_gate(state, m, q[0])
        elif what == "2q":
            bk.apply_gate_2q(state, m, *q)
        elif what == "diag":
            bk.apply_diagonal(state, m, q[0])
        elif what == "phase":
            bk.apply_diagonal_phase(state, m, q[0])
        elif what == "diag2":
            bk.apply_diagonal_2q(state, m, *q)
        elif what == "fused":
            bk.apply_gates_fused(state, m, q)
        else:
            bk.apply_mcgate(state, m, ctrl, q[0])
    return state


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "gates":
        return _run_gates(s)
    if kind == "circuit":
        return s["sim"].run_statevector(s["qc"])[0] if case["host"] else s["sim"].run_statevector_tensor(s["qc"])
    if kind == "plan":
        return s["plan"].execute_from_zero(s["state"])
    if kind == "batch":
        return s["plan"].execute(s["states"])
    if kind == "gradient":
        from qsim_b200.autograd import expectation
        s["theta"].grad = None
        energy = expectation(s["theta"], case["n"], s["ops"], s["obs"])
        energy.sum().backward()
        return {"energy": energy.detach(), "grad": s["theta"].grad}
    if kind == "csr":
        from blackwell_backend.chebyshev import chebyshev_evolve
        return chebyshev_evolve(s["psi"], s["h"], case["t"], precision=1e-6)[0]
    if kind == "pauli":
        from blackwell_backend.chebyshev import chebyshev_evolve_pauli
        return chebyshev_evolve_pauli(s["psi"], s["obs"], case["t"], precision=1e-6)[0]
    if kind == "noise":
        from qsim_b200.noise import run_trajectories
        states, branches = run_trajectories(s["qc"], case["trajectories"], seed=s["seed"])
        return {"states": states, "branches": branches}
    from qsim_b200 import engine as E
    return {"shots": E.sample(s["psi"], case["shots"], generator=s["generator"]),
            "energy": E.expect_pauli_sum(s["psi"], s["obs"]), "probs": E.probs(s["psi"])}


def work(case):
    """Bytes: inputs once and outputs once.  Flops: 14 per amplitude and dense
    2x2 (a complex product and half a sum for each of two entries), 30 per
    dense 4x4, 6 per complex product, 8 per complex multiply-add."""
    kind, N = case["kind"], 1 << case.get("n", 0)
    if kind == "gates":
        per = {"1q": 14, "2q": 30, "diag": 6, "phase": 3, "mcx": 0, "diag2": 6, "fused": 140, "mcu": 3.5}
        return {"bytes": 8 * N, "flops": N * sum(per[g[0]] for g in _gates(case, np.random.default_rng(0)))}
    if kind in ("circuit", "plan"):
        per = {"u": 14, "cz": 0, "ccx": 0, "cp": 1.5, "swap": 0}
        g = _circuit_list(case, np.random.default_rng(0))
        return {"bytes": 8 * N, "flops": N * sum(30 if len(x[1]) == 2 and x[0] == "u" else per[x[0]] for x in g)}
    if kind == "batch":
        widths = _widths(case)
        return {"bytes": 8 * sum(1 << w for w in widths), "flops": sum((30 << w) * w * (w // 2) for w in widths)}
    if kind == "gradient":   # forward, reverse on two vectors with one product per parameter, H psi
        n, B = case["n"], case["batch"]
        return {"bytes": 16 * B * 10 * n, "flops": B * N * (3 * 5 * n * (6 + 6) + 8 * 10 * n + 8 * case["terms"])}
    if kind in ("csr", "pauli"):
        n, t = case["n"], case["t"]
        degree, masks = (n + 10) * t + 20, n + min(20, n * (n - 1) // 2)
        row = 1 + n + 0.5 * (masks - n)
        return {"bytes": 16 * N + (12 * row * N + 4 * N if kind == "csr" else 0), "flops": degree * N * (8 * row + 12)}
    if kind == "noise":
        n, d, T = case["n"], case["depth"], case["trajectories"]
        rot, cx = 2 * n * d, sum((n - i % 2) // 2 for i in range(d))
        return {"bytes": 8 * N * T, "flops": T * N * (rot * 6 + (rot + 2 * cx) * 2 * (4 + 2))}
    return {"bytes": 12 * N + 8 * case["shots"], "flops": N * (3 + 8 * case["terms"])}


# ------------------------------------------------------------- in 64 bits
def _apply(psi, n, q, m, ctrl=()):
    """m (2x2 or 4x4, index bit k on q[k]) on psi [..., 2^n] in place, where all controls are 1.
    m may be a tensor [B, 2, 2] with psi [B, 2^n]."""
    touched = sorted(set(q) | set(ctrl), reverse=True)
    shape, axis, last = [psi.numel() >> n], {}, n
    for t in touched:
        shape += [1 << (last - 1 - t), 2]
        axis[t] = len(shape) - 1
        last = t
    v = psi.view(*shape, 1 << last)

    def part(bits):
        at = [slice(None)] * v.dim()
        for c in ctrl:
            at[axis[c]] = 1
        for k, t in enumerate(q):
            at[axis[t]] = (bits >> k) & 1
        return v[tuple(at)]

    old = [part(b) for b in range(1 << len(q))]
    if isinstance(m, torch.Tensor):
        w = lambda r, c: m[:, r, c].view(-1, *[1] * (old[0].dim() - 1))  # noqa: E731
        zero = lambda r, c: False  # noqa: E731
    else:
        w = lambda r, c: complex(m[r][c])  # noqa: E731
        zero = lambda r, c: m[r][c] == 0  # noqa: E731
    new = [sum(w(r, c) * old[c] for c in range(len(old)) if not zero(r, c)) for r in range(len(old))]
    for r, x in enumerate(new):
        old[r].copy_(x) if isinstance(x, torch.Tensor) else old[r].zero_()


_X = [[0, 1], [1, 0]]


def _play(n, gates, batch=1):
    psi = torch.zeros(batch, 1 << n, dtype=torch.complex128, device=DEV)
    psi[:, 0] = 1
    for what, q, ctrl, m in gates:
        if what == "cz":
            _apply(psi, n, q[1:], [[1, 0], [0, -1]], q[:1])
        elif what == "ccx":
            _apply(psi, n, q[2:], _X, q[:2])
        elif what == "cp":
            _apply(psi, n, q[1:], [[1, 0], [0, complex(math.cos(m), math.sin(m))]], q[:1])
        elif what == "swap":
            _apply(psi, n, q, [[1, 0, 0, 0], [0, 0, 1, 0], [0, 1, 0, 0], [0, 0, 0, 1]])
        elif what == "fused":
            for t, u in zip(q, m):
                _apply(psi, n, (t,), u)
        else:
            _apply(psi, n, q, m, ctrl)
    return psi


def _h_times(rows, psi):
    r = torch.arange(psi.shape[-1], device=DEV)
    out = torch.zeros_like(psi)
    for x, w in rows.items():
        out += w * psi[..., r ^ x]
    return out


def _exact_gradient(case, rng):
    n, B = case["n"], case["batch"]
    gates, count = _ansatz(n)
    xs, zs, cs = _terms(n, case["terms"], rng)
    theta = torch.tensor(rng.uniform(0, 2 * math.pi, (B, count)), dtype=torch.float32, device=DEV).double()

    def matrix(what, p, sign):
        h = sign * theta[:, p] / 2
        if what == "ry":
            return torch.stack([h.cos(), -h.sin(), h.sin(), h.cos()], 1).view(B, 2, 2).to(torch.complex128)
        z = torch.zeros_like(h)
        return torch.complex(torch.stack([h.cos(), z, z, h.cos()], 1), torch.stack([-h.sin(), z, z, h.sin()], 1)).view(B, 2, 2)

    psi = torch.zeros(B, 1 << n, dtype=torch.complex128, device=DEV)
    psi[:, 0] = 1
    for what, q, p in gates:
        _apply(psi, n, q[1:], _X, q[:1]) if what == "cx" else _apply(psi, n, q, matrix(what, p, 1))
    lam, r = torch.zeros_like(psi), torch.arange(1 << n, device=DEV)
    for x, z, c in zip(xs.tolist(), zs.tolist(), cs.tolist()):
        w = c * 1j ** (bin(x & z).count("1") % 4)
        lam += w * ((1.0 - 2.0 * _parity((r ^ x) & z).double()) * psi[:, r ^ x])
    energy = (psi.conj() * lam).sum(1).real
    grad = torch.zeros(B, count, dtype=torch.float64, device=DEV)
    for what, q, p in reversed(gates):
        if what == "cx":
            for v in (psi, lam):
                _apply(v, n, q[1:], _X, q[:1])
            continue
        a, l = (v.view(B, -1, 2, 1 << q[0]) for v in (psi, lam))
        if what == "ry":    # Y psi = (-i a1, i a0)
            im = (l[:, :, 0].conj() * -1j * a[:, :, 1] + l[:, :, 1].conj() * 1j * a[:, :, 0]).imag
        else:
            im = (l[:, :, 0].conj() * a[:, :, 0] - l[:, :, 1].conj() * a[:, :, 1]).imag
        grad[:, p] += im.sum((1, 2))
        u = matrix(what, p, -1)
        _apply(psi, n, q, u)
        _apply(lam, n, q, u)
    return {"energy": energy, "grad": grad}


def _exact_evolution(case, rng, seed):
    n, t = case["n"], case["t"]
    xs, zs, cs = _spin_terms(n, rng)
    rows = _by_mask(n, xs, zs, cs)
    if case["kind"] == "csr":
        rows = {x: w.to(torch.complex64).to(torch.complex128) for x, w in rows.items()}
    x = _random_state(n, seed).to(torch.complex128)
    steps = max(1, math.ceil(float(np.abs(cs).sum()) * t / 16))   # Taylor steps of norm at most 16
    for _ in range(steps):
        term, k = x, 0
        while term.norm() > 1e-14 and k < 120:
            k += 1
            term = _h_times(rows, term) * (-1j * t / (steps * k))
            x = x + term
    return x


def _uniforms(seeds, count):
    """splitmix64 of each seed, the top 53 bits in [0, 1): [seeds, count]."""
    z = seeds[:, None] + np.arange(1, count + 1, dtype=np.uint64)[None] * np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return ((z ^ (z >> np.uint64(31))) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


def _exact_noise(case, rng, seed, p=1e-3):
    """Trajectories with the same uniforms: a depolarizing channel takes X, Y or Z in the last p of [0, 1); damping and
    dephasing jump where u < p P(1), and the state is normalised after either branch."""
    n, T = case["n"], case["trajectories"]
    gates = _brickwork(case, rng)
    seeds = np.uint64(1000003 * seed) + np.arange(T, dtype=np.uint64)
    u = torch.tensor(_uniforms(seeds, 3 * sum(len(q) for _, q, _ in gates)), device=DEV)
    psi = torch.zeros(T, 1 << n, dtype=torch.complex128, device=DEV)
    psi[:, 0] = 1
    eye = torch.eye(2, dtype=torch.complex128, device=DEV)
    paulis = torch.stack([eye, eye.flip(0), torch.tensor([[0, -1j], [1j, 0]], dtype=torch.complex128, device=DEV),
                          torch.diag(torch.tensor([1, -1], dtype=torch.complex128, device=DEV))])
    k = 0
    for what, q, a in gates:
        c, s = math.cos(a / 2), math.sin(a / 2)
        if what == "cx":
            _apply(psi, n, q[1:], _X, q[:1])
        else:
            _apply(psi, n, q, [[c, -s], [s, c]] if what == "ry" else [[complex(c, -s), 0], [0, complex(c, s)]])
        for t in q:
            over = u[:, k] - (1 - p)
            branch = (over >= 0).long() + (over >= p / 3).long() + (over >= 2 * (p / 3)).long()
            _apply(psi, n, (t,), paulis[branch])
            for j, damping in ((k + 1, True), (k + 2, False)):
                v = psi.view(T, -1, 2, 1 << t)
                s0, s1 = ((v[:, :, b].abs() ** 2).sum((1, 2)) for b in (0, 1))
                jump = u[:, j] < p * s1 / (s0 + s1)
                norm = (s0 + (1 - p) * s1).sqrt()
                m = torch.zeros(T, 2, 2, dtype=torch.complex128, device=DEV)
                m[:, 0, 0] = torch.where(jump, 0, 1 / norm)
                m[:, 1, 1] = torch.where(jump, 0 if damping else 1 / s1.sqrt(), math.sqrt(1 - p) / norm)
                if damping:
                    m[:, 0, 1] = torch.where(jump, 1 / s1.sqrt(), 0)
                _apply(psi, n, (t,), m)
            k += 3
    return psi


def exact(case, seed):
    kind, rng, n = case["kind"], np.random.default_rng(seed), case.get("n")
    if kind == "gates":   # the matrices as the program holds them, in 32 bits
        return _play(n, [(w, q, c, np.asarray(m if w == "phase" else m.astype(np.complex64), np.complex128))
                         for w, q, c, m in _gates(case, rng)]).view(-1)
    if kind in ("circuit", "plan"):
        return _play(n, _circuit_list(case, rng)).view(-1)
    if kind == "batch":
        widths, per = _batch(case, rng)
        return torch.cat([_play(w, g).view(-1) for w, g in zip(widths, per)])
    if kind == "gradient":
        return _exact_gradient(case, rng)
    if kind in ("csr", "pauli"):
        return _exact_evolution(case, rng, seed)
    if kind == "noise":
        return {"states": _exact_noise(case, rng, seed), "branches": None}
    psi = _random_state(n, seed).to(torch.complex128)
    xs, zs, cs = _terms(n, case["terms"], rng)
    r, energy = torch.arange(1 << n, device=DEV), 0.0
    for x, z, c in zip(xs.tolist(), zs.tolist(), cs.tolist()):
        w = c * 1j ** (bin(x & z).count("1") % 4)
        energy += (w * (psi.conj() * (1.0 - 2.0 * _parity((r ^ x) & z).double()) * psi[r ^ x]).sum()).real.item()
    return {"shots": None, "energy": energy, "probs": psi.abs() ** 2}
