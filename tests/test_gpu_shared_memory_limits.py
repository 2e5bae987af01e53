"""Calls of one kernel with different amounts of shared memory from several threads, each with its own handle: the limit
is the kernel's, so no call may lower it under another's launch."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(jobs):
    import torch

    torch.cuda.init()
    failed = []
    gate = threading.Barrier(len(jobs))

    def work(job):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                gate.wait()
                job()
        except Exception as e:   # noqa: BLE001 - reported below
            failed.append(e)

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not failed, failed[0]


def _sum(n, terms):
    from qsim_b200.paulis import PauliSum

    x = np.arange(1, terms + 1, dtype=np.uint64)          # as many X masks as terms: the largest table for the count
    return PauliSum(x, np.zeros(terms, np.uint64), np.full(terms, 2.0 ** -10), n)


@pytest.mark.parametrize("what", ["expect", "apply"])
def test_pauli_tables(what):
    import torch
    from qsim_b200 import engine as E

    n, calls = 11, 1500

    def job(terms):
        def run():
            state = E.empty_state(n)
            state.zero_()
            state[0] = 1
            ps = _sum(n, terms)
            for _ in range(calls):
                if what == "expect":
                    assert E.expect_pauli_sum(state, ps) == 0.0
                else:
                    out = E.apply_pauli_sum(state, ps)
            if what == "apply":
                assert float(out.real.sum()) == terms * 2.0 ** -10
            torch.cuda.current_stream().synchronize()
        return run

    _run([job(t) for t in (840, 900, 960, 1024)])


def test_gradients_of_several_widths():
    from qsim_b200 import engine as E
    from qsim_b200.circuit import Circuit, lower
    from qsim_b200.paulis import PauliSum

    def job(n):
        qc = Circuit(n)
        for q in range(n):
            qc.ry(0.0, q, param_index=q)
        ops, theta = lower(qc), np.linspace(0.1, 1.0, n)[None]
        ps = PauliSum(np.zeros(1, np.uint64), np.ones(1, np.uint64), np.ones(1), n)

        def run():
            for _ in range(400):
                e, g = E.adjoint_gradient(n, ops, n, theta, ps)
                assert abs(e[0] - np.cos(0.1)) < 1e-5 and abs(g[0, 0] + np.sin(0.1)) < 1e-5
        return run

    _run([job(n) for n in (4, 8, 11, 12)])
