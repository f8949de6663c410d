"""Gates that visit only the amplitudes a register can have: from a basis state on, a qubit no gate has acted on
keeps its value, and after a measurement the measured one does.

Bar: a register made from an integer gives, value for value, what a register does whose state was set to
the same basis vector (nothing is known of it): every arithmetic, single sweeps, stages and blocks, targets in
all positions, controls on known qubits at and off their values, wide gates, gates after measurements,
and matrices whose entries overflow the register's precision, which make zeros NaN.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gates(rng, n, m):
    from quaru_gb300 import operation as O
    from quaru_gb300.operation import Operation
    from tests.test_gpu_fusion import rand_unitary

    ops = []
    few = [int(x) for x in rng.permutation(n)[: n // 2]]  # the other qubits stay as they are at first
    for i in range(m):
        pool = few if i < 2 * m // 3 else list(range(n))
        t = [int(x) for x in rng.choice(pool, 3, replace=False)]
        c = int(rng.choice([x for x in range(n) if x not in t]))
        k = i % 8
        if k == 0:
            ops.append(Operation(rand_unitary(rng, 1), t[:1]))
        elif k == 1:
            ops.append(O.cnot(t[0], t[1]))
        elif k == 2:
            ops.append(O.to_controlled(Operation(rand_unitary(rng, 1), t[:1]), c))
        elif k == 3:
            ops.append(O.cnot(c, t[0]))
        elif k == 4:
            ops.append(Operation(rand_unitary(rng, 2), t[:2]))
        elif k == 5:
            ops.append(O.hadamard(t[0]))
        elif k == 6:
            ops.append(O.swap(t[0], t[1]))
        else:
            ops.append(Operation(np.diag(np.exp(1j * rng.normal(size=8))), t))
    wide = [int(x) for x in rng.permutation(n)[:7]]
    ops.insert(m // 2, Operation(np.eye(128, dtype=complex)[rng.permutation(128)], wide))
    return ops


def _pair(n, k, precision, arith):
    import quaru_gb300 as q

    a = q.Register.from_int(n, k, precision=precision)
    b = q.Register.from_int(n, k, precision=precision)
    st = np.zeros(1 << n, dtype=np.complex128)
    st[k] = 1.0
    b.state = st
    for r in (a, b):
        r.set_arith(arith)
    return a, b


@pytest.mark.parametrize("fuse", [0, 1, 2])
@pytest.mark.parametrize("precision,arith", [(0, 0), (0, 1), (0, 2), (0, 3), (1, 1)])
@pytest.mark.parametrize("n", [15, 16, 17, 19])
def test_basis_state_equals_state_set(n, precision, arith, fuse):
    rng = np.random.default_rng([n, precision, arith, fuse])
    for k in (0, int(rng.integers(1 << n)), (1 << n) - 1):
        a, b = _pair(n, k, precision, arith)
        first, second = _gates(rng, n, 10), _gates(rng, n, 24)
        draws = [float(x) for x in rng.uniform(size=3)]
        qubits = [int(x) for x in rng.permutation(n)[:3]]
        for r in (a, b):
            r.apply_gates(first, fuse=fuse)
        np.testing.assert_array_equal(a.state, b.state)
        c = a.clone()
        for r in (a, b, c):
            for g in second[:4]:
                r.try_apply_fast(g)
            for t, d in zip(qubits, draws):
                r.measure(t, d)
            r.apply_gates(second, fuse=fuse)
        # the parallel sums of a measurement group their terms alike: the states stay the same values
        np.testing.assert_array_equal(a.state, b.state)
        np.testing.assert_array_equal(a.state, c.state)


@pytest.mark.parametrize("precision,big", [(0, np.inf), (1, 1e300)])
@pytest.mark.parametrize("fuse", [0, 1, 2])
def test_overflowing_entries_assume_nothing(fuse, precision, big):
    import quaru_gb300 as q

    a, b = _pair(16, 5, precision, 1)
    ops = [q.Operation(np.array([[1.0, big], [0.5, 1.0]], dtype=complex), [3])]
    with np.errstate(all="ignore"):
        for r in (a, b):
            r.apply_gates(ops, fuse=fuse)
        x, y = a.state, b.state
    np.testing.assert_array_equal(np.isnan(x), np.isnan(y))
    np.testing.assert_array_equal(x[~np.isnan(x)], y[~np.isnan(y)])


@pytest.mark.parametrize("fuse", [0, None])
def test_captured_gates_serve_any_state(fuse):
    """Gates captured while the register is a basis state, replayed on what they made of it, on a state set later
    and after a measurement."""
    import quaru_gb300 as q
    import torch
    from quaru_gb300 import operation as O

    n = 17
    ops = [O.hadamard(3), O.cnot(3, 16), q.Operation(np.array([[0.6, 0.8], [-0.8, 0.6]]), [9]), O.cnot(9, 0)]

    def run(r):
        if fuse is None:
            for g in ops:
                r.try_apply_fast(g)
        else:
            r.apply_gates(ops, fuse=fuse)

    a, b = q.Register.from_int(n, 0), q.Register.from_int(n, 0)
    run(q.Register.from_int(n, 0))  # the kernels are loaded before the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(a.stream), capture_error_mode="thread_local"):
        run(a)
    st = np.zeros(1 << n, dtype=np.complex128)
    st[12345] = 1j
    for step in ("first", "again", "measured", "set"):
        if step == "measured":
            assert a.measure(5, 0.5) == b.measure(5, 0.5)
            assert a.measure(16, 0.3) == b.measure(16, 0.3)
        if step == "set":
            a.state, b.state = st, st
        with torch.cuda.stream(torch.cuda.ExternalStream(a.stream)):
            graph.replay()
        torch.cuda.synchronize()
        run(b)
        np.testing.assert_array_equal(a.state, b.state)
    a.try_apply_fast(O.hadamard(7))
    b.try_apply_fast(O.hadamard(7))
    np.testing.assert_array_equal(a.state, b.state)
