"""What a register records of its zeros behind measurements: registers whose gates were captured into a graph record
nothing (a replay changes the state behind the library's back), and a collapse whose probability sum is zero or NaN
fills the kept half with NaN, as the reference's division does, whatever was recorded before it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sequence", [False, True])
@pytest.mark.parametrize("n", [5, 12, 15, 17])
def test_replays_behind_a_measurement(n, sequence):
    """Capture, measure, replay; then a clone's gates and measurements of other qubits, against a register that ran the
    same gates itself. QS_ARITH_EXACT on registers of up to 20 qubits: sums in index order, so all bits agree."""
    import quaru_gb300 as q
    import torch
    from quaru_gb300 import operation as O

    ops = [O.hadamard(2), O.cnot(2, n - 1), O.hadamard(1)]

    def run(r):
        for g in ops:
            r.try_apply_fast(g)

    run(q.Register.from_int(n, 0))  # the kernels are loaded before the capture
    a, b = q.Register.from_int(n, 0), q.Register.from_int(n, 0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(a.stream), capture_error_mode="thread_local"):
        run(a)

    def replay():
        with torch.cuda.stream(torch.cuda.ExternalStream(a.stream)):
            graph.replay()
        torch.cuda.synchronize()
        run(b)

    def measure(r, targets, draws):
        if sequence:
            return r.measure_sequence(targets, draws)
        return [r.measure(t, d) for t, d in zip(targets, draws)]

    replay()
    assert measure(a, [2, n - 1], [0.3, 0.6]) == measure(b, [2, n - 1], [0.3, 0.6])
    replay()
    c = a.clone()
    assert measure(a, [1, 0, 2, n - 1], [0.9, 0.5, 0.4, 0.7]) == measure(b, [1, 0, 2, n - 1], [0.9, 0.5, 0.4, 0.7])
    np.testing.assert_array_equal(a.state, b.state)
    # the clone: the state before those measurements
    d = q.Register.from_int(n, 0)
    d.state = c.state
    for r in (c, d):
        r.try_apply_fast(O.not_(2))
        r.apply_gates([O.hadamard(0), O.cnot(n - 1, 0)], fuse=1)
    np.testing.assert_array_equal(c.state, d.state)
    assert measure(c, [0, 1], [0.2, 0.8]) == measure(d, [0, 1], [0.2, 0.8])
    np.testing.assert_array_equal(c.state, d.state)


@pytest.mark.parametrize("precision,arith", [(0, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("form", ["calls", "sequence", "in_place"])
@pytest.mark.parametrize("n", [6, 15, 17])
def test_collapse_onto_nothing(n, form, precision, arith, monkeypatch):
    """Draws above 1 take outcome 1 of qubits that are 0: 0 / 0 on the whole kept half, then gates."""
    import quaru_gb300 as q
    from quaru_gb300 import operation as O

    if form == "in_place":
        monkeypatch.setenv("QS_MEASURE_COMPACT", "off")
    targets = [n - 2, 3, 0, n - 1]
    for bad in range(4):  # the measurement that has nothing to collapse onto
        draws = [0.5] * 4
        draws[bad] = 1.5
        g = q.Register.from_int(n, 0, precision=precision)
        g.set_arith(arith)
        want = np.zeros(1 << n, dtype=complex)
        want[0] = 1.0
        i = np.arange(1 << n)
        outcomes = []
        for t, d in zip(targets, draws):  # src/register.rs:306-339
            p0 = np.sum(np.abs(want[(i >> t & 1) == 0]) ** 2)
            p1 = np.sum(np.abs(want[(i >> t & 1) == 1]) ** 2)
            res = bool(d > p0)
            with np.errstate(all="ignore"):
                want = np.where((i >> t & 1) == res, want / np.sqrt(p1 if res else p0), 0.0)
            outcomes.append(res)
        got = g.measure_sequence(targets, draws) if form != "calls" else [g.measure(t, d) for t, d in zip(targets, draws)]
        assert got == outcomes
        for op, move in ((None, None), (O.not_(targets[bad]), 1 << targets[bad]), (O.not_(1), 2)):
            if op is not None:
                g.try_apply_fast(op)
                want = want[i ^ move]
            s = g.state
            np.testing.assert_array_equal(np.isnan(s), np.isnan(want))
            np.testing.assert_array_equal(s[~np.isnan(s)], want[~np.isnan(want)])


@pytest.mark.parametrize("arith", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [6, 13, 16])
def test_fused_blocks_that_overflow(n, arith):
    """Finite gates whose fused block is not: it makes NaN of zeros, those of measured qubits too."""
    import quaru_gb300 as q

    ops = [q.Operation(np.array([[2.0, 1.0], [1.0, -2.0]], dtype=complex), [1]),
           q.Operation(np.array([[0.5, 1.0], [1e308, 1e308]], dtype=complex), [3])]
    a, b = q.Register.from_int(n, 0), q.Register.from_int(n, 0)
    for r in (a, b):
        r.set_arith(arith)
    a.measure_sequence([n - 1, 2], [0.5, 0.5])
    st = np.zeros(1 << n, dtype=complex)
    st[0] = 1.0
    b.state = st
    for r in (a, b):
        r.apply_gates(ops, fuse=2, max_width=4)
    x, y = a.state, b.state
    np.testing.assert_array_equal(np.isnan(x), np.isnan(y))
    assert np.isnan(x).any()
    assert not a.measure(3, 0.25) and not b.measure(3, 0.25)  # the half without NaN
    np.testing.assert_array_equal(np.isnan(a.state), np.isnan(b.state))
