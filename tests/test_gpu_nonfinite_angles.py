"""Gradients at parameters that are not finite: the cosine and sine of an infinity or NaN are NaN, so the energy and
the derivative of every rotation are, whatever the tiles' number format. Parameters that no rotation takes keep
derivative 0, and the other circuits of a batch their values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _circuit(n, axis):
    from quaru_gb300 import ParamGate
    from quaru_gb300 import operation as O

    make = {"rx": ParamGate.rx, "ry": ParamGate.ry, "rz": ParamGate.rz}[axis]
    gates = [ParamGate.ry(q, q) for q in range(n)] + [make(n // 2, n), ParamGate.fixed(O.cnot(0, n - 1)), ParamGate.rx(0, n + 1)]
    return gates, n + 3  # the last parameter belongs to no gate


@pytest.mark.parametrize("precision,arith", [(0, 0), (0, 1), (0, 2), (0, 3), (1, 1)])
@pytest.mark.parametrize("axis", ["rx", "ry", "rz"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n", [3, 9, 13])
def test_single(n, value, axis, precision, arith):
    import quaru_gb300 as q

    gates, count = _circuit(n, axis)
    params = np.linspace(0.1, 1.0, count)
    reg = q.Register.from_int(n, 0, precision=precision)
    reg.set_arith(arith)
    before = reg.adjoint_gradient(gates, params, [(0.5, 0, 1), (0.25, 2, 0)])
    bad = params.copy()
    bad[n] = value
    energy, grad = reg.adjoint_gradient(gates, bad, [(0.5, 0, 1), (0.25, 2, 0)])
    assert np.isnan(energy)
    assert np.isnan(grad[:-1]).all() and grad[-1] == 0.0
    unused = params.copy()
    unused[-1] = value  # of no gate: nothing changes
    again = reg.adjoint_gradient(gates, unused, [(0.5, 0, 1), (0.25, 2, 0)])
    assert again[0] == before[0]
    np.testing.assert_array_equal(again[1], before[1])


@pytest.mark.parametrize("precision,arith", [(0, 0), (0, 1), (0, 2), (1, 1)])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_batch(value, precision, arith):
    from quaru_gb300.batch import Batch

    circuits, at = [], [0]
    for n, axis in ((3, "rx"), (9, "ry"), (13, "rz"), (12, "rx")):
        gates, count = _circuit(n, axis)
        circuits.append((n, gates, count, [(0.5, 0, 1), (0.25, 2, 0)]))
        at.append(at[-1] + count)
    b = Batch(circuits, precision=precision, arith=arith, chunk_log2=11, ctas_per_sm=2)
    params = np.linspace(0.1, 1.0, at[-1])
    e0, g0 = b.run(params)
    assert np.isfinite(e0).all() and np.isfinite(g0).all()
    for c in range(4):
        bad = params.copy()
        bad[at[c] + circuits[c][0]] = value
        e, g = b.run(bad)
        assert np.isnan(e[c])
        assert np.isnan(g[at[c]:at[c + 1] - 1]).all() and g[at[c + 1] - 1] == 0.0
        rest = np.r_[0:at[c], at[c + 1]:at[-1]]
        np.testing.assert_array_equal(g[rest], g0[rest])
        np.testing.assert_array_equal(np.delete(e, c), np.delete(e0, c))
    e, g = b.run(params)
    np.testing.assert_array_equal(e, e0)
    np.testing.assert_array_equal(g, g0)
