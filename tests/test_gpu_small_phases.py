"""RZ by small angles on complex64 registers: the imaginary parts that such a phase makes keep their relative
accuracy, through the products of a run of RZ gates.

RY(pi / 2) and RZ(t_k) on every qubit with H = sum_k c_k X_k has dE/dt_k = -c_k sin t_k. Every amplitude's imaginary part is
a sum of the angles, each term of a derivative at most sum |c t|; 24 float roundings per gate as in the other
gradient tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, e, rng):
    from quaru_gb300 import ParamGate

    t = 10.0 ** -e * rng.uniform(0.5, 2.0, n) * rng.choice([-1.0, 1.0], n)
    c = rng.uniform(0.5, 2.0, n)
    gates = [ParamGate.ry(k, 0) for k in range(n)] + [ParamGate.rz(k, 1 + k) for k in range(n)]
    return gates, np.concatenate([[np.pi / 2], t]), t, c, [(c[k], 1 << k, 0) for k in range(n)]


def _check(n, t, c, grad):
    want = -c * np.sin(t)
    tol = 24 * 2 * n * 2.0 ** -24 * np.sum(np.abs(c * t))
    assert np.all(np.abs(grad[1:] - want) <= tol), (np.max(np.abs(grad[1:] - want)), tol)


@pytest.mark.parametrize("e", [3, 8, 10, 12, 16, 18, 20, 25])
@pytest.mark.parametrize("n", [1, 2, 5, 9, 11, 13])
def test_single(n, e):
    import quaru_gb300 as q

    gates, params, t, c, terms = _problem(n, e, np.random.default_rng([n, e]))
    reg = q.Register.from_int(n, 0, precision=q.QS_PREC_C64)
    _check(n, t, c, reg.adjoint_gradient(gates, params, terms)[1])


@pytest.mark.parametrize("e", [3, 12, 20])
def test_batch(e):
    import quaru_gb300 as q
    from quaru_gb300.batch import Batch

    rng = np.random.default_rng(e)
    problems = [(n, *_problem(n, e, rng)) for n in (1, 8, 11, 12)]
    b = Batch([(n, g, p.size, h) for n, g, p, t, c, h in problems], precision=q.QS_PREC_C64, chunk_log2=11, ctas_per_sm=2)
    _, grads = b.run(np.concatenate([p for _, _, p, _, _, _ in problems]))
    at = 0
    for n, g, p, t, c, h in problems:
        _check(n, t, c, grads[at:at + p.size])
        at += p.size
