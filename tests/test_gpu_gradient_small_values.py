"""Gradients in QS_ARITH_EXACT hold amplitudes in FP64: derivatives and energies that hang on amplitudes far below the
state's norm keep their relative accuracy.

RY(t_i) on every qubit of |0..0> with H = sum_i c_i Z_i has dE/dt_i = -c_i sin t_i. Every amplitude is a product of at
most n factors, the derivative a sum of terms of one sign times differences of H's diagonal, which cancel by at most
sum |c| / |c_i|; 24 roundings per gate as in the other gradient tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _angles(rng, n):
    t = 10.0 ** -rng.uniform(3, 25, n) * rng.choice([-1.0, 1.0], n)
    t[0] = 1e-24
    return t


def _check(n, t, c, energy, grad):
    tol = 24 * n * 2.0 ** -53 * np.sum(np.abs(c)) / np.abs(c)
    want = -c * np.sin(t)
    assert np.all(np.abs(grad - want) <= tol * np.abs(want)), np.max(np.abs(grad / want - 1))
    assert abs(energy - np.sum(c * np.cos(t))) <= 24 * n * 2.0 ** -53 * np.sum(np.abs(c))


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 11, 13, 15])
def test_single(n):
    import quaru_gb300 as q
    from quaru_gb300 import ParamGate

    rng = np.random.default_rng(n)
    t, c = _angles(rng, n), rng.uniform(0.5, 2.0, n)
    reg = q.Register.from_int(n, 0)  # QS_ARITH_EXACT unless told otherwise
    energy, grad = reg.adjoint_gradient([ParamGate.ry(k, k) for k in range(n)], t, [(c[k], 0, 1 << k) for k in range(n)])
    _check(n, t, c, energy, grad)


def test_batch():
    import quaru_gb300 as q
    from quaru_gb300 import ParamGate
    from quaru_gb300.batch import Batch

    rng = np.random.default_rng(77)
    sizes = (1, 8, 11, 12, 14)
    t = [_angles(rng, n) for n in sizes]
    c = [rng.uniform(0.5, 2.0, n) for n in sizes]
    b = Batch([(n, [ParamGate.ry(k, k) for k in range(n)], n, [(x[k], 0, 1 << k) for k in range(n)]) for n, x in zip(sizes, c)],
              arith=q.QS_ARITH_EXACT, chunk_log2=11, ctas_per_sm=2)
    energies, grads = b.run(np.concatenate(t))
    at = 0
    for n, tt, cc, e in zip(sizes, t, c, energies):
        _check(n, tt, cc, e, grads[at:at + n])
        at += n
