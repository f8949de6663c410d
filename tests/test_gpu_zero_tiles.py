"""Gradients where whole tiles of the sweeps stay zero: circuits on a few qubits of a basis state, with observables
that put lambda where psi is zero, dense fixed gates among the rotations, and negative zeros in the state.

Bar: the adjoint walk in plain numpy within the bound of the sweeps' own tests (24 m 2^-53 or 2^-24 of the
norms' product, m gates)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _circuit(n, few, rng, fixed):
    from quaru_gb300 import Operation, ParamGate
    from quaru_gb300 import operation as O

    make = (ParamGate.rx, ParamGate.ry, ParamGate.rz)
    gates = []
    for i in range(40):
        t = [int(x) for x in rng.permutation(few)]
        if fixed and i % 9 == 4:
            m = np.linalg.qr(rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2)))[0]
            gates.append(ParamGate.fixed(Operation(m, t[:1])))
        elif i % 3 == 2:
            gates.append(ParamGate.fixed(O.cnot(t[0], t[1])))
        else:
            gates.append(make[i % 3 if i % 2 else 1](t[0], len([g for g in gates if g.kind])))
    npar = len([g for g in gates if g.kind])
    terms = [(0.7, 0, 1 << few[0]), (-0.4, 1 << few[1], 0), (0.9, (1 << (n - 1)) | (1 << few[0]), 1 << few[2]),
             (1.3, 1 << (n - 1), 0), (0.2, 0, (1 << few[2]) | 1)]
    return gates, rng.uniform(0, 4 * math.pi, npar), terms


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("n,few", [(12, [0, 1, 2]), (13, [0, 6, 12]), (14, [11, 12, 13]), (14, [3, 9, 12])])
def test_gradient_with_zero_tiles(n, few, fixed, precision):
    import quaru_gb300 as q
    from quaru_gb300.batch import Batch
    from tests.test_gpu_sweep_programs import _reference

    rng = np.random.default_rng([n, few[1], fixed, precision])
    gates, params, terms = _circuit(n, few, rng, fixed)
    psi = np.full(1 << n, complex(-0.0, -0.0))
    psi[0] = 1.0
    reg = q.Register.from_int(n, 0, precision=precision)
    reg.set_arith(q.QS_ARITH_FMA)
    reg.state = psi
    energy, grad = reg.adjoint_gradient(gates, params, terms)
    e, g, scale = _reference(psi, n, gates, params, terms)
    tol = 24 * len(gates) * (2.0 ** -24 if precision else 2.0 ** -53) * scale
    assert abs(energy - e) <= tol
    assert np.max(np.abs(grad - g)) <= tol
    be, bg = Batch([(n, gates, params.size, terms)], precision=precision, arith=q.QS_ARITH_FMA).run(params)
    assert abs(be[0] - e) <= tol
    assert np.max(np.abs(bg - g)) <= tol
