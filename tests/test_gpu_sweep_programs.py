"""Gradients of random circuits against the adjoint walk in plain numpy, over what the sweeps' pass programs
tell apart: tiles of every size (a partial warp up to several tiles), rotations of every axis next to each
other on one qubit, runs of RZ before and behind runs of CNOT, X and SWAP (with controls inside and outside
the tile), shared parameters, other fixed gates, half-turn and zero angles, states with zeros and of large
spread; and a fixed gate that is not unitary, on registers of one tile, which keep the gates' order (with
such a gate the walk's inner products depend on it, and several tiles move gates past disjoint ones).

Tolerance: an application of a gate leaves at most 8 roundings on an amplitude, and an inner product sees
three such walks of m gates, so 24 m 2^-53 (complex128) or 2^-24 (complex64) of the norms' product."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAULI = {1: np.array([[0, 1], [1, 0]]), 2: np.array([[0, -1j], [1j, 0]]), 3: np.diag([1.0, -1.0])}


def _apply(psi, n, m, targets):
    k = len(targets)
    axes = [n - 1 - t for t in reversed(targets)]
    v = np.moveaxis(psi.reshape([2] * n), axes, range(k))
    shape = v.shape
    v = (m @ v.reshape(1 << k, -1)).reshape(shape)
    return np.moveaxis(v, range(k), axes).reshape(-1)


def _pauli(psi, x, z):
    j = np.arange(psi.size) ^ x
    sign = np.array([(-1) ** bin(z & int(i)).count("1") for i in j])
    return 1j ** bin(x & z).count("1") * sign * psi[j]


def _reference(psi, n, gates, params, terms):
    def matrix(g):
        if g.kind == 0:
            return g.op.matrix, g.op.targets
        th = params[g.param]
        return math.cos(th / 2) * np.eye(2) - 1j * math.sin(th / 2) * PAULI[g.kind], [g.target]

    for g in gates:
        psi = _apply(psi, n, *matrix(g))
    lam = sum(c * _pauli(psi, x, z) for c, x, z in terms)
    energy = float(np.vdot(psi, lam).real)
    grad = np.zeros(len(params))
    scale = np.linalg.norm(psi) * sum(abs(c) for c, _, _ in terms) * np.linalg.norm(psi)
    for g in reversed(gates):
        if g.kind:
            grad[g.param] += np.vdot(lam, _apply(psi, n, PAULI[g.kind], [g.target])).imag
        m, t = matrix(g)
        psi, lam = _apply(psi, n, m.conj().T, t), _apply(lam, n, m.conj().T, t)
        scale = max(scale, np.linalg.norm(psi) * np.linalg.norm(lam))
    return energy, grad, scale


def _circuit(n, m, rng, batch, unitary=True):
    from quaru_gb300 import Operation, ParamGate
    from quaru_gb300 import operation as O

    make = (ParamGate.rx, ParamGate.ry, ParamGate.rz)
    gates, npar = [], 0
    while len(gates) < m:
        k = int(rng.integers(10))
        q = [int(t) for t in rng.permutation(n)]
        if k < 2:  # a layer of RZ and a ladder, in either order
            layer = [ParamGate.rz(t, npar + t) for t in range(n)]
            npar += n
            ladder = [ParamGate.fixed(O.cnot(q[i], q[i + 1])) for i in range(n - 1)]
            gates += layer + ladder if k else ladder + layer
        elif k < 6 or n == 1:
            p = npar if rng.random() < 0.8 or not npar else int(rng.integers(npar))
            npar = max(npar, p + 1)
            gates.append(make[int(rng.integers(3))](q[0], p))
        elif k == 6:
            gates.append(ParamGate.fixed(O.cnot(q[0], q[1])))
        elif k == 7:
            gates.append(ParamGate.fixed(O.hadamard(q[0])))
        elif k == 8:
            gates.append(ParamGate.fixed(O.not_(q[0]) if rng.random() < 0.5 else O.phase(q[0])))
        elif not batch:
            kind = int(rng.integers(3)) if n > 2 else 0
            gates.append(ParamGate.fixed((O.swap(q[0], q[1]), O.cnx(q[:2], q[2]) if n > 2 else None,
                                          O.to_controlled(O.ry(0.7, q[0]), q[1]))[kind]))
    if not unitary:
        gates.insert(m // 2, ParamGate.fixed(Operation(np.array([[1.0, 0.25], [0.5j, 0.75]]), [n // 2])))
    params = rng.uniform(0, 4 * math.pi, max(1, npar))
    special = rng.random(params.size)
    params[special < 0.1] = 0.0
    params[(special > 0.1) & (special < 0.2)] = math.pi
    terms = [(float(rng.normal()), int(rng.integers(1 << n)), int(rng.integers(1 << n))) for _ in range(4)]
    terms += [(float(rng.normal()), 0, 1 << (n - 1)), (float(rng.normal()), 1, 0)]
    return gates, params, terms


def _state(kind, n, rng):
    if kind == "basis":
        v = np.zeros(1 << n, dtype=complex)
        v[(1 << n) - 1] = 1.0
        return v
    v = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    if kind == "spread":
        v *= 10.0 ** rng.uniform(-12, 0, 1 << n)
        v[rng.random(1 << n) < 0.2] = 0.0
        v[0] += 1e-3
        return v * 37.0  # not normalised
    return v / np.linalg.norm(v)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["basis", "random", "spread"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 13])
def test_gradient_is_the_adjoint_walk(n, kind, precision):
    import quaru_gb300 as q

    for trial in range(2):
        rng = np.random.default_rng([n, len(kind), precision, trial])
        gates, params, terms = _circuit(n, 90, rng, False, unitary=trial == 0 or n > 8)
        psi = _state(kind, n, rng)
        if precision:
            psi = psi.astype(np.complex64).astype(complex)
        reg = q.Register.from_int(n, 0, precision=precision)
        reg.set_arith(q.QS_ARITH_FMA)
        reg.state = psi
        energy, grad = reg.adjoint_gradient(gates, params, terms)
        np.testing.assert_array_equal(reg.state, psi)
        e, g, scale = _reference(psi, n, gates, params, terms)
        tol = 24 * len(gates) * (2.0 ** -24 if precision else 2.0 ** -53) * scale
        assert abs(energy - e) <= tol
        assert np.max(np.abs(grad - g)) <= tol * max(1, np.max(np.bincount([x.param for x in gates if x.kind])))


@pytest.mark.parametrize("precision,arith", [(0, 1), (0, 2), (1, 1)])
@pytest.mark.parametrize("unitary", [True, False])
def test_batch_is_the_adjoint_walk(precision, arith, unitary):
    from quaru_gb300.batch import Batch

    rng = np.random.default_rng([7, precision, arith, unitary])
    circuits, params, want = [], [], []
    for n in (1, 2, 3, 5, 8, 9, 10, 11, 12, 13):
        gates, p, terms = _circuit(n, 70, rng, True, unitary or n % 2 == 1 or n > 11)
        circuits.append((n, gates, p.size, terms))
        params.append(p)
        psi = np.zeros(1 << n, dtype=complex)
        psi[0] = 1.0
        want.append((*_reference(psi, n, gates, p, terms), len(gates),
                     np.max(np.bincount([x.param for x in gates if x.kind]))))
    e, g = Batch(circuits, precision=precision, arith=arith, chunk_log2=11, ctas_per_sm=2).run(np.concatenate(params))
    at = 0
    for (we, wg, scale, m, shared), p, got in zip(want, params, e):
        # a double-float gate keeps 2^-47 of an amplitude
        tol = 24 * m * scale * (2.0 ** -24 if precision else 2.0 ** -47 if arith == 2 else 2.0 ** -53)
        assert abs(got - we) <= tol
        assert np.max(np.abs(g[at:at + p.size] - wg)) <= tol * shared
        at += p.size


def test_infinite_amplitudes_are_not_lost():
    """A state with an infinity or NaN has no finite energy or gradient, in fixed point either."""
    import quaru_gb300 as q

    rng = np.random.default_rng(3)
    for bad in (np.inf, np.nan):
        gates, params, terms = _circuit(9, 40, rng, False)
        reg = q.Register.from_int(9, 0)
        psi = _state("random", 9, rng)
        psi[17] = bad
        reg.state = psi
        energy, grad = reg.adjoint_gradient(gates, params, terms)
        assert not np.isfinite(energy)
        used = np.unique([x.param for x in gates if x.kind])
        assert not np.isfinite(grad[used]).any()
