"""Operand images of complex128 tensor-core blocks, built on the device from the blocks' matrices.

Bar: a block applied to a basis vector is a column of its matrix to within the product's own bound: eight units of
X.Y / 2^60, where the input 1 is X = 2^54 and the output component's largest entry is Y >= 2^53 (2^-44 of that
entry), and roundings below 2^-52 of it. Rows of every scale, zero rows, entries that round up to the next digit
and entries far below their row's largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["unitary", "scales", "digits", "sparse"])
@pytest.mark.parametrize("targets", [[0, 1, 2, 3, 4], [11, 2, 7, 0, 9]])
def test_columns_of_a_block(kind, targets):
    import quaru_gb300 as q

    n = 12
    rng = np.random.default_rng([len(kind), targets[0]])
    m = rng.normal(size=(32, 32)) + 1j * rng.normal(size=(32, 32))
    if kind == "unitary":
        m = np.linalg.qr(m)[0]
    elif kind == "scales":
        m *= np.ldexp(1.0, rng.integers(-300, 300, 32))[:, None]
        m *= np.ldexp(1.0, rng.integers(-70, 1, (32, 32)))
    elif kind == "digits":  # 2 - 2^-52, halves of a digit, powers of two, both signs
        pick = np.array([2 - 2.0 ** -52, 1 + 2.0 ** -9, 2.0 ** -7 * (1 - 2.0 ** -53), 1.0, 0.5, 0.0])
        m = rng.choice(pick, (32, 32)) * rng.choice([-1, 1], (32, 32)) + 1j * rng.choice(pick, (32, 32))
    else:
        m = np.where(rng.random((32, 32)) < 0.1, m, 0.0)
        m[5] = 0.0
    top = np.maximum(np.abs(m.real), np.abs(m.imag)).max(axis=1)
    for j in (0, 13, 31):
        start = sum((j >> b & 1) << t for b, t in enumerate(targets))
        g = q.Register.from_int(n, start)
        g.set_arith(q.QS_ARITH_FX64)
        g.apply_gates([q.Operation(m, targets)], fuse=2)
        st = g.state
        rows = np.array([sum((i >> b & 1) << t for b, t in enumerate(targets)) for i in range(32)])
        off = st[rows] - m[:, j]
        assert np.all(np.maximum(np.abs(off.real), np.abs(off.imag)) <= top * (2.0 ** -44 + 2.0 ** -52)), j
        st[rows] = 0.0
        assert not st.any()
