"""Fused blocks whose matrix has an infinity or NaN, on registers whose blocks run on the tensor cores: the amplitudes it
reaches are not finite, the others are those of the gate-by-gate form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,arith", [(0, 3), (1, 1)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, complex(0, -np.inf)])
@pytest.mark.parametrize("n", [12, 14, 17])
def test_not_finite_is_not_lost(n, bad, precision, arith):
    import quaru_gb300 as q
    from tests.test_gpu_fusion import rand_unitary

    rng = np.random.default_rng(n)
    ops = [q.Operation(rand_unitary(rng, 2), [1, 9]), q.Operation(rand_unitary(rng, 2), [4, 8])]
    m = rand_unitary(rng, 1).astype(complex)
    m[1, 1] = bad
    ops.append(q.Operation(m, [n - 1]))
    v = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    v /= np.linalg.norm(v)
    g = q.Register.from_int(n, 0, precision=precision)
    g.set_arith(arith)
    g.state = v
    g.apply_gates(ops, fuse=2, max_width=5)
    s = g.state
    top = np.arange(1 << n) >> (n - 1) & 1 == 1  # row 1 of the last gate
    assert not np.isfinite(s[top]).any()
    h = q.Register.from_int(n, 0, precision=precision)
    h.set_arith(1)
    h.state = v
    for op in ops:
        h.try_apply_fast(op)
    w = h.state
    # a block is one matrix: where it shares a qubit with the bad gate, zeros times its entry are NaN too
    ok = np.isfinite(s)
    np.testing.assert_allclose(s[ok], w[ok], atol=1e-6 if precision else 1e-13)
    if precision == 0:
        assert not np.isfinite(w[top]).any() and np.isfinite(w[~top]).all()
