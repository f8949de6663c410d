"""Collapses of complex128 registers: the kept amplitudes as correctly rounded quotients from integers.

Bar: bit for bit the IEEE quotient of amplitude and sqrt(probability) (numpy's), for every arithmetic, over significands
at the edges (powers of two, all ones, those of the divisor, random), all exponents that give normal quotients,
subnormal amplitudes and quotients, zeros of both signs; the other half becomes +0."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 5, 13])
@pytest.mark.parametrize("scale", [0, -300, 300, -511, 500])
def test_kept_amplitudes_are_ieee_quotients(n, scale, arith):
    import quaru_gb300 as q

    rng = np.random.default_rng([n, abs(scale), arith])
    N = 2 << n
    mant = rng.choice(np.array([1.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 1.5]), N)
    v = np.where(rng.random(N) < 0.6, rng.uniform(1.0, 2.0, N), mant) * rng.choice([-1.0, 1.0], N)
    spread = rng.integers(-60, 1, N)
    spread = np.where(rng.random(N) < 0.05, -1100 - scale, spread)  # down to subnormals
    with np.errstate(under="ignore"):
        v = np.ldexp(v, scale + spread)
    v[rng.random(N) < 0.05] = 0.0
    v[rng.random(N) < 0.05] *= -0.0
    s = v.view(np.complex128)
    for target in sorted({0, n - 1}):
        for draw in (0.0, 1e300):  # mostly outcome 1, outcome 0
            g = q.Register.from_int(n, 0)
            g.set_arith(arith)
            g.state = s
            outcome = g.measure(target, draw)
            total = g.last_probs[outcome]
            live = (np.arange(1 << n) >> target & 1) == outcome
            out = g.state
            with np.errstate(all="ignore"):
                want = s[live].view(np.float64) / math.sqrt(total)
            np.testing.assert_array_equal(out[live].view(np.uint64), want.view(np.uint64))
            assert not out[~live].view(np.uint64).any()


@pytest.mark.parametrize("arith", [0, 1])
@pytest.mark.parametrize("top", [-1010, -1000, -980, -960, -930, -905])
def test_small_normal_amplitudes(top, arith):
    """Amplitudes whose remainder x - q d has bits below the subnormal range (from about 2^-968 down), beside one large
    amplitude that sets the divisor; enough of them to meet the quotients near the middle of two doubles."""
    import quaru_gb300 as q

    n = 18
    rng = np.random.default_rng([-top, arith])
    v = np.ldexp(rng.uniform(1.0, 2.0, 2 << n) * rng.choice([-1.0, 1.0], 2 << n), top - rng.integers(0, 12, 2 << n))
    v[0], v[1] = 0.7390851332151607, 0.0
    s = v.view(np.complex128)
    g = q.Register.from_int(n, 0)
    g.set_arith(arith)
    g.state = s
    assert not g.measure(n - 1, 0.0)
    d = math.sqrt(g.last_probs[0])
    assert 0.739 < d < 0.74
    want = s[:1 << (n - 1)].view(np.float64) / d
    np.testing.assert_array_equal(g.state[:1 << (n - 1)].view(np.float64).view(np.uint64), want.view(np.uint64))
