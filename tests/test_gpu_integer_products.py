"""Dense one-qubit gates whose products run on the integer pipes: the reference's amplitudes bit for bit,
and the FP64 FMA form within its own rounding, at the edges of what the integer form takes (zeros,
powers of two, significands that round up to the next binade, exponents inside and outside its range,
subnormal, infinite and NaN components; coefficients that are zero, tiny or huge)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _components(rng, N):
    """Components of every kind, mixed so that pairs meet in all combinations."""
    v = rng.standard_normal(N)
    k = rng.integers(0, 12, N)
    ones = np.ldexp(2.0 - 2.0 ** -52, rng.integers(-30, 3, N))           # all ones: carries
    v = np.where(k == 0, 0.0, v)
    v = np.where(k == 1, -0.0, v)
    v = np.where(k == 2, np.ldexp(1.0, rng.integers(-60, 60, N)), v)
    v = np.where(k == 3, ones, v)
    v = np.where(k == 4, v * np.ldexp(1.0, rng.integers(-1000, -700, N)), v)
    v = np.where(k == 5, v * np.ldexp(1.0, rng.integers(700, 900, N)), v)
    v = np.where(k == 6, np.ldexp(rng.integers(1, 9, N).astype(float), -1074), v)  # subnormal
    return v


def _state(rng, n, special):
    N = 1 << n
    s = _components(rng, N) + 1j * _components(rng, N)
    if special:
        s.real[rng.integers(N)] = np.inf
        s.imag[rng.integers(N)] = np.nan
    return s


def _matrices(rng):
    z = rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2))
    rx = np.array([[0.6, -0.8j], [-0.8j, 0.6]])                       # zero parts
    return {
        "haar": np.linalg.qr(z)[0],
        "rx": rx,
        "hadamard": np.array([[1, 1], [1, -1]]) * (0.7071067811865476 + 0j),
        "edge": np.array([[2.0 - 2.0 ** -52, -(1.0 + 2.0 ** -52)], [2.0 ** -99, 2.0 ** 99]]) + 0j,
        "complex_edge": np.array([[2.0 ** -100, 1j], [-3.0, 1 + 2.0 ** 99 * 1j]]),
        "outside": np.array([[2.0 ** -120, 1.0], [1.0, 2.0 ** 120]]) + 0.5j,
    }


def _gate(m, s, t, control):
    """m on qubit t of s, every product and sum rounded to double."""
    out = s.copy()
    i = np.arange(s.size)
    i = i[(i >> t & 1) == 0]
    if control is not None:
        i = i[(i >> control & 1) == 1]
    a, b = s[i], s[i | 1 << t]

    def times(c, x):
        if not m.imag.any():
            return c.real * x.real, c.real * x.imag
        return c.real * x.real - c.imag * x.imag, c.real * x.imag + c.imag * x.real

    for r, k in ((0, i), (1, i | 1 << t)):
        (pr, pi), (qr, qi) = times(m[r, 0], a), times(m[r, 1], b)
        out.real[k] = pr + qr
        out.imag[k] = pi + qi
    return out


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("kind", ["haar", "rx", "hadamard", "edge", "complex_edge", "outside"])
@pytest.mark.parametrize("n", [1, 2, 9, 14])
def test_exact_form_is_the_oracle(n, kind, special):
    import quaru_gb300 as q
    from quaru_gb300 import operation as O
    from oracle.oracle import OracleRegister

    rng = np.random.default_rng([n, len(kind), special])
    m = _matrices(rng)[kind]
    for t in sorted({0, n // 2, n - 1}):
        ops = [q.Operation(m, [t])]
        if n > 1:
            ops.append(O.to_controlled(q.Operation(m, [t]), (t + 1) % n))  # tuples with a fixed bit
        for op in ops:
            s = _state(rng, n, special)
            g, o = q.Register.from_int(n, 0), OracleRegister(s.copy(), n)
            g.state = s
            g.try_apply_fast(op)
            with np.errstate(all="ignore"):
                if special:
                    # the oracle multiplies an infinity by the gate's zeros (rows it leaves alone,
                    # imaginary parts of a real matrix), the engine has no such products
                    want = _gate(m, s, t, (t + 1) % n if len(op.targets) == 2 else None)
                else:
                    o.try_apply_fast(op.matrix, op.targets)
                    want = o.state
            np.testing.assert_array_equal(g.state.view(np.float64), want.view(np.float64))


@pytest.mark.parametrize("kind", ["haar", "rx", "hadamard", "edge", "complex_edge"])
@pytest.mark.parametrize("n", [1, 9])
def test_fma_form_within_its_rounding(n, kind):
    """Four roundings per output of partial sums no larger than the sum of the terms' magnitudes:
    within 4 * 2^-53 of it (plus a subnormal unit), checked in extended precision."""
    import quaru_gb300 as q

    rng = np.random.default_rng([n, len(kind), 9])
    m = _matrices(rng)[kind]
    for t in sorted({0, n - 1}):
        s = _state(rng, n, False)
        g = q.Register.from_int(n, 0)
        g.set_arith(q.QS_ARITH_FMA)
        g.state = s
        g.try_apply_fast(q.Operation(m, [t]))
        got = g.state.reshape(-1, 2, 1 << t)
        x = s.reshape(-1, 2, 1 << t)
        re, im = x.real.astype(np.longdouble), x.imag.astype(np.longdouble)
        for r in (0, 1):
            mr, mi = m[r].real.astype(np.longdouble), m[r].imag.astype(np.longdouble)
            terms = {"real": [mr[0] * re[:, 0], -mi[0] * im[:, 0], mr[1] * re[:, 1], -mi[1] * im[:, 1]],
                     "imag": [mr[0] * im[:, 0], mi[0] * re[:, 0], mr[1] * im[:, 1], mi[1] * re[:, 1]]}
            for part, ts in terms.items():
                off = np.abs(getattr(got[:, r], part) - sum(ts))
                room = sum(np.abs(v) for v in ts) * np.longdouble(2.0 ** -51 + 2.0 ** -60) + np.longdouble(2.0 ** -1072)
                assert np.all(off <= room)
