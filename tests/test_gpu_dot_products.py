"""Dense complex one-qubit gates in FMA arithmetic on registers of 17 qubits and more: sums of four products as one
integer.

Bar: where the pair's non-zero components lie within 2^17 of the largest (exponent fields 300 to 1699),
each output is within 2^-53 of itself plus 2^-54 of its largest product; any other pair, and any other
matrix, keeps the bound of the FMA chain, four roundings of the terms' magnitudes. Inputs at the edges:
17 and 18 binades apart, the first and last exponents, both zeros, all-ones significands, products that
cancel, coefficients that are integers at 2^-60 of the
largest one's binade, down to the last, and one that is not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
L = np.longdouble


def _state(rng, n, span):
    N = 2 << n
    v = rng.uniform(1.0, 2.0, N) * rng.choice([-1.0, 1.0], N)
    v = np.where(rng.random(N) < 0.1, np.copysign(2.0 - 2.0 ** -52, v), v)
    v = np.ldexp(v, rng.integers(-span, 1, N)) if span else v
    v = np.where(rng.random(N) < 0.1, np.copysign(0.0, v), v)
    return v.view(np.complex128)


def _matrix(rng, kind):
    z = rng.normal(size=(2, 2)) + 1j * rng.normal(size=(2, 2))
    if kind == "haar":
        return np.linalg.qr(z)[0]
    if kind == "rx":
        return np.array([[0.6, -0.8j], [-0.8j, 0.6]])
    a = 1.0 - 2.0 ** -53
    if kind == "small":  # parts at 2^-8: the last that fit for every significand
        return np.array([[a, 2.0 ** -8 * (1 + 2.0 ** -52)], [2.0 ** -8 * (2 - 2.0 ** -52) * 1j, -a + 2.0 ** -8 * 1j]])
    if kind == "below":  # one that does not
        return np.array([[a, 2.0 ** -9 * (1 + 2.0 ** -52)], [0.5j, -a]])
    if kind == "cancel":
        return np.array([[0.5 + 0.5j, 0.5 + 0.5j], [0.5 - 0.5j, -0.5 + 0.5j]])
    return 2.0 ** 40 * z  # large


def _fits(m):
    parts = m.view(np.float64).ravel()
    scaled = np.ldexp(parts, 60 - int(np.frexp(np.abs(parts).max())[1]))
    return bool(np.all(scaled == np.floor(scaled)))


@pytest.mark.parametrize("kind", ["haar", "rx", "small", "below", "cancel", "large"])
@pytest.mark.parametrize("span,shift", [(0, 0), (4, 0), (17, 0), (18, 0), (60, 0), (3, 676), (3, 677), (0, -723), (0, -724)])
@pytest.mark.parametrize("n,t,control", [(17, 0, None), (17, 3, None), (17, 16, 2), (18, 0, 17)])
def test_outputs_are_sums_rounded_once(n, t, control, span, shift, kind):
    import quaru_gb300 as q
    from quaru_gb300 import operation as O

    rng = np.random.default_rng([n, t, span, abs(shift), len(kind)])
    m = _matrix(rng, kind)
    assert kind in ("haar", "large") or _fits(m) == (kind != "below")
    s = _state(rng, n, span)
    if kind == "cancel":
        i = np.arange(1 << n)
        lo = i[i >> t & 1 == 0]
        s[lo | 1 << t] = s[lo] * rng.choice([1.0, -1.0, 1.0 + 2.0 ** -52], lo.size)
    s = np.ldexp(s.view(np.float64), shift).view(np.complex128)
    g = q.Register.from_int(n, 0)
    g.set_arith(q.QS_ARITH_FMA)
    g.state = s
    op = q.Operation(m, [t])
    g.try_apply_fast(op if control is None else O.to_controlled(op, control))
    got = g.state
    i = np.arange(1 << n)
    i = i[(i >> t & 1) == 0]
    if control is not None:
        i = i[(i >> control & 1) == 1]
    rest = np.setdiff1d(np.arange(1 << n), np.concatenate([i, i | 1 << t]))
    np.testing.assert_array_equal(got[rest].view(np.float64), s[rest].view(np.float64))
    i = np.concatenate([i[:64], i[-64:], rng.choice(i, 2000)])
    x = [s[i].real, s[i].imag, s[i | 1 << t].real, s[i | 1 << t].imag]
    expo = np.array([np.where(v == 0.0, -5000, np.frexp(v)[1] + 1022) for v in x])
    E = expo.max(axis=0)
    integer = (E >= 300) & (E < 1700) & np.all((expo >= E - 17) | (expo == -5000), axis=0) & _fits(m)
    x = [v.astype(L) for v in x]
    for r in (0, 1):
        out = got[i | (r << t)]
        ar, ai, br, bi = (L(v) for v in (m[r, 0].real, m[r, 0].imag, m[r, 1].real, m[r, 1].imag))
        for part, c in (("real", (ar, -ai, br, -bi)), ("imag", (ai, ar, bi, br))):
            terms = [c[0] * x[0], c[1] * x[1], c[2] * x[2], c[3] * x[3]]
            want = terms[0] + terms[1] + terms[2] + terms[3]
            mags = np.abs(np.array(terms))
            # the reference itself: extended products and sums, at least 64 bits
            room = np.where(integer, np.abs(want) * L(2.0 ** -53) + mags.max(axis=0) * L(2.0 ** -54),
                            mags.sum(axis=0) * L(2.0 ** -51)) + mags.sum(axis=0) * L(2.0 ** -61)
            off = np.abs(getattr(out, part).astype(L) - want)
            assert np.all(off <= room), (part, r)


def test_values_do_not_depend_on_what_is_known_of_the_state():
    """The register's size decides the form, not how much of it a gate has to visit."""
    import quaru_gb300 as q

    rng = np.random.default_rng(5)
    for n in (16, 17, 19):
        a, b = q.Register.from_int(n, 3), q.Register.from_int(n, 3)
        b.state = a.state
        ops = [q.Operation(_matrix(rng, "haar"), [int(t)]) for t in rng.permutation(n)[:6]] * 2
        for r in (a, b):
            r.set_arith(q.QS_ARITH_FMA)
            r.apply_gates(ops, fuse=0)
        np.testing.assert_array_equal(a.state, b.state)


@pytest.mark.parametrize("k", [7, 8, 9, 20, 24, 25, 30, 39, 40, 49, 58, 59])
@pytest.mark.parametrize("full", [False, True])
def test_small_parts_with_few_bits(full, k):
    """Parts far below the largest that are integers at 2^-60 all the same: an output that only such parts feed keeps
    the bound of the integer sums (see above). RX by 2^(1 - k) and a row of small parts, on pairs whose other
    components are zero, or none of them."""
    import quaru_gb300 as q

    n, t, e = 17, 4, 2.0 ** -k
    rng = np.random.default_rng([k, full])
    for m in (np.array([[1.0, -1j * e], [-1j * e, 1.0]]), np.array([[1.0, 0.5], [e + e * 1j, e - 1j * e]])):
        s = _state(rng, n, 17)
        if not full:
            s[rng.random(s.size) < 0.5] = 0.0
        g = q.Register.from_int(n, 0)
        g.set_arith(q.QS_ARITH_FMA)
        g.state = s
        g.try_apply_fast(q.Operation(m, [t]))
        got = g.state
        i = np.arange(1 << n)
        i = i[(i >> t & 1) == 0]
        a, b = s[i], s[i | 1 << t]
        x = [v.astype(L) for v in (a.real, a.imag, b.real, b.imag)]
        for r in (0, 1):
            out = got[i | (r << t)]
            ar, ai, br, bi = (L(v) for v in (m[r, 0].real, m[r, 0].imag, m[r, 1].real, m[r, 1].imag))
            for part, c in (("real", (ar, -ai, br, -bi)), ("imag", (ai, ar, bi, br))):
                terms = np.array([c[0] * x[0], c[1] * x[1], c[2] * x[2], c[3] * x[3]])
                want = terms.sum(axis=0)
                mags = np.abs(terms)
                # four roundings of the chain, and the reference's own
                room = mags.sum(axis=0) * L(2.0 ** -51 + 2.0 ** -61)
                assert np.all(np.abs(getattr(out, part).astype(L) - want) <= room), (part, r)
