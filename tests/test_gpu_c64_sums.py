"""Probability sums and collapses of complex64 registers on the integer and FP32 pipes.

Bar: (1) both probabilities of every target, on states whose magnitudes run over the whole float range
(zeros and subnormals included), agree with exactly rounded sums of the exact squares to 64 roundings of
2^-53 (at most 10 additions in a row per thread, lane, warp and block at these sizes, 13 binary orders of
partial sums to spare), also where one outcome is 2^-70 of the other; (2) collapsed amplitudes are the
float nearest to the amplitude times the double 1/sqrt(total) but for one in 2^-16 rounded ties (here
none may differ by more than one unit in the last place), with the sign of zeros kept; (3) infinities and
NaN give the non-finite sums that FP64 gives.
"""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(rng, n, kind):
    v = rng.normal(size=2 << n)
    if kind == "wide":
        v *= 2.0 ** rng.integers(-148, 60, size=v.size)
    elif kind == "mixed":
        v *= 2.0 ** rng.integers(-148, 1, size=v.size)
    elif kind == "tiny":
        v *= 2.0 ** rng.integers(-148, -90, size=v.size)
    elif kind == "rare":  # one outcome of target n - 1 far below the other
        v[1 << n:] *= 2.0 ** -35
    if kind != "normal":
        v[rng.random(v.size) < 0.2] = 0.0
        v[rng.random(v.size) < 0.1] *= -0.0
    return v.astype(np.float32)


def _register(n, f):
    import quaru_gb300 as q

    r = q.Register.from_int(n, 0, precision=1)
    r.state = (f.astype(np.float64)).view(np.complex128)
    return r


def _check_sums(got, f, target):
    sq = (f.astype(np.float64) ** 2).reshape(-1, 2)  # exact: 48 bits, and no square of a float underflows
    idx = np.arange(sq.shape[0])
    for b in (0, 1):
        want = math.fsum(sq[(idx >> target & 1) == b].ravel())
        assert abs(got[b] - want) <= 64 * 2.0 ** -53 * want, (target, b, got, want)


@pytest.mark.parametrize("kind", ["normal", "wide", "mixed", "tiny", "rare"])
@pytest.mark.parametrize("n", [1, 2, 9, 10, 11, 12, 13, 17])
def test_probability_sums_and_collapse(n, kind):
    f = _state(np.random.default_rng(n + 31 * len(kind)), n, kind)
    idx = np.arange(1 << n)
    for target in sorted({0, 1, 7, 8, 9, 10, n - 1}):
        if target >= n:
            continue
        r = _register(n, f)
        outcome = r.measure(target, 0.5)
        _check_sums(r.last_probs, f, target)
        total = r.last_probs[outcome]
        live = (idx >> target & 1) == outcome
        if total > 0.0:
            with np.errstate(under="ignore"):
                ref = (f.reshape(-1, 2)[live].astype(np.float64) * (1.0 / math.sqrt(total))).astype(np.float32)
            out = r.state.view(np.float64).astype(np.float32).reshape(-1, 2)
            ulp = np.spacing(np.abs(ref)).astype(np.float64)
            assert np.all(np.abs(out[live].astype(np.float64) - ref) <= ulp)
            assert np.array_equal(np.signbit(out[live]), np.signbit(ref))
            assert not out[~live].any()
        if n > 1 and total > 0.0:  # the sums that come with a collapse
            other = (target + 1 + n // 2) % n
            s = _register(n, f)
            s.measure_sequence([target, other], [0.5, 0.5])
            _check_sums(s.last_sequence_probs[1], out.ravel(), other)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_amplitudes(bad):
    n = 11
    f = _state(np.random.default_rng(1), n, "normal")
    f[2 * 700] = bad
    r = _register(n, f)
    r.measure(0, 0.5)
    p = r.last_probs
    assert (math.isnan(p[0]) if math.isnan(bad) else p[0] == math.inf) and math.isfinite(p[1])
