"""Probability sums in the reference's order (src/register.rs:306-315) are the sequential FP64 sums bit
for bit, whichever kernel takes the size: numpy's cumulative sum adds one element after another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(kind, n, rng):
    N = 1 << n
    v = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    if kind == "random":
        return v / np.linalg.norm(v)
    if kind == "ties":  # few significant bits: squares that end half an ulp past the running sum
        v = rng.integers(-3, 4, N) * 2.0 ** rng.integers(-28, -24, N) + 1j * rng.integers(-3, 4, N) * 2.0 ** -26
        v[0] = v[N // 2] = 1.0 + 2.0 ** -30
        return v
    if kind == "spread":  # thirty decades, zeros and subnormal squares between them
        v = v * 10.0 ** rng.uniform(-170, 2, N)
        v[rng.random(N) < 0.3] = 0.0
        return v
    if kind == "growing":  # a binade is left every few squares
        return v * 2.0 ** (np.arange(N) * (600.0 / N) - 300.0)
    if kind == "basis":
        v = np.zeros(N, dtype=complex)
        v[N - 1] = 1.0
        return v
    if kind == "infinite":
        v[N // 3] = np.inf
        return v
    v[N // 3] = np.nan
    return v


@pytest.mark.parametrize("kind", ["random", "ties", "spread", "growing", "basis", "infinite", "nan"])
@pytest.mark.parametrize("n", [1, 2, 7, 12, 13, 14, 15, 18, 20])
def test_sums_are_the_sequential_ones(n, kind):
    import quaru_gb300 as q

    rng = np.random.default_rng([n, len(kind)])
    v = _state(kind, n, rng)
    for target in sorted({0, n // 2, n - 1}):
        g = q.Register.from_int(n, 0)
        g.state = v
        g.measure(target, 0.0)
        with np.errstate(all="ignore"):
            s = (v.real * v.real + v.imag * v.imag).reshape(-1, 2, 1 << target)
            want = [float(np.add.accumulate(np.concatenate([[0.0], s[:, b].ravel()]))[-1]) for b in (0, 1)]
        np.testing.assert_array_equal(np.array(g.last_probs), np.array(want))
        if np.isfinite(want).all() and n > 1 and want[0] > 0:  # a second measurement, on what the first one left
            w = g.state
            other = (target + 1) % n
            g.measure(other, 0.0)
            s = (w.real * w.real + w.imag * w.imag).reshape(-1, 2, 1 << other)
            want = [float(np.add.accumulate(np.concatenate([[0.0], s[:, b].ravel()]))[-1]) for b in (0, 1)]
            np.testing.assert_array_equal(np.array(g.last_probs), np.array(want))
