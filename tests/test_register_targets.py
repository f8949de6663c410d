"""Targets of a gate call as the engine gets them, on a stand-in for the library's entry point (no GPU)."""
import numpy as np
import pytest


@pytest.fixture
def calls(monkeypatch):
    from quaru_gb300 import _lib

    got = []

    def apply(handle, matrix, rows, cols, targets, k, err):
        got.append(np.frombuffer(targets, dtype=np.uintp, count=k).tolist())
        return 0

    monkeypatch.setattr(_lib, "apply_at", apply)
    return got


@pytest.mark.parametrize("targets", [[2 ** 64], [2 ** 64 + 1], [0, 2 ** 65], [-1], [0, -2 ** 63], [2 ** 70] * 9])
def test_targets_outside_size_t_are_refused(calls, targets):
    from quaru_gb300 import Operation, Register

    with pytest.raises(OverflowError):
        Register(0).try_apply_fast(Operation(np.eye(1 << len(targets), dtype=complex), targets))
    assert not calls


@pytest.mark.parametrize("targets", [[0], [2 ** 64 - 1], [3, 1], [np.int64(4), np.uint8(2)], np.array([5, 6]), (7, 1)])
def test_targets_inside_size_t_pass(calls, targets):
    from quaru_gb300 import Operation, Register

    Register(0).try_apply_fast(Operation(np.eye(1 << len(targets), dtype=complex), targets))
    assert calls == [[int(t) for t in targets]]
