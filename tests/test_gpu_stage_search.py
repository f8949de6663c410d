"""Stages whose qubits are chosen by a search where that gives fewer (fuse=1 on states of 64 MiB and more).

Bar: the exact arithmetic stays bit-identical to single sweeps (the stages reorder commuting gates only), the other
forms stay within their fused bounds of it; ladders and rings of CNOTs, for which the search takes fewer stages
(one window runs several layers), and mixed gates, at the smallest register that searches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,arith,tol", [(0, 0, 0.0), (0, 1, 1e-12), (1, 1, 1e-4)])
@pytest.mark.parametrize("kind", ["ladder", "mixed"])
def test_searched_stages_equal_single_sweeps(kind, precision, arith, tol):
    import quaru_gb300 as q
    from quaru_gb300 import operation as O
    from tests.fixtures import floored_rel_err, value_equal
    from tests.test_gpu_fusion import mixed_circuit, rand_unitary

    n = 22 + precision
    rng = np.random.default_rng(n)
    if kind == "ladder":
        ops = []
        for _ in range(3):
            ops += [q.Operation(rand_unitary(rng, 1), [t]) for t in range(n)]
            ops += [O.cnot(t, (t + 1) % n) for t in range(n)]
    else:
        ops = mixed_circuit(rng, n, 60)
    states = []
    for fuse in (0, 1):
        r = q.Register.from_int(n, 5, precision=precision)
        r.set_arith(arith)
        r.apply_gates(ops, fuse=fuse, tile_qubits=0 if fuse == 0 else 11)
        states.append(r.state)
    if tol == 0.0:
        assert value_equal(states[1], states[0])
    else:
        assert floored_rel_err(states[1], states[0]) <= tol
