"""Dense blocks whose qubits are chosen by a search (fuse=2 on states of 128 MiB and more).

Bar: (1) on the CPU, the blocks' product equals gate-by-gate application within 1e-12 (the bound of the
plain fusion: some hundred FP64 products of unitary matrices), for gates of 0 to 6 qubits in any order and
every block width, and a layered circuit takes fewer blocks than first-come claiming; (2) on the GPU, at
the smallest registers that take the search, fused equals unfused within the bounds of the fused forms
(1e-12 complex128, 1e-4 complex64).
"""
from __future__ import annotations

import struct
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


def _unitary(rng, k):
    z = rng.normal(size=(1 << k, 1 << k)) + 1j * rng.normal(size=(1 << k, 1 << k))
    return np.linalg.qr(z)[0]


@pytest.fixture(scope="module")
def fusers():
    out = ROOT / "tests" / "cpp" / "_build"
    out.mkdir(exist_ok=True)
    exes = []
    for name in ("fuse_check", "fuse_search_check"):
        exe = out / f"{name}_s"
        subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(ROOT / "include"), str(ROOT / f"tests/cpp/{name}.cpp"),
                        str(ROOT / "quaru_gb300/csrc/qs_fuse.cpp"), "-o", str(exe)], check=True)
        exes.append(exe)
    return exes


def _fused(exe, n, W, ops, st):
    buf = bytearray(struct.pack("<3i", n, W, len(ops)))
    for u, t in ops:
        buf += struct.pack("<i", len(t)) + struct.pack(f"<{len(t)}i", *t)
        buf += np.ascontiguousarray(u, dtype=np.complex128).tobytes()
    r = subprocess.run([str(exe)], input=bytes(buf) + st.tobytes(), capture_output=True, check=True)
    return np.frombuffer(r.stdout[: 16 << n], dtype=np.complex128), struct.unpack("<i", r.stdout[16 << n:])[0]


def _apply(n, ops, st):
    s = st.copy()
    for u, t in ops:
        k = len(t)
        v = s.reshape((2,) * n)
        axes = [n - 1 - q for q in reversed(t)]  # target 0 is the matrix's lowest bit
        v = np.moveaxis(v, axes, range(k))
        shape = v.shape
        v = (u @ v.reshape(1 << k, -1)).reshape(shape)
        s = np.ascontiguousarray(np.moveaxis(v, range(k), axes)).reshape(-1)
    return s


@pytest.mark.parametrize("W", [2, 3, 4, 5])
@pytest.mark.parametrize("kinds", [(1, 2), (0, 1, 2, 3), (1, 2, 5, 6), (1,), (2,), (6,)])
def test_searched_blocks_reproduce_gate_by_gate(fusers, W, kinds):
    n = 9
    rng = np.random.default_rng(100 * W + len(kinds) + sum(kinds))
    ops = []
    for _ in range(40):
        k = int(rng.choice(kinds))
        ops.append((_unitary(rng, k), [int(x) for x in rng.permutation(n)[:k]]))
    st = rng.normal(size=1 << n) + 1j * rng.normal(size=1 << n)
    st /= np.linalg.norm(st)
    got, _ = _fused(fusers[1], n, W, ops, st)
    assert np.max(np.abs(got - _apply(n, ops, st))) < 1e-12


def test_search_takes_fewer_blocks_on_a_layered_circuit(fusers):
    from quaru_gb300.workloads import flatten, layered_circuit

    n = 12
    ops = [(g.matrix, list(g.targets)) for g in flatten(layered_circuit(n, 10, 3))]
    st = np.zeros(1 << n, dtype=np.complex128)
    st[0] = 1.0
    a, plain = _fused(fusers[0], n, 5, ops, st)
    b, searched = _fused(fusers[1], n, 5, ops, st)
    assert np.max(np.abs(a - b)) < 1e-12
    assert searched < plain


@pytest.mark.gpu
@pytest.mark.parametrize("n,precision,arith,tol", [(23, 0, 3, 1e-12), (24, 1, 1, 1e-4), (23, 0, 1, 1e-12)])
def test_searched_blocks_on_registers(n, precision, arith, tol):
    import quaru_gb300 as q
    from tests.fixtures import floored_rel_err
    from tests.test_gpu_fusion import mixed_circuit
    from quaru_gb300.workloads import flatten, layered_circuit

    ops = flatten(layered_circuit(n, 3, 5)) + mixed_circuit(np.random.default_rng(n), n, 30)
    regs = []
    for fuse in (0, 2):
        r = q.Register.from_int(n, 0, precision=precision)
        r.set_arith(1 if fuse == 0 else arith)
        r.apply_gates(ops, fuse=fuse)
        regs.append(r.state)
    assert floored_rel_err(regs[1], regs[0]) <= tol
