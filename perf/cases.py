"""The workloads this engine's speed is measured on: what programs have it do, through its public
entry points, over the range of sizes, precisions, arithmetic forms and fusion options it offers.

Families (the "kind" of a case):
  calls     a program that applies one gate per call, reads the amplitudes and measures every qubit
            (the reference's own style of use): registers of a few to about fourteen qubits, where
            launches and calls are the cost
  circuit   a whole circuit in one call, then all qubits measured as one sequence: the layered
            random-circuit family (per layer a Haar-random gate on every qubit, then CNOTs on a random
            matching). Up to 22 qubits the program reads the amplitudes too; a larger state is only
            measured, as programs of that size do. A register is made per run, as there is no call
            that resets one.
  gradient  energy and adjoint gradient of a hardware-efficient ansatz (RY and RZ on every qubit, then
            a CNOT ladder, per layer): the forward and the reverse sweep of one optimiser step
  batch     the same for many circuits of uneven size in one call

Complex64 registers hold 32-bit amplitudes, so what a program keeps of them is 32-bit numbers.
"""
import math

import numpy as np
import torch

C128, C64 = 0, 1                       # QS_PREC_*
EXACT, FMA, DF64, FX64 = 0, 1, 2, 3    # QS_ARITH_*
READ_STATE_MAX = 22                    # largest register whose amplitudes a program reads back


def listed():
    return [
        # The 12-qubit, 200-gate circuit over the whole gate set, one call per gate, default arithmetic.
        {"name": "calls_12q", "kind": "calls", "n": 12, "gates": 200},
        # A mid-size circuit in one call with every option at its default (the reference's arithmetic,
        # one sweep per gate); amplitudes read, then measured in the reference's summation order.
        {"name": "circuit_19q_exact", "kind": "circuit", "n": 19, "gates": 224, "prec": C128, "arith": EXACT, "fuse": 0},
        # A large state with every option at its default: the dense sweeps in the reference's order.
        {"name": "circuit_27q_exact", "kind": "circuit", "n": 27, "gates": 40, "prec": C128, "arith": EXACT, "fuse": 0},
        # The 28-qubit layered circuit in plain FP64, one sweep per gate.
        {"name": "circuit_28q_fp64", "kind": "circuit", "n": 28, "gates": 84, "prec": C128, "arith": FMA, "fuse": 0},
        # The same size with 5-qubit blocks in the FP64-accurate fixed-point form.
        {"name": "circuit_28q_blocks", "kind": "circuit", "n": 28, "gates": 420, "prec": C128, "arith": FX64, "fuse": 2},
        # The mixed-precision form at 30 qubits: complex64 state, 5-qubit 3xTF32 blocks.
        {"name": "circuit_30q_c64_blocks", "kind": "circuit", "n": 30, "gates": 180, "prec": C64, "arith": FMA, "fuse": 2},
        # Complex64 with cache-blocked stages, which keep every gate's own arithmetic; an odd size.
        {"name": "circuit_27q_c64_stages", "kind": "circuit", "n": 27, "gates": 320, "prec": C64, "arith": FMA, "fuse": 1},
        # An optimiser step on a small problem: 8 qubits, 4 layers.
        {"name": "gradient_8q", "kind": "gradient", "n": 8, "layers": 4, "prec": C128, "arith": FMA},
        # The 20-qubit, 400-parameter ansatz in FP64 and in the mixed-precision form.
        {"name": "gradient_20q_fp64", "kind": "gradient", "n": 20, "layers": 10, "prec": C128, "arith": FMA},
        {"name": "gradient_20q_c64", "kind": "gradient", "n": 20, "layers": 10, "prec": C64, "arith": FMA},
        # Batches of ansatz circuits of uneven size (10 to 22 qubits, 4 to 12 layers), both precisions.
        {"name": "batch_fp64", "kind": "batch", "count": 64, "qmin": 10, "qmax": 22, "lmin": 4, "lmax": 12, "prec": C128, "arith": FMA},
        {"name": "batch_c64", "kind": "batch", "count": 128, "qmin": 10, "qmax": 22, "lmin": 4, "lmax": 12, "prec": C64, "arith": FMA},
    ]


def draw(rng):
    kind = rng.choice(["calls", "circuit", "circuit", "circuit", "gradient", "gradient", "batch"])
    if kind == "calls":
        return {"kind": kind, "n": rng.randint(3, 14), "gates": int(round(20 * 15 ** rng.random()))}
    prec = rng.choice([C128, C128, C64])
    arith = rng.choice([EXACT, FMA, DF64, FX64]) if prec == C128 else FMA
    if kind == "circuit":
        n = rng.randint(13, 28)
        fuse = rng.choice([0, 0, 1, 2])
        # so that no circuit takes longer than the longest listed one
        gates = rng.randint(30, max(60, 600 >> max(0, n - 22)))
        return {"kind": kind, "n": n, "gates": gates, "prec": prec, "arith": arith, "fuse": fuse}
    if arith == EXACT:
        arith = FMA
    if kind == "gradient":
        return {"kind": kind, "n": rng.randint(3, 21), "layers": rng.randint(1, 12), "prec": prec, "arith": arith}
    qmin = rng.randint(4, 14)
    lmin = rng.randint(1, 6)
    return {"kind": kind, "count": int(round(4 * 16 ** rng.random())), "qmin": qmin, "qmax": qmin + rng.randint(0, 20 - qmin),
            "lmin": lmin, "lmax": lmin + rng.randint(0, 6), "prec": prec, "arith": arith}


# ---------------------------------------------------------------- inputs, from the seed alone
def _haar(rng):
    z = rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2))
    q, r = np.linalg.qr(z)
    d = np.diagonal(r)
    return np.ascontiguousarray(q * (d / np.abs(d)))


_X = np.array([[0, 1], [1, 0]], dtype=np.complex128)
_CNOT = np.array([[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, 0, 1], [0, 0, 1, 0]], dtype=np.complex128)  # targets [target, control]
_SWAP = np.array([[1, 0, 0, 0], [0, 0, 1, 0], [0, 1, 0, 0], [0, 0, 0, 1]], dtype=np.complex128)


def _gates(case, seed):
    """The circuit as plain (matrix, targets) pairs and one uniform draw per qubit."""
    rng = np.random.default_rng([seed, case["n"]])
    n, gates = case["n"], []
    if case["kind"] == "calls":  # uniform over H, X, Y, Z, phase, CNOT, SWAP, Toffoli and Haar gates
        toffoli = np.eye(8, dtype=np.complex128)
        toffoli[6:, 6:] = _X
        for _ in range(case["gates"]):
            k = int(rng.integers(9))
            t = [int(x) for x in rng.permutation(n)[:3]]
            if k == 0:
                gates.append((np.array([[1, 1], [1, -1]], dtype=np.complex128) * 0.7071067811865476, t[:1]))
            elif k == 1:
                gates.append((_X, t[:1]))
            elif k == 2:
                gates.append((np.array([[0, -1j], [1j, 0]]), t[:1]))
            elif k == 3:
                gates.append((np.diag([1.0 + 0j, -1.0]), t[:1]))
            elif k == 4:
                gates.append((np.diag([1.0 + 0j, np.exp(2j * math.pi * rng.random())]), t[:1]))
            elif k == 5:
                gates.append((_CNOT, t[:2]))
            elif k == 6:
                gates.append((_SWAP, t[:2]))
            elif k == 7:
                gates.append((toffoli, t[:3]))
            else:
                gates.append((_haar(rng), t[:1]))
    else:
        while len(gates) < case["gates"]:  # layers; the last one may be cut short
            gates += [(_haar(rng), [q]) for q in range(n)]
            p = [int(x) for x in rng.permutation(n)]
            gates += [(_CNOT, [p[2 * i], p[2 * i + 1]]) for i in range(n // 2)]
    return gates[:case["gates"]], rng.random(n)


def _ansatz(n, layers):
    """The ansatz as ("ry" or "rz", qubit, parameter) and ("cx", control, target) steps."""
    steps, p = [], 0
    for _ in range(layers):
        for axis in ("ry", "rz"):
            for q in range(n):
                steps.append((axis, q, p))
                p += 1
        steps += [("cx", q, q + 1) for q in range(n - 1)]
    return steps, p


def _problem(case, seed):
    """(n, layers, parameters, terms) of each ansatz of a case; terms are (coefficient, x mask, z mask).
    The sizes of a batch belong to the case, the parameters and observables to the seed."""
    rng = np.random.default_rng([seed, 77])
    if case["kind"] == "gradient":
        shapes = [(case["n"], case["layers"])]
    else:
        r = np.random.default_rng([case["count"], case["qmin"], case["qmax"]])
        shapes = [(int(r.integers(case["qmin"], case["qmax"] + 1)), int(r.integers(case["lmin"], case["lmax"] + 1)))
                  for _ in range(case["count"])]
    out = []
    for n, layers in shapes:
        terms = []
        if case["kind"] == "gradient":  # sum_i a_i Z_i Z_{i+1} + sum_i b_i X_i
            terms += [(float(rng.normal()), 0, 3 << i) for i in range(n - 1)]
            terms += [(float(rng.normal()), 1 << i, 0) for i in range(n)]
        else:                           # n random Z, ZZ and X terms
            for _ in range(n):
                k, a, b = int(rng.integers(3)), int(rng.integers(n)), int(rng.integers(1, n))
                z = (0, 1 << a, (1 << a) | (1 << ((a + b) % n)))[k]
                terms.append((float(rng.normal()), 0 if k else 1 << a, z))
        out.append((n, layers, 2.0 * math.pi * rng.random(2 * n * layers), terms))
    return out


def _param_gates(n, layers):
    import quaru_gb300 as q
    from quaru_gb300 import operation as O

    steps, _ = _ansatz(n, layers)
    return [q.ParamGate.ry(a, b) if s == "ry" else q.ParamGate.rz(a, b) if s == "rz" else q.ParamGate.fixed(O.cnot(a, b))
            for s, a, b in steps]


def prepare(case, seed):
    import quaru_gb300 as q

    if case["kind"] in ("calls", "circuit"):
        gates, draws = _gates(case, seed)
        return {"case": case, "ops": [q.Operation(m, t) for m, t in gates], "draws": [float(x) for x in draws]}
    problem = _problem(case, seed)
    if case["kind"] == "gradient":
        n, layers, params, terms = problem[0]
        reg = q.Register.from_int(n, 0, case["prec"])
        reg.set_arith(case["arith"])
        return {"case": case, "reg": reg, "circuit": q.ParamCircuit(_param_gates(n, layers)), "params": params, "terms": q.PauliSum(terms)}
    from quaru_gb300.batch import Batch

    circuits = [(n, _param_gates(n, layers), len(params), terms) for n, layers, params, terms in problem]
    # the work-item size and the CTAs per SM that the tuner picks for such batches, given so that every
    # run is the same program
    chunk, ctas = (14, 4) if case["prec"] == C64 else (12, 3)
    batch = Batch(circuits, precision=case["prec"], chunk_log2=chunk, ctas_per_sm=ctas, arith=case["arith"])
    return {"case": case, "batch": batch, "params": np.concatenate([p for _, _, p, _ in problem])}


def _kept(case, x):
    x = np.asarray(x)
    if case["prec"] == C64 and x.dtype.kind in "fc":
        x = x.astype(np.complex64 if x.dtype.kind == "c" else np.float32)
    return x


def run(state):
    import quaru_gb300 as q

    case = state["case"]
    kind = case["kind"]
    if kind == "calls":
        reg = q.Register.from_int(case["n"], 0)
        for op in state["ops"]:
            reg.apply(op)
        amplitudes = reg.state
        outcomes, probs = [], []
        for t, draw_ in enumerate(state["draws"]):
            outcomes.append(reg.measure(t, draw_))
            probs.append(reg.last_probs)
        return {"state": amplitudes, "outcomes": np.array(outcomes, dtype=np.int64), "probs": np.array(probs)}
    if kind == "circuit":
        n, c64 = case["n"], case["prec"] == C64
        reg = q.Register.from_int(n, 0, case["prec"])
        reg.set_arith(case["arith"])
        opts = {"fuse": case["fuse"]}
        if case["fuse"] == 1:    # the documented tile size, not a tuned one
            opts["tile_qubits"] = min(12 if c64 else 11, max(9 if c64 else 8, n - 7))
        elif case["fuse"] == 2:  # the documented block width
            opts["max_width"] = 5 if c64 or case["arith"] == FX64 else 3 if case["arith"] == DF64 else 2
        reg.apply_gates(state["ops"], **opts)
        out = {"state": _kept(case, reg.state)} if n <= READ_STATE_MAX else {}
        out["outcomes"] = np.array(reg.measure_sequence(range(n), state["draws"]), dtype=np.int64)
        out["probs"] = _kept(case, reg.last_sequence_probs)
        return out
    if kind == "gradient":
        energy, grad = state["reg"].adjoint_gradient(state["circuit"], state["params"], state["terms"])
    else:
        energy, grad = state["batch"].run(state["params"])
    return {"energy": _kept(case, energy), "grad": _kept(case, grad)}


def work(case):
    """Bytes: each sweep that the caller asks for reads and writes the amplitudes it changes (one sweep
    per gate with fuse 0; one for the whole circuit otherwise), a measurement reads the state once.
    Flops: of the gates' real arithmetic."""
    if case["kind"] in ("calls", "circuit"):
        n = case["n"]
        N, amp = 2.0 ** n, 8 if case.get("prec") == C64 else 16
        if case["kind"] == "calls":   # on average half of the gates are 1-qubit dense or diagonal ones
            return {"bytes": N * amp * (2 * 0.75 * case["gates"] + 2), "flops": N * (5 * case["gates"] + 4 * n)}
        whole, left = divmod(case["gates"], n + n // 2)
        dense = whole * n + min(left, n)
        cnots = case["gates"] - dense
        sweeps = dense + 0.5 * cnots if case["fuse"] == 0 else 1  # a CNOT changes half of the amplitudes
        return {"bytes": N * amp * (2 * sweeps + 2), "flops": N * (14 * dense + 8)}
    flops = nbytes = 0.0
    for n, layers, params, terms in _problem(case, 0):
        # a rotation: 6 operations per amplitude, once forward and twice backward, and 4 for its inner product
        flops += 2.0 ** n * (22.0 * len(params) + 4.0 * len(terms) + 4)
        nbytes += (8 if case["prec"] == C64 else 16) * 2.0 ** n + 16.0 * len(params)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------- the same in 64 bits, by plain torch
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _basis(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device=_device())
    psi[0] = 1.0
    return psi


def _apply(psi, n, m, targets):
    if m is _CNOT:
        t, c = targets
        v = psi.view([2] * n)
        at = [slice(None)] * n
        at[n - 1 - c] = 1
        v = v[tuple(at)]                       # the control's half; the target's axis moves by one above it
        axis = n - 1 - t - (1 if t < c else 0)
        a, b = v.select(axis, 0), v.select(axis, 1)
        keep = a.clone()
        a.copy_(b)
        b.copy_(keep)
        return psi
    if len(targets) == 1:
        v = psi.view(1 << (n - 1 - targets[0]), 2, 1 << targets[0])
        a, b = v[:, 0], v[:, 1]
        new = a * complex(m[0, 0])
        new.add_(b, alpha=complex(m[0, 1]))
        b.mul_(complex(m[1, 1])).add_(a, alpha=complex(m[1, 0]))
        a.copy_(new)
        return psi
    k = len(targets)
    axes = [n - 1 - t for t in reversed(targets)]  # the matrix index's highest bit first
    rest = [a for a in range(n) if a not in axes]
    v = psi.view([2] * n).permute(axes + rest).reshape(1 << k, -1)
    v = torch.as_tensor(m, dtype=torch.complex128, device=psi.device) @ v
    back = [0] * n
    for i, a in enumerate(axes + rest):
        back[a] = i
    return v.reshape([2] * n).permute(back).reshape(-1).contiguous()


def _exact_circuit(case, seed):
    gates, draws = _gates(case, seed)
    n = case["n"]
    psi = _basis(n)
    for m, t in gates:
        psi = _apply(psi, n, m, t)
    out = {}
    if case["kind"] == "calls" or n <= READ_STATE_MAX:
        out["state"] = psi.cpu().numpy()
    p = torch.view_as_real(psi).square().sum(-1)
    del psi
    outcomes, probs = [], []
    for q in range(n):  # qubit 0 first: the lowest index bit of what is left
        v = p.view(-1, 2)
        p0, p1 = float(v[:, 0].sum()), float(v[:, 1].sum())
        one = draws[q] > p0
        outcomes.append(bool(one))
        probs.append((p0, p1))
        p = (v[:, 1] if one else v[:, 0]) / (p1 if one else p0)
    out["outcomes"] = np.array(outcomes, dtype=np.int64)
    out["probs"] = np.array(probs)
    return out


def _signs(n, mask):
    i = torch.arange(1 << n, device=_device())
    x = i & mask
    for s in (16, 8, 4, 2, 1):
        x = x ^ (x >> s)
    return 1.0 - 2.0 * (x & 1).double()


def _exact_gradient(n, layers, params, terms):
    steps, _ = _ansatz(n, layers)

    def rotate(psi, axis, q, theta):
        c, s = math.cos(theta / 2), math.sin(theta / 2)
        v = psi.view(1 << (n - 1 - q), 2, 1 << q)
        if axis == "rz":
            v[:, 0].mul_(complex(c, -s))
            v[:, 1].mul_(complex(c, s))
        else:
            a = v[:, 0].clone()
            v[:, 0].mul_(c).sub_(v[:, 1], alpha=s)
            v[:, 1].mul_(c).add_(a, alpha=s)

    psi = _basis(n)
    for s, a, b in steps:
        if s == "cx":
            _apply(psi, n, _CNOT, [b, a])
        else:
            rotate(psi, s, a, params[b])
    lam = torch.zeros_like(psi)
    diagonal = torch.zeros(1 << n, dtype=torch.float64, device=psi.device)
    for c, x, z in terms:
        if x == 0:
            diagonal += c * _signs(n, z)
        else:  # X on one qubit
            q = x.bit_length() - 1
            lam.view(-1, 2, 1 << q).add_(psi.view(-1, 2, 1 << q).flip(1), alpha=c)
    lam += diagonal * psi
    energy = (torch.view_as_real(psi) * torch.view_as_real(lam)).sum()
    got = []
    for s, a, b in reversed(steps):
        if s == "cx":
            _apply(psi, n, _CNOT, [b, a])
            _apply(lam, n, _CNOT, [b, a])
            continue
        if s == "rz":  # Im<lambda|Z|psi>
            w = (lam.real * psi.imag - lam.imag * psi.real).view(-1, 2, 1 << a)
            got.append((b, w[:, 0].sum() - w[:, 1].sum()))
        else:          # Im<lambda|Y|psi>
            p, l = torch.view_as_real(psi).view(-1, 2, 2 << a), torch.view_as_real(lam).view(-1, 2, 2 << a)
            got.append((b, (l[:, 1] * p[:, 0]).sum() - (l[:, 0] * p[:, 1]).sum()))
        rotate(psi, s, a, -params[b])
        rotate(lam, s, a, -params[b])
    grad = np.zeros(len(params))
    values = torch.stack([v for _, v in got]).cpu().numpy()
    for (b, _), v in zip(got, values):
        grad[b] += v
    return float(energy), grad


def exact(case, seed):
    if case["kind"] in ("calls", "circuit"):
        return _exact_circuit(case, seed)
    got = [_exact_gradient(*p) for p in _problem(case, seed)]
    if case["kind"] == "gradient":
        return {"energy": np.asarray(got[0][0]), "grad": got[0][1]}
    return {"energy": np.array([e for e, _ in got]), "grad": np.concatenate([g for _, g in got])}
