// qs_sweep.cpp — host side of the gradient sweeps: builds the pass programs of qs_sweep.h.
#include "qs_sweep.h"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace qs {

namespace {

// An X, CNOT (control on 1 or 0) or SWAP as an affine index map: target ^= control (^ 1).
struct Move {
    int kind = 0;  // 0: none, 1: X / CNOT, 2: SWAP
    int target = 0, control = -1;
    bool on_zero = false;
};

Move as_move(const OpDesc& op) {
    Move m;
    if (op.kind != OP_MONO_PF) return m;
    if (op.k == 1 && op.perm[0] == 1 && op.perm[1] == 0 && op.pf[0] == PF_ONE && op.pf[1] == PF_ONE &&
        __builtin_popcountll(op.fixmask) <= 1) {
        m.kind = 1;
        m.target = op.tq[0];
        if (op.fixmask) {
            m.control = __builtin_ctzll(op.fixmask);
            m.on_zero = op.fixval == 0;
        }
    } else if (op.k == 2 && op.fixmask == 0 && op.perm[0] == 0 && op.perm[1] == 2 && op.perm[2] == 1 &&
               op.perm[3] == 3 && op.pf[0] == PF_SKIP && op.pf[1] == PF_ONE && op.pf[2] == PF_ONE &&
               op.pf[3] == PF_SKIP) {
        m.kind = 2;
        m.target = op.tq[0];
        m.control = op.tq[1];
    }
    return m;
}

struct Builder {
    const std::vector<SweepGate>& gates;
    const TileStage& st;
    std::vector<TileOp>* ops;
    int T, RB;
    std::vector<uint64_t> qm;
    std::vector<Move> mv;
    std::vector<int> left;  // gates not placed yet, in order

    bool fixed_point, reverse, ordered;

    Builder(const std::vector<SweepGate>& g, const TileStage& s, bool fx, bool rev, bool ord,
            std::vector<TileOp>* o)
        : gates(g), st(s), ops(o), fixed_point(fx), reverse(rev), ordered(ord) {
        T = st.T;
        RB = sw_register_bits(T);
        for (size_t i = 0; i < g.size(); i++) {
            uint64_t m = 0;
            Move v;
            if (g[i].axis) {
                m = 1ull << g[i].target;
            } else {
                m = g[i].fixed->fixmask;
                for (int j = 0; j < g[i].fixed->k; j++) m |= 1ull << g[i].fixed->tq[j];
                v = as_move(*g[i].fixed);
                if (g[i].fixed->kind == OP_NOOP) continue;  // an identity
            }
            qm.resize(i + 1, 0);
            mv.resize(i + 1);
            qm[i] = m;
            mv[i] = v;
            left.push_back(int(i));
        }
        qm.resize(g.size(), 0);
        mv.resize(g.size());
    }

    int local(int q) const {
        if (q < st.L) return q;
        for (size_t i = 0; i < st.high.size(); i++)
            if (st.high[i] == q) return st.L + int(i);
        return -1;
    }

    bool turn(int i) const { return gates[i].axis == QS_GATE_RX || gates[i].axis == QS_GATE_RY; }

    // The gates of a moves pass: with phase_first the RZ gates come before the moves.
    void collect_moves(bool phase_first, std::vector<int>* rz, std::vector<int>* moves) const {
        uint64_t blocked = 0, first = 0, second = 0;  // qubits of the earlier / the later half taken so far
        uint64_t outside = 0;
        rz->clear();
        moves->clear();
        for (int i : left) {
            const bool z = gates[i].axis == QS_GATE_RZ, m = mv[i].kind != 0;
            bool ok = (z || m) && !(qm[i] & blocked);
            const bool early = z == phase_first;  // belongs to the half that runs first
            if (ok && early && (qm[i] & second)) ok = false;
            if (ok && z && (qm[i] & (early ? first : second)))  // one RZ per qubit and pass
                for (int k : *rz) ok = ok && !(qm[k] & qm[i]);
            uint64_t out = 0;
            if (ok && m && mv[i].control >= 0 && local(mv[i].control) < 0) out = 1ull << mv[i].control;
            if (ok && __builtin_popcountll(outside | out) > kSwOutside) ok = false;
            if (!ok) {
                if (ordered) break;
                blocked |= qm[i];
                continue;
            }
            outside |= out;
            (early ? first : second) |= qm[i];
            (z ? rz : moves)->push_back(i);
        }
    }

    // The rotations of a pass: those that can run now on the lowest tile bits that have any.
    std::vector<int> collect_rotations(uint32_t* bits) const {
        uint64_t blocked = 0;
        std::vector<int> got;
        *bits = 0;
        for (int i : left) {
            if (turn(i) && !(qm[i] & blocked)) *bits |= 1u << local(gates[i].target);
            else if (ordered) break;
            else blocked |= qm[i];
            if (ordered && __builtin_popcount(*bits) == std::min(RB, T)) break;
        }
        uint32_t use = 0;
        for (uint32_t b = *bits; b && __builtin_popcount(use) < RB; b &= b - 1) use |= b & -b;
        blocked = 0;
        for (int i : left) {  // one per bit: a second one waits for the next pass
            if (turn(i) && !(qm[i] & blocked) && (use >> local(gates[i].target) & 1u)) got.push_back(i);
            else if (ordered) break;
            blocked |= qm[i];
        }
        *bits = use;
        return got;
    }

    void place(const std::vector<int>& g) {
        std::vector<int> rest;
        for (int i : left)
            if (std::find(g.begin(), g.end(), i) == g.end()) rest.push_back(i);
        left.swap(rest);
    }

    // Room in program p for nrot more rotations and (diag) one more factor table.
    static bool room(const SweepProgram& p, size_t nrot, bool diag) {
        return p.passes.size() < size_t(kSwMaxPass) && p.rots.size() + nrot <= size_t(kSwMaxRot) &&
               (!diag || p.ndiag < kSwMaxDiag);
    }

    static SweepPass blank() {
        SweepPass p;
        std::memset(&p, 0, sizeof(p));
        p.diag = -1;
        p.op = -1;
        for (int j = 0; j < 3; j++) p.rot[j] = -1;
        for (int b = 0; b < kSwMaxT; b++) {
            p.zrot[b] = -1;
            p.col[b] = uint16_t(1u << b);
        }
        return p;
    }

    std::vector<SweepProgram> run() {
        std::vector<SweepProgram> progs(1);
        while (!left.empty()) {
            uint32_t bits = 0;
            const std::vector<int> rot = collect_rotations(&bits);
            if (!rot.empty()) {
                if (!room(progs.back(), rot.size(), false)) progs.emplace_back();
                SweepProgram& P = progs.back();
                SweepPass p = blank();
                p.kind = SW_ROT;
                for (int b = T - 1; b >= 0 && __builtin_popcount(bits) < std::min(RB, T); b--) bits |= 1u << b;
                int pos[3] = {0, 0, 0}, np = 0, lo = 0;
                for (int b = 0; b < T; b++)
                    if (bits >> b & 1u) pos[np++] = b;
                for (int j = 0; j < np; j++) p.rbit[j] = uint8_t(pos[j]);
                for (int j = 0; j <= np; j++) {
                    const int hi = j < np ? pos[j] : T;
                    uint32_t m = 0;
                    for (int b = lo; b < hi; b++) m |= 1u << b;
                    p.seg[j] = m;
                    lo = hi + 1;
                }
                for (size_t k = 0; k < rot.size(); k++) {
                    const int lb = local(gates[rot[k]].target);
                    const int j = int(std::find(pos, pos + np, lb) - pos);
                    if (gates[rot[k]].axis == QS_GATE_RX) p.rx |= uint8_t(1 << j);
                    p.rot[j] = int8_t(P.rots.size());
                    P.rots.push_back(gates[rot[k]].gate);
                }
                P.passes.push_back(p);
                place(rot);
                continue;
            }
            std::vector<int> rz, moves, rz2, moves2;
            collect_moves(false, &rz, &moves);
            // inner products take the amplitudes behind the move by their own index, so the reverse walk
            // has its phases behind the move
            if (!reverse) collect_moves(true, &rz2, &moves2);
            const bool phase_first = rz2.size() + moves2.size() > rz.size() + moves.size();
            if (phase_first) {
                rz.swap(rz2);
                moves.swap(moves2);
            }
            if (!rz.empty() || !moves.empty()) {
                if (!room(progs.back(), rz.size(), !rz.empty())) progs.emplace_back();
                SweepProgram& P = progs.back();
                SweepPass p = blank();
                p.kind = SW_MOVE;
                p.phase_first = phase_first ? 1 : 0;
                p.moves = moves.empty() ? 0 : 1;
                if (!rz.empty()) p.diag = int8_t(P.ndiag++);
                for (int i : rz) {
                    p.zrot[local(gates[i].target)] = int8_t(P.rots.size());
                    P.rots.push_back(gates[i].gate);
                }
                // f = f_1 f_2 ... f_m for the moves in order: later moves act on the index first, so the
                // map is built from the last to the first. Row form: bit b of f(x) is the parity of
                // x & row[b], of the outside controls out[b], and a constant.
                std::vector<uint32_t> row(T);
                std::vector<uint64_t> out(T, 0);
                uint32_t flip = 0;
                for (int b = 0; b < T; b++) row[b] = 1u << b;
                for (size_t k = moves.size(); k-- > 0;) {
                    const Move& m = mv[moves[k]];
                    const int t = local(m.target);
                    if (m.kind == 2) {
                        const int c = local(m.control);
                        std::swap(row[t], row[c]);
                        std::swap(out[t], out[c]);
                        const uint32_t d = ((flip >> t) ^ (flip >> c)) & 1u;
                        flip ^= (d << t) | (d << c);
                    } else if (m.control < 0) {
                        flip ^= 1u << t;
                    } else {
                        const int c = local(m.control);
                        if (c >= 0) {
                            row[t] ^= row[c];
                            out[t] ^= out[c];
                            flip ^= ((flip >> c) & 1u) << t;
                        } else {
                            out[t] ^= 1ull << m.control;
                        }
                        if (m.on_zero) flip ^= 1u << t;
                    }
                }
                for (int b = 0; b < T; b++) {
                    p.col[b] = 0;
                    for (int r = 0; r < T; r++)
                        if (row[r] >> b & 1u) p.col[b] |= uint16_t(1u << r);
                }
                uint64_t seen = 0;
                for (int b = 0; b < T; b++) seen |= out[b];
                for (; seen; seen &= seen - 1) {
                    const int q = __builtin_ctzll(seen);
                    uint16_t m = 0;
                    for (int b = 0; b < T; b++)
                        if (out[b] >> q & 1ull) m |= uint16_t(1u << b);
                    p.oq[p.nout] = uint8_t(q);
                    p.om[p.nout++] = m;
                }
                p.flip = uint16_t(flip);
                P.passes.push_back(p);
                std::vector<int> all = rz;
                all.insert(all.end(), moves.begin(), moves.end());
                place(all);
                continue;
            }
            // a gate of neither kind runs on its own
            if (!room(progs.back(), 0, false)) progs.emplace_back();
            SweepPass p = blank();
            p.kind = SW_FIXED;
            p.op = int32_t(ops->size());
            TileOp t = make_tile_op(*gates[left[0]].fixed, st);
            if (fixed_point)  // the entries as limbs (FxLimb), where the double-float coefficients sit otherwise
                for (int i = 0; i < 16; i++) {
                    const long long C = std::llrint(t.m[i] * 0x1p60);
                    const long long l = (long long)((unsigned long long)C << 34) >> 34;
                    const int32_t lo = int32_t(l), hi = int32_t((C - l) >> 30);
                    std::memcpy(&t.dfh[i], &hi, 4);
                    std::memcpy(&t.dfl[i], &lo, 4);
                }
            ops->push_back(t);
            progs.back().passes.push_back(p);
            left.erase(left.begin());
        }
        if (progs.back().passes.empty()) progs.pop_back();
        return progs;
    }
};

}  // namespace

std::vector<SweepProgram> build_sweep(const std::vector<SweepGate>& gates, const TileStage& st, bool fixed_point,
                                      bool reverse, bool ordered, std::vector<TileOp>* ops) {
    return Builder(gates, st, fixed_point, reverse, ordered, ops).run();
}

bool is_unitary(const double* m, size_t k) {
    const size_t d = size_t(1) << k;
    for (size_t r = 0; r < d; r++)
        for (size_t c = 0; c <= r; c++) {
            double re = r == c ? -1.0 : 0.0, im = 0.0;
            for (size_t j = 0; j < d; j++) {
                const double *a = m + 2 * (r * d + j), *b = m + 2 * (c * d + j);
                re += a[0] * b[0] + a[1] * b[1];
                im += a[1] * b[0] - a[0] * b[1];
            }
            if (!(std::fabs(re) < 1e-9 && std::fabs(im) < 1e-9)) return false;
        }
    return true;
}

}  // namespace qs
