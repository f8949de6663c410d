// qs_fuse.cpp — dense-block gate fusion (host, FP64).
//
// The reference's closest feature is QuantumCircuit's reduction passes
// (src/operation.rs:114-269), which multiply or kron neighbouring gates by
// heuristics (and cancel equal consecutive real gates, which is only correct
// for involutions). Here a block is the exact FP64 product of the gates it
// absorbs, in their application order; a gate is moved ahead only past gates
// with which it shares no qubit.
#include "qs_fuse.h"

#include <algorithm>
#include <cstring>

namespace qs {

static uint64_t gate_mask(const qs_gate& g) {
    uint64_t m = 0;
    for (size_t j = 0; j < g.k; j++) m |= 1ull << g.targets[j];
    return m;
}

// U <- G_expanded * U, where U is 2^k x 2^k over `qubits` and G acts on a subset.
static void left_multiply(std::vector<double>& U, const std::vector<int>& qubits, const qs_gate& g) {
    const int k = int(qubits.size());
    const uint64_t dim = 1ull << k;
    const int kg = int(g.k);
    const uint64_t gd = 1ull << kg;
    std::vector<int> lb(kg);  // local bit of gate target j inside the block
    uint64_t gmask = 0;
    for (int j = 0; j < kg; j++) {
        lb[j] = int(std::find(qubits.begin(), qubits.end(), int(g.targets[j])) - qubits.begin());
        gmask |= 1ull << lb[j];
    }
    // row by row of the result: the gate's rows r_0 .. of U combined over all columns at once
    const size_t w = 2 * dim;
    std::vector<double> in(gd * w);
    std::vector<uint64_t> row(gd);
    for (uint64_t base = 0; base < dim; base++) {
        if (base & gmask) continue;
        for (uint64_t i = 0; i < gd; i++) {
            uint64_t r = base;
            for (int j = 0; j < kg; j++)
                if (i >> j & 1) r |= 1ull << lb[j];
            row[i] = r;
            std::copy(U.begin() + long(r * w), U.begin() + long((r + 1) * w), in.begin() + long(i * w));
        }
        for (uint64_t i = 0; i < gd; i++) {
            double* out = U.data() + row[i] * w;
            std::fill(out, out + w, 0.0);
            for (uint64_t j = 0; j < gd; j++) {
                const double gr = g.matrix[2 * (i * gd + j)], gi = g.matrix[2 * (i * gd + j) + 1];
                const double* col = in.data() + j * w;
                for (size_t c = 0; c < w; c += 2) {
                    out[c] += gr * col[c] - gi * col[c + 1];
                    out[c + 1] += gr * col[c + 1] + gi * col[c];
                }
            }
        }
    }
}

namespace {

// Chooses the qubits of the next block. A block's pass over the state costs the same whatever it holds, so
// the set that absorbs the most multi-qubit gates wins (1-qubit gates come along wherever they are).
// From every multi-qubit gate that can run now, a set grows by the qubits of a gate that stops it, or of
// another gate that can run now, whichever absorbs the most per qubit added.
class BlockSearch {
public:
    BlockSearch(const qs_gate* gates, size_t m, int W) : W_(W), mask_(m), lists_(64) {
        for (size_t i = 0; i < m; i++) {
            mask_[i] = gate_mask(gates[i]);
            if (gates[i].k >= 2)
                for (uint64_t q = mask_[i]; q; q &= q - 1) lists_[__builtin_ctzll(q)].push_back(int(i));
        }
        std::fill(head_, head_ + 64, 0);
    }

    void placed(int gate) {  // a gate goes into a block: it was the next one on each of its qubits
        if (__builtin_popcountll(mask_[gate]) < 2) return;
        for (uint64_t q = mask_[gate]; q; q &= q - 1) head_[__builtin_ctzll(q)]++;
    }

    uint64_t best() const {
        std::vector<uint64_t> ready;
        for (int q = 0; q < 64; q++) {
            const int g = next(q, head_[q]);
            if (g >= 0 && __builtin_ctzll(mask_[g]) == q && runs(mask_[g], g) && __builtin_popcountll(mask_[g]) <= W_)
                ready.push_back(mask_[g]);
        }
        uint64_t best_set = 0;
        int best_count = 0;
        for (const uint64_t seed : ready) {
            uint64_t S = seed, stops[8];
            int nstops = 0, have = absorbed(S, stops, &nstops);
            while (__builtin_popcountll(S) < W_) {
                uint64_t add = 0, others[8];
                int n = 0, add_have = 0;
                double gain = 0.0;
                auto consider = [&](uint64_t m) {
                    const int extra = __builtin_popcountll(m & ~S);
                    if (!extra || __builtin_popcountll(S) + extra > W_) return;
                    const int count = absorbed(S | m, others, &n);
                    const double g = double(count - have) / extra;
                    if (g > gain) gain = g, add = m & ~S, add_have = count;
                };
                for (int i = 0; i < nstops; i++) consider(stops[i]);
                for (const uint64_t m : ready)
                    if (!(m & S)) consider(m);
                if (!add) break;
                S |= add;
                have = absorbed(S, stops, &nstops);
            }
            if (have > best_count || (have == best_count && __builtin_popcountll(S) < __builtin_popcountll(best_set))) {
                best_count = have;
                best_set = S;
            }
        }
        return best_set;
    }

private:
    int W_;
    std::vector<uint64_t> mask_;
    std::vector<std::vector<int>> lists_;  // per qubit: its multi-qubit gates in order
    int head_[64];                         // the first not placed yet

    int next(int q, int at) const { return at < int(lists_[q].size()) ? lists_[q][at] : -1; }
    bool runs(uint64_t m, int gate) const {  // the next gate on each of its qubits
        for (uint64_t q = m; q; q &= q - 1)
            if (next(__builtin_ctzll(q), head_[__builtin_ctzll(q)]) != gate) return false;
        return true;
    }
    // Multi-qubit gates that a block on S absorbs; stops: the gates that end it on some qubit (up to 8).
    int absorbed(uint64_t S, uint64_t* stops, int* nstops) const {
        int at[64];
        for (uint64_t q = S; q; q &= q - 1) at[__builtin_ctzll(q)] = head_[__builtin_ctzll(q)];
        int count = 0;
        for (bool more = true; more;) {
            more = false;
            for (uint64_t s = S; s; s &= s - 1) {
                const int q = __builtin_ctzll(s);
                const int g = next(q, at[q]);
                if (g < 0 || (mask_[g] & ~S)) continue;
                bool all = true;
                for (uint64_t t = mask_[g]; t; t &= t - 1) all = all && next(__builtin_ctzll(t), at[__builtin_ctzll(t)]) == g;
                if (!all) continue;
                for (uint64_t t = mask_[g]; t; t &= t - 1) at[__builtin_ctzll(t)]++;
                count++;
                more = true;
            }
        }
        *nstops = 0;
        for (uint64_t s = S; s; s &= s - 1) {
            const int q = __builtin_ctzll(s), g = next(q, at[q]);
            if (g >= 0 && (mask_[g] & ~S) && *nstops < 8) stops[(*nstops)++] = mask_[g];
        }
        return count;
    }
};

}  // namespace

std::vector<FusedBlock> fuse_blocks(const qs_gate* gates, size_t m, int W, bool search) {
    std::vector<FusedBlock> blocks;
    std::vector<int> remaining(m);
    for (size_t i = 0; i < m; i++) remaining[i] = int(i);
    BlockSearch chooser(gates, search ? m : 0, W);
    while (!remaining.empty()) {
        // qubits of the block so far; qubits of gates left behind
        uint64_t bq = search ? chooser.best() : 0, blocked = 0;
        // the chosen set first; what room it leaves is claimed by the gates in turn
        std::vector<int> members, rest;
        for (int idx : remaining) {
            const uint64_t qm = gate_mask(gates[idx]);
            if (qm & blocked) {
                blocked |= qm;
                rest.push_back(idx);
                continue;
            }
            if (__builtin_popcountll(bq | qm) <= W || (members.empty() && !bq)) {
                if (__builtin_popcountll(bq | qm) > W) {  // a gate wider than W: its own block
                    members.push_back(idx);
                    bq |= qm;
                    blocked = ~0ull;  // close the block
                    continue;
                }
                bq |= qm;
                members.push_back(idx);
            } else {
                blocked |= qm;
                rest.push_back(idx);
            }
        }
        FusedBlock b;
        bq = 0;  // the qubits its gates use
        for (int idx : members) {
            bq |= gate_mask(gates[idx]);
            if (search) chooser.placed(idx);
        }
        for (int q = 0; q < 64; q++)
            if (bq >> q & 1ull) b.qubits.push_back(q);
        const uint64_t dim = 1ull << b.qubits.size();
        b.u.assign(2 * dim * dim, 0.0);
        for (uint64_t i = 0; i < dim; i++) b.u[2 * (i * dim + i)] = 1.0;
        for (int idx : members) left_multiply(b.u, b.qubits, gates[idx]);
        b.members = members;
        blocks.push_back(std::move(b));
        remaining.swap(rest);
    }
    return blocks;
}

void pad_block(FusedBlock* b, int k, int n) {
    while (int(b->qubits.size()) < k) {
        int q = 0;
        while (q < n && std::find(b->qubits.begin(), b->qubits.end(), q) != b->qubits.end()) q++;
        if (q >= n) return;
        // insert q keeping qubits sorted; the matrix gains an identity factor on q
        std::vector<int> nq = b->qubits;
        nq.push_back(q);
        std::sort(nq.begin(), nq.end());
        const int pos = int(std::find(nq.begin(), nq.end(), q) - nq.begin());
        const uint64_t od = 1ull << b->qubits.size(), nd = od << 1;
        std::vector<double> nu(2 * nd * nd, 0.0);
        auto expand = [&](uint64_t i, uint64_t bit) {  // insert `bit` at position pos of index i
            const uint64_t lo = i & ((1ull << pos) - 1ull);
            return ((i >> pos) << (pos + 1)) | (bit << pos) | lo;
        };
        for (uint64_t r = 0; r < od; r++)
            for (uint64_t c = 0; c < od; c++)
                for (uint64_t bit = 0; bit < 2; bit++) {
                    const uint64_t R = expand(r, bit), C = expand(c, bit);
                    nu[2 * (R * nd + C)] = b->u[2 * (r * od + c)];
                    nu[2 * (R * nd + C) + 1] = b->u[2 * (r * od + c) + 1];
                }
        b->qubits = nq;
        b->u.swap(nu);
    }
}

}  // namespace qs
