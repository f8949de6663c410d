// qs_circuit.cu — gate dispatch and the circuit runner.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "qs_circuit.h"
#include "qs_kernels.h"
#include "qs_fuse.h"
#include "qs_tile.h"

namespace qs {

static int fail(cudaError_t e, const char* what, std::string* msg) {
    if (msg) *msg = std::string(what) + ": " + cudaGetErrorString(e);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return QS_OUT_OF_MEMORY;
    }
    return QS_CUDA_ERROR;
}

static int apply_visited(void* state, int n, int reg_qubits, int prec, int arith, const OpDesc& op, cudaStream_t s,
                         int sms, std::string* msg);

int apply_op(void* state, int n, int prec, int arith, const OpDesc& op, cudaStream_t s, int sms, std::string* msg,
             LiveSpace* live) {
    if (op.kind == OP_NOOP) return QS_OK;
    if (op.k > kMaxBigK) {
        if (msg) *msg = "dense or monomial sub-operation wider than " + std::to_string(kMaxBigK) + " qubits";
        return QS_INVALID_ARGUMENT;
    }
    if (live && live->mask) {
        // A circuit starts from a basis state and a gate frees its own qubits only: of the first layer on 28
        // qubits a gate on qubit q has 2^(q + 1) amplitudes to visit (28 qubits, 84 gates: 113.6 ms without
        // this, 96.5 ms with it).
        // The known qubits act as controls at their values, the highest ones at 0 as a smaller register.
        const uint64_t targets = target_mask(op), known = live->mask & ~targets;
        const uint64_t val = live->val;
        live->release(targets);
        if (known) {
            if ((op.fixval ^ val) & op.fixmask & known) return QS_OK;  // a control that no amplitude meets
            OpDesc r = op;
            r.fixmask |= known;
            r.fixval |= val & known;
            int m = n;
            while (m > 1 && (r.fixmask & ~r.fixval) >> (m - 1) & 1ull) r.fixmask &= ~(1ull << --m);
            return apply_visited(state, m, n, prec, arith, r, s, sms, msg);
        }
    }
    return apply_visited(state, n, n, prec, arith, op, s, sms, msg);
}

// On the register's first 2^n amplitudes.
static int apply_visited(void* state, int n, int reg_qubits, int prec, int arith, const OpDesc& op, cudaStream_t s,
                         int sms, std::string* msg) {
    if (op.k <= kMaxSmallK) {
        cudaError_t e = launch_op(op, state, n, prec, arith, s, sms, reg_qubits);
        return e == cudaSuccess ? QS_OK : fail(e, "gate kernel", msg);
    }
    // Wide gate: tables in device memory, read the pre-gate state from a copy.
    std::vector<uint64_t> off, off_src;
    std::vector<uint8_t> pf;
    std::vector<int8_t> lane;
    std::vector<unsigned char> mat;
    big_op_host_tables(op, prec, &off, &off_src, &pf, &lane, &mat);
    const size_t amp = prec == QS_PREC_C64 ? 8 : 16;
    const size_t sbytes = (size_t(1) << n) * amp;
    unsigned char* blob = nullptr;
    const size_t o_off = 0, o_src = o_off + off.size() * 8, o_pf = o_src + off_src.size() * 8,
                 o_lane = o_pf + ((pf.size() + 15) / 16) * 16, o_mat = o_lane + ((lane.size() + 15) / 16) * 16,
                 o_state = o_mat + ((mat.size() + 255) / 256) * 256, total = o_state + sbytes;
    cudaError_t e = device_alloc((void**)&blob, total, s);
    if (e != cudaSuccess) return fail(e, "wide gate buffers", msg);
    BigOpBuffers b;
    b.off = reinterpret_cast<const uint64_t*>(blob + o_off);
    b.off_src = reinterpret_cast<const uint64_t*>(blob + o_src);
    b.pf = blob + o_pf;
    b.lane = reinterpret_cast<const int8_t*>(blob + o_lane);
    b.mat = blob + o_mat;
    if (!off.empty()) e = cudaMemcpyAsync(blob + o_off, off.data(), off.size() * 8, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && !off_src.empty())
        e = cudaMemcpyAsync(blob + o_src, off_src.data(), off_src.size() * 8, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && !pf.empty()) e = cudaMemcpyAsync(blob + o_pf, pf.data(), pf.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && !lane.empty())
        e = cudaMemcpyAsync(blob + o_lane, lane.data(), lane.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess && !mat.empty()) e = cudaMemcpyAsync(blob + o_mat, mat.data(), mat.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(blob + o_state, state, sbytes, cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) e = launch_op_big(op, state, blob + o_state, n, prec, arith, b, s, sms);
    cudaFreeAsync(blob, s);
    return e == cudaSuccess ? QS_OK : fail(e, "wide gate", msg);
}

// Every entry finite in the register's precision: zeros stay zeros.
static bool all_finite(const std::vector<double>& m, int prec) {
    for (double v : m)
        if (!std::isfinite(prec == QS_PREC_C64 ? double(float(v)) : v)) return false;
    return true;
}

// fuse == 2: dense blocks of up to max_width qubits. On registers of at least 12 qubits, complex64
// or complex128 in fixed-point arithmetic, the blocks run on the tensor cores inside 12-qubit
// tiles; otherwise each block is one dense gate sweep.
static int run_blocks(void* state, int n, int prec, int arith, const qs_gate* gates, size_t m,
                      const qs_circuit_options& opts, cudaStream_t s, int sms, std::string* msg, LiveSpace* live,
                      bool* overflow) {
    // Tensor-core blocks inside 12-qubit tiles: 3xTF32 on complex64 registers; on complex128
    // registers in fixed-point arithmetic, the FP64-accurate split-integer product (k_tile_oz).
    const bool oz = (prec == QS_PREC_C128) && arith == QS_ARITH_FX64 && n >= 12;
    const bool tensor = ((prec == QS_PREC_C64) && n >= 12) || oz;
    // automatic width: where each block's sweep stays cheap. Tensor-core blocks cost the same at any
    // width up to 5; complex128 double-float blocks run the double-float dense kernel up to 3
    // qubits (4- and 5-qubit blocks fall back to FP64, which GB300 runs at 1/64 of the FP32 rate);
    // FP64 blocks cost as many FP64 operations per amplitude as the gates they fuse, so 2 only halves
    // the sweeps.
    const int autow = tensor ? 5 : (prec == QS_PREC_C128 && arith == QS_ARITH_DF64) ? 3 : 2;
    const int W = std::max(2, std::min(5, opts.max_width > 0 ? opts.max_width : autow));
    // Choosing a block's qubits takes 15 us of host time and saves 0.3 of a pass over the state: worth it
    // from states of 128 MiB (a pass of 40 us and more).
    const bool search = (uint64_t(prec == QS_PREC_C64 ? 8 : 16) << n) >= (uint64_t(128) << 20);
    std::vector<FusedBlock> blocks = fuse_blocks(gates, m, W, search);
    std::vector<OpDesc> ops;
    std::vector<float> frags;
    std::vector<double> mats;
    for (FusedBlock& b : blocks) {
        const bool finite = all_finite(b.u, prec);
        if (live && !finite) *live = LiveSpace{};
        if (overflow && !finite) *overflow = true;
        std::vector<size_t> tq(b.qubits.begin(), b.qubits.end());
        OpDesc op;
        // digits of an infinity or NaN are digits of nothing: such a block is a dense sweep of its own
        if (tensor && int(b.qubits.size()) <= 5 && (finite || !oz)) {
            pad_block(&b, 5, n);
            op.kind = OP_BLOCK;
            op.k = 5;
            op.orig_k = 5;
            for (int j = 0; j < 5; j++) op.tq[j] = b.qubits[j];
            op.touched_rows = 32;
            const size_t per = 4 * kBlockFragFloat4;  // floats per complex64 block
            op.block = int(oz ? mats.size() / 2048 : frags.size() / per);
            if (oz) {
                mats.insert(mats.end(), b.u.begin(), b.u.end());
            } else {
                frags.resize(frags.size() + per);
                block_fragments(b.u, frags.data() + frags.size() - per);
            }
        } else {
            tq.assign(b.qubits.begin(), b.qubits.end());
            classify_gate(b.u.data(), tq.size(), tq.data(), &op);
        }
        ops.push_back(std::move(op));
    }
    if (!tensor) {
        for (const OpDesc& op : ops) {
            int rc = apply_op(state, n, prec, arith, op, s, sms, msg, live);
            if (rc) return rc;
        }
        return QS_OK;
    }
    // rows of 128 bytes: 16 complex64 amplitudes leave eight of the tile's qubits to the stage's two blocks
    // (30 qubits, 4 layers: 9 stages against 11 with rows of 256 bytes)
    const int T = std::min(12, n), L = std::min(oz ? 5 : 4, T);
    std::vector<TileStage> stages = plan_tiles(ops, n, T, L, false, oz ? kMaxOzBlocks : kMaxTcBlocks, true);
    return run_tiled(state, n, prec, arith, ops, stages, s, sms, msg, &frags, nullptr, live, &mats);
}

int run_circuit(void* state, int n, int prec, int arith, const std::vector<OpDesc>& ops, const qs_gate* gates,
                const qs_circuit_options& opts, cudaStream_t s, int sms, std::string* msg, int* derr_dev,
                LiveSpace* live, bool* overflow) {
    if (opts.fuse == 2 && gates)
        return run_blocks(state, n, prec, arith, gates, ops.size(), opts, s, sms, msg, live, overflow);
    if (opts.fuse >= 1) {
        // Tile qubits: 32 KiB of shared memory per tile by default; below 19 (complex64) or 18
        // (complex128) qubits smaller tiles, so that up to 128 blocks share the state (complex64
        // keeps the 9 tile qubits its register passes need).
        int T = opts.tile_qubits;
        if (T <= 0) {
            const int cap = prec == QS_PREC_C64 ? 12 : 11, floor = prec == QS_PREC_C64 ? 9 : 8;
            T = std::max(floor, std::min(cap, n - 7));
        }
        T = std::min(T, n);
        const int L = std::min(5, T);
        const bool exact_order = prec == QS_PREC_C128 && arith == QS_ARITH_EXACT;
        std::vector<TileStage> stages = plan_tiles(ops, n, T, L, exact_order);
        // Choosing each stage's qubits (60..100 us of host time for 400 gates) gives fewer stages for some circuits
        // and more for others (layers of random pairs: 27 qubits 13 for 14, complex64 19.2 ms to 17.7 ms; 24
        // qubits 15 for 14). Taken where it gives fewer, on states of 64 MiB and more: a stage takes 60 us there.
        if ((uint64_t(prec == QS_PREC_C64 ? 8 : 16) << n) >= (uint64_t(64) << 20)) {
            std::vector<TileStage> searched = plan_tiles(ops, n, T, L, exact_order, kMaxStageOps, false, true);
            if (searched.size() < stages.size()) stages.swap(searched);
        }
        return run_tiled(state, n, prec, arith, ops, stages, s, sms, msg, nullptr, derr_dev, live);
    }
    for (size_t g = 0; g < ops.size(); g++) {
        int rc = apply_op(state, n, prec, arith, ops[g], s, sms, msg, live);
        if (rc) return rc;
    }
    return QS_OK;
}

}  // namespace qs
