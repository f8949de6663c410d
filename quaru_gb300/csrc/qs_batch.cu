// qs_batch.cu — forward + adjoint gradients for a batch of circuits in one persistent launch.
//
// No counterpart in the reference. Each circuit's gates are planned into tiled stages (the planner
// of the fused forward path, qs_plan.cpp): forward stages, one step forming lambda = H psi with the
// energy partial sums, and reverse stages walking the gates backwards (rotations with their
// Im<lambda|A|psi> partials, fixed gates un-applied from psi and lambda). A work item is
// (circuit c, step s, chunk j): a range of tiles of one stage, each tile loaded once into shared
// memory, taken through all of the stage's gates and written back once (or, for the H psi step, a
// range of amplitude pairs). Items are ordered by step round across circuits, so an item only ever
// waits for items handed out before it; those are held by running CTAs, which makes the schedule
// deadlock-free without any co-residency assumption. Every wait is bounded: when it gives up it
// raises an error flag that makes every CTA return, and the host reports QS_TIMEOUT.
//
// The whole pass (parameter upload, state reset, persistent kernel, partial reduction, result
// download) is captured once in a CUDA graph; a run writes new parameters into pinned memory and
// replays it. A stage runs as a pass program of qs_sweep.cuh (complex64 tiles, or complex128 ones in
// fixed point; in FP64 where a fixed gate is not unitary). Complex128 batches with QS_ARITH_DF64 hold the
// tiles of stages made of rotations and CNOTs as double-float values (FP32 pipe), one gate after another,
// with the inner products accumulated in FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <limits>
#include <sstream>
#include <string>
#include <vector>

#include "qs_device.cuh"
#include "qs_kernels.h"
#include "qs_reduce.cuh"
#include "qs_rot.cuh"
#include "qs_sweep.cuh"
#include "qs_sweep.h"
#include "qs_tile.h"
#include "qs_tma.cuh"

namespace qs {
namespace {

constexpr int kBT = 256;
constexpr int kCnot = 17;  // CNOT
constexpr int kBTileMax = 11;  // tile qubits
constexpr int kBMaxRot = kMaxStageOps;  // rotations per stage
constexpr long long kWaitCycles = 20000000000LL;  // ~10 s at 2 GHz: dependency waits give up after this

struct BCirc {
    unsigned long long psi, lam;
    int n, nterms, term_off, nsteps, counter_off, nrot;
    int epart_off, rpart_off;  // partials: energy (2^nche_log), then rotation r at rpart_off + r * 2^ncht_log
    int nche_log, ncht_log;    // chunks of the H psi step and of every tile stage
    int T, stage_off, nfwd;    // tile qubits, first stage, forward stages (step nfwd is H psi)
};

struct BStage {
    int op_off, nops, nrot, df;  // df: double-float tiles, gates op_off .. op_off + nops
    int L, H, prog, pad;         // prog: the stage's program otherwise
    uint8_t pos[16];   // the tile's qubits, sorted (its base index skips them)
    uint8_t high[8];   // qubit of local bit L + b
};

struct BOp {
    int kind;   // QS_GATE_RX / RY / RZ, kCnot
    int tb;     // local target bit
    int cb;     // CNOT: local control bit, or -1
    int cglob;  // CNOT: control qubit outside the tile, or -1
    int cs;     // rotation: index of (cos, sin) of theta/2
    int rslot;  // rotation: circuit-level slot
    int lrot;   // rotation: stage-local slot
    int pad;
};

struct BPauli {
    double c;
    unsigned long long x, z;
    float ch, cl;  // c as a float pair (complex64 circuits)
    uint32_t cls;  // |x & z| mod 4: the term's factor i^cls
    uint32_t pad_;
};

template <typename T>
struct St;
template <>
struct St<double2> {
    static __device__ __forceinline__ double2 ld(const double2* p, uint64_t i) { return __ldcg(p + i); }
    static __device__ __forceinline__ void st(double2* p, uint64_t i, double2 v) { __stcg(p + i, v); }
    static __device__ __forceinline__ double2 d(double2 v) { return v; }
    static __device__ __forceinline__ double2 from(double2 v) { return v; }
};
template <>
struct St<float2> {
    static __device__ __forceinline__ float2 ld(const float2* p, uint64_t i) { return __ldcg(p + i); }
    static __device__ __forceinline__ void st(float2* p, uint64_t i, float2 v) { __stcg(p + i, v); }
    // integer-pipe conversion (exact for normal floats; subnormals read as zero)
    static __device__ __forceinline__ double2 d(float2 v) { return make_double2(df_f2d(v.x), df_f2d(v.y)); }
    static __device__ __forceinline__ float2 from(double2 v) { return make_float2(float(v.x), float(v.y)); }
};

template <typename T>
__global__ void __launch_bounds__(kBT) k_batch_reset(const BCirc* __restrict__ circs) {
    const BCirc C = circs[blockIdx.y];
    T* psi = reinterpret_cast<T*>(C.psi);
    const uint64_t N = 1ull << C.n;
    for (uint64_t i = uint64_t(blockIdx.x) * kBT + threadIdx.x; i < N; i += uint64_t(gridDim.x) * kBT)
        St<T>::st(psi, i, St<T>::from(make_double2(i == 0 ? 1.0 : 0.0, 0.0)));
}

__device__ __forceinline__ uint32_t pair_index(uint32_t p, int tb) {
    return ((p >> tb) << (tb + 1)) | (p & ((1u << tb) - 1u));
}

// One gate of a double-float stage on the tile(s) in shared memory. fwd: psi only; reverse: psi and lambda,
// with a rotation's inner-product term accumulated (before it is un-applied).
template <int AXIS>
__device__ __forceinline__ DfAcc tile_rot_df(float4* sp, float4* sl, uint32_t half, int tb, double c, double sn,
                                              bool fwd) {
    float ch, cl, sh, slo;
    df_split(c, ch, cl);
    df_split(fwd ? sn : -sn, sh, slo);
    DfAcc acc;
    for (uint32_t p = threadIdx.x; p < half; p += kBT) {
        const uint32_t i0 = pair_index(p, tb), i1 = i0 | (1u << tb);
        float4 a = sp[i0], b = sp[i1];
        if (!fwd) {
            float4 l0 = sl[i0], l1 = sl[i1];
            adj_im_df_acc<AXIS>(acc, l0, l1, a, b);
            df_rot_pair<AXIS>(ch, cl, sh, slo, l0, l1);
            sl[i0] = l0;
            sl[i1] = l1;
        }
        df_rot_pair<AXIS>(ch, cl, sh, slo, a, b);
        sp[i0] = a;
        sp[i1] = b;
    }
    return acc;
}

template <typename E>
__device__ __forceinline__ void tile_cnot(E* s, uint32_t half, int tb, int cb) {
    for (uint32_t p = threadIdx.x; p < half; p += kBT) {
        const uint32_t i0 = pair_index(p, tb);
        if (cb >= 0 && !((i0 >> cb) & 1u)) continue;
        const uint32_t i1 = i0 | (1u << tb);
        const E t = s[i0];
        s[i0] = s[i1];
        s[i1] = t;
    }
}

// Tiles [first, first + count) of a double-float stage.
__device__ __noinline__ void batch_df(const BCirc& C, const BStage& S, const BOp* __restrict__ ops,
                                      const double2* __restrict__ cs, uint64_t first, uint64_t count, bool fwd,
                                      unsigned char* smem, double* __restrict__ partials, uint32_t j) {
    float4* fp = reinterpret_cast<float4*>(smem);
    float4* fl = fp + (1u << kBTileMax);
    uint64_t* rowoff = reinterpret_cast<uint64_t*>(fl + (1u << kBTileMax));
    double* sacc = reinterpret_cast<double*>(rowoff + (1 << kTileMaxHigh));  // [kBMaxRot][8 warps]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double2* psi = reinterpret_cast<double2*>(C.psi);
    double2* lam = reinterpret_cast<double2*>(C.lam);
    const uint32_t tsize = 1u << C.T, half = tsize >> 1, lmask = (1u << S.L) - 1u;
    for (int r = threadIdx.x; r < (1 << S.H); r += kBT) {
        uint64_t o = 0;
        for (int b = 0; b < S.H; b++)
            if (r >> b & 1) o |= 1ull << S.high[b];
        rowoff[r] = o;
    }
    if (!fwd)
        for (int r = threadIdx.x; r < S.nrot * (kBT / 32); r += kBT) sacc[r] = 0.0;
    __syncthreads();
    for (uint64_t t = first; t < first + count; t++) {
        uint64_t base = t;  // insert the tile's qubits as zero bits
        for (int k = 0; k < C.T; k++) {
            const int q = S.pos[k];
            base = ((base >> q) << (q + 1)) | (base & ((1ull << q) - 1ull));
        }
        auto split = [](double2 v) {
            float4 f;
            df_split(v.x, f.x, f.y);
            df_split(v.y, f.z, f.w);
            return f;
        };
        auto join = [](float4 f) {
            return make_double2(__dadd_rn(df_f2d(f.x), df_f2d(f.y)), __dadd_rn(df_f2d(f.z), df_f2d(f.w)));
        };
        for (uint32_t i = threadIdx.x; i < tsize; i += kBT) {
            const uint64_t g = base + rowoff[i >> S.L] + (i & lmask);
            fp[i] = split(__ldcg(psi + g));
            if (!fwd) fl[i] = split(__ldcg(lam + g));
        }
        __syncthreads();
        for (int o = 0; o < S.nops; o++) {
            const BOp op = ops[S.op_off + o];
            if (op.kind == kCnot) {
                if (op.cglob < 0 || ((base >> op.cglob) & 1ull)) {  // outside control: the whole tile
                    tile_cnot(fp, half, op.tb, op.cb);
                    if (!fwd) tile_cnot(fl, half, op.tb, op.cb);
                }
            } else {
                const double2 t2 = cs[op.cs];
                DfAcc f;
                if (op.kind == QS_GATE_RX) f = tile_rot_df<QS_GATE_RX>(fp, fl, half, op.tb, t2.x, t2.y, fwd);
                else if (op.kind == QS_GATE_RY) f = tile_rot_df<QS_GATE_RY>(fp, fl, half, op.tb, t2.x, t2.y, fwd);
                else f = tile_rot_df<QS_GATE_RZ>(fp, fl, half, op.tb, t2.x, t2.y, fwd);
                if (!fwd) {  // float pairs over the warp, one FP64 rejoin
                    f.warp_reduce();
                    if (lane == 0) sacc[op.lrot * (kBT / 32) + warp] += __dadd_rn(df_f2d(f.s), df_f2d(f.c));
                }
            }
            __syncthreads();
        }
        for (uint32_t i = threadIdx.x; i < tsize; i += kBT) {
            const uint64_t g = base + rowoff[i >> S.L] + (i & lmask);
            __stcg(psi + g, join(fp[i]));
            if (!fwd) __stcg(lam + g, join(fl[i]));
        }
        __syncthreads();
    }
    if (!fwd)  // this item's partial of every rotation of the stage
        for (int o = threadIdx.x; o < S.nops; o += kBT) {
            const BOp op = ops[S.op_off + o];
            if (op.kind == kCnot) continue;
            double v = 0.0;
            for (int w = 0; w < kBT / 32; w++) v += sacc[op.lrot * (kBT / 32) + w];
            partials[C.rpart_off + (size_t(op.rslot) << C.ncht_log) + j] = v;
        }
}

// The sweep programs' tables, and what a run fills in from its parameters.
struct BSweep {
    const SweepRange* ranges;
    const SweepPass* passes;
    const TileOp* fixed;
    const SweepCoef* coefs;
    const double* sigmas;
    const int* rslot;  // circuit-level slot of each program rotation
};

// Tiles [j * tpi, (j + 1) * tpi) of a stage through its program.
template <typename T, int RB, bool REV>
__device__ void batch_sweep(const BCirc& C, const BStage& S, const BSweep& W, uint64_t first, uint64_t count, bool store,
                            unsigned char* smem, double* __restrict__ partials, uint32_t j) {
    using G = typename Sw<T>::Glob;
    const SweepRange R = W.ranges[S.prog];
    T* sp = reinterpret_cast<T*>(smem);
    T* sl = sp + (1u << kBTileMax);
    const SweepSide<T> side(reinterpret_cast<unsigned char*>(sl + (1u << kBTileMax)), R.npass, R.nrot, R.ndiag, REV);
    const SweepTile t{C.T, S.L, R.npass, R.nrot, R.ndiag, store, W.sigmas[S.prog]};
    for (int r = threadIdx.x; r < (1 << S.H); r += kBT) {
        uint64_t o = 0;
        for (int b = 0; b < S.H; b++)
            if (r >> b & 1) o |= 1ull << S.high[b];
        side.rowoff[r] = o;
    }
    sw_begin<T>(side, W.passes + R.pass0, R.npass, W.coefs + R.coef0, R.nrot, C.T, REV, t.sigma, kBT);
    for (uint64_t k = first; k < first + count; k++) {
        uint64_t base = k;  // insert the tile's qubits as zero bits
        for (int i = 0; i < C.T; i++) {
            const int q = S.pos[i];
            base = ((base >> q) << (q + 1)) | (base & ((1ull << q) - 1ull));
        }
        G* psi = reinterpret_cast<G*>(C.psi);
        sw_tile<T, RB, REV, true>(psi, psi, reinterpret_cast<G*>(C.lam), base, t, sp, sl, side, W.fixed, kBT);
    }
    if (REV)  // this item's partial of every rotation of the stage
        for (int r = threadIdx.x; r < R.nrot; r += kBT)
            partials[C.rpart_off + (size_t(W.rslot[R.coef0 + r]) << C.ncht_log) + j] = sw_total<T>(side, r, kBT);
}

// T: the tile type; DF: stages marked df run as double-float tiles.
template <typename TT, bool DF>
__global__ void __launch_bounds__(kBT, DF || sizeof(TT) == 8 ? 3 : 2)
    k_batch(const BCirc* __restrict__ circs, const BStage* __restrict__ stages, const BOp* __restrict__ ops,
            const BPauli* __restrict__ terms, const double2* __restrict__ cs, const __grid_constant__ BSweep sweep,
            const uint32_t* __restrict__ seg_first, const int4* __restrict__ segs, int nsegs, uint32_t nitems,
            unsigned int* __restrict__ counters, double* __restrict__ partials, unsigned int* __restrict__ ticket,
            int* __restrict__ err) {
    using T = typename Sw<TT>::Glob;
    static_assert(!DF || sizeof(T) == 16, "double-float tiles hold complex128 states");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t s_item;
    __shared__ int s_seg, s_stop;
    for (;;) {
        if (threadIdx.x == 0) {
            s_item = atomicAdd(ticket, 1u);
            s_stop = (s_item >= nitems) || (*reinterpret_cast<volatile int*>(err) != 0);
            if (!s_stop) {  // segment holding this item: last seg_first <= item
                int lo = 0, hi = nsegs - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (seg_first[mid] <= s_item) lo = mid; else hi = mid - 1;
                }
                s_seg = lo;
            }
        }
        __syncthreads();
        if (s_stop) return;
        const int4 sg = segs[s_seg];
        const int c = sg.x, s = sg.y, prevnch = sg.w;
        const uint32_t j = s_item - seg_first[s_seg];
        const BCirc C = circs[c];
        if (s > 0 && threadIdx.x == 0) {  // every chunk of the previous step must be done
            if (!counter_wait_bounded(counters + C.counter_off + s - 1, unsigned(prevnch), kWaitCycles)) {
                atomicExch(err, 1);
                s_stop = 1;
            }
            __threadfence();
        }
        __syncthreads();
        if (s_stop) return;
        T* psi = reinterpret_cast<T*>(C.psi);
        T* lam = reinterpret_cast<T*>(C.lam);
        if (s == C.nfwd) {  // lambda = H psi over amplitudes [2 p0, 2 p1), energy partial
            const int cl = C.n - 1 - C.nche_log;
            const uint64_t p0 = uint64_t(j) << cl, p1 = p0 + (1ull << cl);
            double e = 0.0;
            DfAcc eacc;  // complex64: the energy terms as a compensated float pair
            for (uint64_t i = 2 * p0 + threadIdx.x; i < 2 * p1; i += kBT) {
                if constexpr (sizeof(T) == 8) {  // complex64: products and sums in compensated float pairs
                    DfAcc fre, fim;
                    for (int t = 0; t < C.nterms; t++) {
                        const BPauli& P = terms[C.term_off + t];
                        const uint64_t k = i ^ P.x;
                        const float2 v = St<T>::ld(psi, k);
                        const bool neg = __popcll(P.z & k) & 1;
                        const float ch = neg ? -P.ch : P.ch, cl = neg ? -P.cl : P.cl;
                        float xr, xi;  // i^cls * v
                        switch (P.cls) {
                            case 0: xr = v.x; xi = v.y; break;
                            case 1: xr = -v.y; xi = v.x; break;
                            case 2: xr = -v.x; xi = -v.y; break;
                            default: xr = v.y; xi = -v.x; break;
                        }
                        fre.add_prod(ch, xr);
                        fre.c = __fmaf_rn(cl, xr, fre.c);
                        fim.add_prod(ch, xi);
                        fim.c = __fmaf_rn(cl, xi, fim.c);
                    }
                    const float2 lv = make_float2(__fadd_rn(fre.s, fre.c), __fadd_rn(fim.s, fim.c));
                    St<T>::st(lam, i, lv);
                    const float2 pv = St<T>::ld(psi, i);  // energy term Re(conj(psi_i) lambda_i)
                    eacc.add_prod(pv.x, lv.x);
                    eacc.add_prod(pv.y, lv.y);
                    continue;
                }
                double re = 0.0, im = 0.0;
                for (int t = 0; t < C.nterms; t++) {
                    const BPauli P = terms[C.term_off + t];
                    const uint64_t k = i ^ P.x;
                    const double2 v = St<T>::d(St<T>::ld(psi, k));
                    double cf = P.c;
                    if (__popcll(P.z & k) & 1) cf = -cf;
                    switch (__popcll(P.x & P.z) & 3) {
                        case 0: re = fma(cf, v.x, re); im = fma(cf, v.y, im); break;
                        case 1: re = fma(-cf, v.y, re); im = fma(cf, v.x, im); break;
                        case 2: re = fma(-cf, v.x, re); im = fma(-cf, v.y, im); break;
                        default: re = fma(cf, v.y, re); im = fma(-cf, v.x, im); break;
                    }
                }
                St<T>::st(lam, i, St<T>::from(make_double2(re, im)));
                const double2 pv = St<T>::d(St<T>::ld(psi, i));
                e = fma(pv.x, re, fma(pv.y, im, e));
            }
            if constexpr (sizeof(T) == 8) e = __dadd_rn(df_f2d(eacc.s), df_f2d(eacc.c));
            double dummy = 0.0;
            rd_block_sum2<kBT>(e, dummy);
            if (threadIdx.x == 0) partials[C.epart_off + j] = e;
        } else {  // a tiled stage: tiles [j * tpi, (j + 1) * tpi)
            const bool fwd = s < C.nfwd;
            const BStage S = stages[C.stage_off + (fwd ? s : s - 1)];
            const uint64_t tpi = 1ull << (C.n - C.T - C.ncht_log);
            bool done = false;
            if constexpr (DF) {
                if (S.df) {
                    batch_df(C, S, ops, cs, uint64_t(j) * tpi, tpi, fwd, smem_raw, partials, j);
                    done = true;
                }
            }
            if (!done) {
                const bool store = s + 1 < C.nsteps;  // nothing reads the vectors after the last step
                const int rb = sw_register_bits(C.T);
#define QS_B(RB)                                                                                                  \
    if (fwd)                                                                                                      \
        batch_sweep<TT, RB, false>(C, S, sweep, uint64_t(j) * tpi, tpi, store, smem_raw, partials, j);            \
    else                                                                                                          \
        batch_sweep<TT, RB, true>(C, S, sweep, uint64_t(j) * tpi, tpi, store, smem_raw, partials, j)
                if (rb == 3) {
                    QS_B(3);
                } else if (rb == 2) {
                    QS_B(2);
                } else {
                    QS_B(1);
                }
#undef QS_B
            }
        }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(counters + C.counter_off + s, 1u);
    }
}

// res[r] = sum of partials[rtab[r].x .. + rtab[r].y), in a fixed order, times weights[wtab[r]] (wtab[r] < 0: 1).
__global__ void __launch_bounds__(kBT) k_batch_reduce(const double* __restrict__ partials, const int2* __restrict__ rtab,
                                                      const int* __restrict__ wtab, const double* __restrict__ weights,
                                                      int nres, double* __restrict__ res) {
    for (int r = blockIdx.x; r < nres; r += gridDim.x) {
        const int2 t = rtab[r];
        double a = 0.0, b = 0.0;
        for (int i = threadIdx.x; i < t.y; i += kBT) a += partials[t.x + i];
        rd_block_sum2<kBT>(a, b);
        if (threadIdx.x == 0) res[r] = wtab[r] < 0 ? a : a * weights[wtab[r]];
    }
}

}  // namespace
}  // namespace qs

struct qs_batch {
    int prec = QS_PREC_C128, arith = QS_ARITH_FMA, count = 0, sms = 1, chunk_log = 12, ctas = 2;
    cudaStream_t stream = nullptr;
    unsigned char* arena = nullptr;
    qs::BCirc* dcirc = nullptr;
    qs::BStage* dstages = nullptr;
    qs::BOp* dops = nullptr;
    qs::BPauli* dterms = nullptr;
    double2* dcs = nullptr;
    uint32_t* dseg_first = nullptr;
    int4* dsegs = nullptr;
    unsigned int* dcounters = nullptr;
    double* dpart = nullptr;
    double* dres = nullptr;
    int2* drtab = nullptr;
    int* dwtab = nullptr;        // per result: coefficient whose weight it takes, -1: none
    qs::SweepRange* dranges = nullptr;
    qs::SweepPass* dpasses = nullptr;
    qs::SweepRot* drots = nullptr;
    qs::TileOp* dfixed = nullptr;
    int* drslot = nullptr;
    qs::SweepCoef* dcoefs = nullptr;
    double* dweights = nullptr;
    double* dsigmas = nullptr;
    int nprogs = 0;
    const void* kernel = nullptr;  // the k_batch instance
    int* derr = nullptr;
    unsigned int* dticket = nullptr;
    double2* hcs = nullptr;   // pinned: (cos, sin) of theta/2 per rotation
    double* hres = nullptr;   // pinned: results
    int* herr = nullptr;      // pinned
    int nsegs = 0, nres = 0, ncs = 0, ncounters = 0;
    uint32_t nitems = 0;
    size_t total_params = 0, smem = 0;
    std::vector<size_t> param_off;
    std::vector<int> cs_param;       // parameter index (global) of each rotation
    std::vector<int> res_circ_base;  // first result of each circuit
    std::vector<std::vector<int>> rot_param;  // per circuit: parameter index (local) of rotation slot r
    std::vector<qs::BCirc> hcirc;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};

namespace {

using namespace qs;

bool is_cnot(const qs_param_gate& g) {
    if (g.k != 2 || !g.matrix) return false;
    static const double c[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 0, 1, 0, 0, 1, 0};
    for (int r = 0; r < 4; r++)
        for (int cc = 0; cc < 4; cc++)
            if (g.matrix[2 * (r * 4 + cc)] != c[r * 4 + cc] || g.matrix[2 * (r * 4 + cc) + 1] != 0.0) return false;
    return true;
}

size_t al(size_t x) { return (x + 255) / 256 * 256; }

void release(qs_batch* b) {
    if (!b) return;
    struct Gone {
        ~Gone() { object_destroyed(); }
    } gone;
    if (b->stream) cudaStreamSynchronize(b->stream);
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    if (b->arena) cudaFree(b->arena);
    if (b->hcs) cudaFreeHost(b->hcs);
    if (b->hres) cudaFreeHost(b->hres);
    if (b->herr) cudaFreeHost(b->herr);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

// Chunks of step s of circuit C for the current chunk size (the H psi step counts pair chunks).
int step_chunks(const BCirc& C, int s) { return 1 << (s == C.nfwd ? C.nche_log : C.ncht_log); }

// Work-item schedule: segments (circuit, step, chunks, chunks of the previous step) by step round.
void build_schedule(qs_batch* b, std::vector<uint32_t>* first, std::vector<int4>* segs, uint64_t* nitems) {
    first->clear();
    segs->clear();
    int maxsteps = 0;
    for (const auto& c : b->hcirc) maxsteps = std::max(maxsteps, c.nsteps);
    uint64_t item = 0;
    for (int s = 0; s < maxsteps; s++)
        for (int c = 0; c < b->count; c++) {
            const BCirc& C = b->hcirc[c];
            if (s >= C.nsteps) continue;
            const int nch = step_chunks(C, s);
            first->push_back(uint32_t(item));
            segs->push_back(make_int4(c, s, nch, s > 0 ? step_chunks(C, s - 1) : 0));
            item += uint64_t(nch);
        }
    *nitems = item;
}

// Shared memory of a block: two tiles and what the batch's largest program (or a double-float stage) keeps beside
// them. By the programs in it, not their limits: a double-float batch of rotations and CNOTs has none, and three
// blocks fit an SM for two (128 circuits of 10 to 22 qubits: 332 ms with two, 280 ms with three).
size_t batch_smem(int prec, bool df, const std::vector<SweepRange>& programs) {
    int npass = 1, nrot = 1, ndiag = 1;
    for (const SweepRange& r : programs) {
        npass = std::max(npass, r.npass);
        nrot = std::max(nrot, r.nrot);
        ndiag = std::max(ndiag, r.ndiag);
    }
    if (prec == QS_PREC_C64)
        return 2 * (sizeof(float2) << kBTileMax) + SweepSide<float2>::bytes(npass, nrot, ndiag, true, kTileMaxHigh);
    size_t side = df ? (size_t(8) << kTileMaxHigh) + size_t(kBMaxRot) * (kBT / 32) * 8 : 0;
    if (!programs.empty())
        side = std::max({side, SweepSide<FxC>::bytes(npass, nrot, ndiag, true, kTileMaxHigh),
                         SweepSide<double2>::bytes(npass, nrot, ndiag, true, kTileMaxHigh)});
    return 2 * (sizeof(double2) << kBTileMax) + side;
}

cudaError_t capture(qs_batch* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec), b->exec = nullptr;
    if (b->graph) cudaGraphDestroy(b->graph), b->graph = nullptr;
    cudaStream_t s = b->stream;
    cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    if (b->ncs) cudaMemcpyAsync(b->dcs, b->hcs, sizeof(double2) * b->ncs, cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(b->dcounters, 0, sizeof(unsigned int) * b->ncounters, s);
    cudaMemsetAsync(b->dticket, 0, sizeof(unsigned int), s);
    cudaMemsetAsync(b->derr, 0, sizeof(int), s);
    const dim3 rg(uint32_t(b->sms * 2), uint32_t(b->count));
    if (b->nprogs)
        k_sweep_coefs<<<b->nprogs, 64, 0, s>>>(b->dranges, b->dpasses, b->drots, b->dcs, b->dcoefs, b->dweights,
                                              b->dsigmas);
    const BSweep sw{b->dranges, b->dpasses, b->dfixed, b->dcoefs, b->dsigmas, b->drslot};
    if (b->prec == QS_PREC_C64)
        k_batch_reset<float2><<<rg, kBT, 0, s>>>(b->dcirc);
    else
        k_batch_reset<double2><<<rg, kBT, 0, s>>>(b->dcirc);
#define QS_BATCH(T, DF)                                                                                              \
    if (b->kernel == reinterpret_cast<const void*>(k_batch<T, DF>))                                                  \
    k_batch<T, DF><<<b->sms * b->ctas, kBT, b->smem, s>>>(b->dcirc, b->dstages, b->dops, b->dterms, b->dcs, sw,      \
                                                          b->dseg_first, b->dsegs, b->nsegs, b->nitems, b->dcounters, \
                                                          b->dpart, b->dticket, b->derr)
    QS_BATCH(float2, false);
    QS_BATCH(FxC, false);
    QS_BATCH(double2, false);
    QS_BATCH(FxC, true);
    QS_BATCH(double2, true);
#undef QS_BATCH
    k_batch_reduce<<<std::min(b->nres, b->sms * 8), kBT, 0, s>>>(b->dpart, b->drtab, b->dwtab, b->dweights, b->nres,
                                                                b->dres);
    cudaMemcpyAsync(b->hres, b->dres, sizeof(double) * b->nres, cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(b->herr, b->derr, sizeof(int), cudaMemcpyDeviceToHost, s);
    e = cudaStreamEndCapture(s, &b->graph);
    if (e != cudaSuccess) return e;
    return cudaGraphInstantiate(&b->exec, b->graph, 0);
}

// Planning form of one gate (targets forced into the tile, controls free): rotations and fixed
// 1-qubit gates as dense 1-qubit gates on their target, CNOT as classified (target + control).
OpDesc plan_desc(const qs_param_gate& G, bool cnot) {
    OpDesc d;
    if (cnot) {
        classify_gate(G.matrix, 2, G.targets, &d);
        return d;
    }
    d.kind = OP_DENSE;
    d.k = d.orig_k = 1;
    d.tq[0] = int(G.targets[0]);
    d.m.assign(8, 0.0);
    d.touched_rows = 2;
    return d;
}

// The tables plan_circuit fills.
struct BTables {
    std::vector<BStage> stages;
    std::vector<BOp> ops;
    std::vector<SweepRange> ranges;
    std::vector<SweepPass> passes;
    std::vector<SweepRot> rots;
    std::vector<TileOp> fixed;
    std::vector<int> rslot;
    std::vector<int> wtab;  // per rotation slot of the circuit being planned
};

// Stages of one circuit (forward gates, then the reverse sweep) into the tables. Double-float stages hold
// rotations and CNOTs; the others become programs.
void plan_circuit(const qs_batch_circuit& q, int T, int prec, bool df_ok, bool unitary, bool fixed_point, BCirc* C,
                  const std::vector<int>& cs_of, const std::vector<int>& rslot_of, BTables* tb) {
    const int n = int(q.n);
    const int L = std::min(T, df_ok || !unitary ? 5 : prec == QS_PREC_C64 ? 4 : 3);  // rows of 128 bytes
    std::vector<char> cnot(q.m);
    for (size_t g = 0; g < q.m; g++) cnot[g] = q.gates[g].kind == QS_GATE_FIXED && q.gates[g].k == 2;
    auto emit = [&](const std::vector<int>& order, bool fwd) {
        std::vector<OpDesc> list, fixed(q.m);
        for (int g : order) {
            const qs_param_gate& G = q.gates[g];
            list.push_back(plan_desc(G, cnot[g]));
            if (G.kind != QS_GATE_FIXED) continue;
            if (cnot[g] || fwd) {
                classify_gate(G.matrix, G.k, G.targets, &fixed[g]);
            } else {  // the adjoint of a 1-qubit gate
                const double* m = G.matrix;
                const double h[8] = {m[0], -m[1], m[4], -m[5], m[2], -m[3], m[6], -m[7]};
                classify_gate(h, 1, G.targets, &fixed[g]);
            }
        }
        const std::vector<TileStage> st = plan_tiles(list, n, T, L, false, kMaxStageOps, false, !df_ok && unitary);
        int count = 0;
        for (const TileStage& S : st) {
            BStage B{};
            B.prog = -1;
            B.op_off = int(tb->ops.size());
            B.L = S.L;
            B.H = int(S.high.size());
            std::vector<int> qpos;
            for (int qb = 0; qb < S.L; qb++) qpos.push_back(qb);
            for (int qb : S.high) qpos.push_back(qb);
            std::sort(qpos.begin(), qpos.end());
            for (size_t i = 0; i < qpos.size(); i++) B.pos[i] = uint8_t(qpos[i]);
            for (int i = 0; i < B.H; i++) B.high[i] = uint8_t(S.high[i]);
            auto local = [&](int qb) -> int {
                if (qb < S.L) return qb;
                for (int i = 0; i < B.H; i++)
                    if (S.high[i] == qb) return S.L + i;
                return -1;
            };
            bool moves = df_ok;
            for (int idx : S.ops) moves = moves && (q.gates[order[idx]].kind != QS_GATE_FIXED || cnot[order[idx]]);
            if (moves) {
                B.df = 1;
                for (int idx : S.ops) {
                    const int g = order[idx];
                    const qs_param_gate& G = q.gates[g];
                    BOp o{};
                    o.cb = o.cglob = -1;
                    o.tb = local(int(G.targets[0]));
                    if (cnot[g]) {  // CNOT's matrix: targets[1] = 1 swaps the rows of targets[0]
                        o.kind = kCnot;
                        o.cb = local(int(G.targets[1]));
                        if (o.cb < 0) o.cglob = int(G.targets[1]);
                    } else {
                        o.kind = G.kind;
                        o.cs = cs_of[g];
                        o.rslot = rslot_of[g];
                        o.lrot = B.nrot++;
                    }
                    tb->ops.push_back(o);
                    B.nops++;
                }
                tb->stages.push_back(B);
                count++;
                continue;
            }
            std::vector<SweepGate> sg;
            for (int idx : S.ops) {
                SweepGate e;
                e.gate = order[idx];
                const qs_param_gate& G = q.gates[e.gate];
                if (G.kind == QS_GATE_FIXED) {
                    e.fixed = &fixed[e.gate];
                } else {
                    e.axis = G.kind;
                    e.target = int(G.targets[0]);
                }
                sg.push_back(e);
            }
            for (const SweepProgram& p : build_sweep(sg, S, fixed_point, !fwd, !unitary, &tb->fixed)) {
                B.prog = int(tb->ranges.size());
                tb->ranges.push_back(SweepRange{int(tb->passes.size()), int(p.passes.size()), int(tb->rots.size()),
                                                int(p.rots.size()), p.ndiag, !fixed_point, prec == QS_PREC_C64, 0});
                for (int g : p.rots) {
                    if (!fwd) tb->wtab[rslot_of[g]] = int(tb->rots.size());
                    tb->rots.push_back(SweepRot{cs_of[g], q.gates[g].kind});
                    tb->rslot.push_back(rslot_of[g]);
                }
                tb->passes.insert(tb->passes.end(), p.passes.begin(), p.passes.end());
                tb->stages.push_back(B);
                count++;
            }
        }
        return count;
    };
    std::vector<int> order(q.m);
    for (size_t g = 0; g < q.m; g++) order[g] = int(g);
    C->stage_off = int(tb->stages.size());
    C->nfwd = emit(order, true);
    std::reverse(order.begin(), order.end());
    const int nrev = emit(order, false);
    C->nsteps = C->nfwd + 1 + nrev;
}

}  // namespace

extern "C" int qs_batch_create(const qs_batch_circuit* circuits, size_t count, const qs_batch_options* opts,
                               qs_batch** out, size_t* err) {
    qs::TraceRange trace("qs_batch_create");
    auto fail = [&](int code, const std::string& m) {
        set_last_error_message(m);
        return code;
    };
    if (!out || !circuits || count == 0) return fail(QS_INVALID_ARGUMENT, "need at least one circuit");
    *out = nullptr;
    qs_batch_options o{};
    o.precision = QS_PREC_C128;
    o.arith = QS_ARITH_FMA;
    if (opts) o = *opts;
    if (o.precision != QS_PREC_C128 && o.precision != QS_PREC_C64) return fail(QS_INVALID_ARGUMENT, "unknown precision");
    auto* b = new qs_batch();
    object_created();
    b->prec = o.precision;
    b->arith = o.arith;
    b->count = int(count);
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, dev);
    // ---- validate and plan
    BTables tb;
    std::vector<BPauli> terms;
    std::vector<int> wtab;
    const bool df_ok = b->prec == QS_PREC_C128 && b->arith == QS_ARITH_DF64;
    bool unitary = true;  // fixed-point tiles need gates that keep norms
    for (size_t c = 0; c < count && unitary; c++)
        for (size_t g = 0; g < circuits[c].m && circuits[c].gates && unitary; g++) {
            const qs_param_gate& G = circuits[c].gates[g];
            if (G.kind == QS_GATE_FIXED && G.k == 1 && G.matrix) unitary = is_unitary(G.matrix, 1);
        }
    const bool fixed_point = b->prec == QS_PREC_C128 && sweep_fixed_point(b->arith, unitary);
    const size_t amp = b->prec == QS_PREC_C64 ? 8 : 16;
    size_t state_bytes = 0;
    int counters = 0;
    for (size_t c = 0; c < count; c++) {
        const qs_batch_circuit& q = circuits[c];
        if (q.n < 1 || q.n > 30 || (q.m && !q.gates) || (q.nterms && !q.terms)) {
            if (err) err[2] = c;
            release(b);
            return fail(QS_INVALID_ARGUMENT, "circuit " + std::to_string(c) + ": bad size or null table");
        }
        BCirc C{};
        C.n = int(q.n);
        C.T = std::min(kBTileMax, C.n);
        C.nterms = int(q.nterms);
        C.term_off = int(terms.size());
        b->param_off.push_back(b->total_params);
        b->total_params += q.nparams;
        std::vector<int> rp, cs_of(q.m, -1), rslot_of(q.m, -1);
        for (size_t g = 0; g < q.m; g++) {
            const qs_param_gate& G = q.gates[g];
            const bool rotk = G.kind == QS_GATE_RX || G.kind == QS_GATE_RY || G.kind == QS_GATE_RZ;
            if (rotk) {
                if (G.k != 1 || !G.targets || G.targets[0] >= q.n || G.param < 0 || size_t(G.param) >= q.nparams) {
                    if (err) err[0] = G.targets ? G.targets[0] : 0, err[2] = c;
                    release(b);
                    return fail(QS_INVALID_ARGUMENT, "circuit " + std::to_string(c) + " gate " + std::to_string(g) +
                                                         ": bad rotation");
                }
                cs_of[g] = int(b->cs_param.size());
                rslot_of[g] = int(rp.size());
                b->cs_param.push_back(int(b->param_off[c]) + G.param);
                rp.push_back(G.param);
            } else if (G.kind == QS_GATE_FIXED && G.k == 1 && G.matrix && G.targets && G.targets[0] < q.n) {
            } else if (G.kind == QS_GATE_FIXED && is_cnot(G) && G.targets && G.targets[0] < q.n &&
                       G.targets[1] < q.n && G.targets[0] != G.targets[1]) {
            } else {
                if (err) err[2] = c;
                release(b);
                return fail(QS_INVALID_ARGUMENT, "circuit " + std::to_string(c) + " gate " + std::to_string(g) +
                                                     ": the batch path takes rotations, 1-qubit gates and CNOTs");
            }
        }
        for (size_t t = 0; t < q.nterms; t++) {
            if ((q.terms[t].x_mask | q.terms[t].z_mask) >> q.n) {
                if (err) err[2] = c;
                release(b);
                return fail(QS_INVALID_ARGUMENT, "circuit " + std::to_string(c) + ": Pauli term acts on a qubit >= n");
            }
            const double c = q.terms[t].coeff;
            const float ch = float(c);
            terms.push_back({c, q.terms[t].x_mask, q.terms[t].z_mask, ch, float(c - double(ch)),
                             uint32_t(__builtin_popcountll(q.terms[t].x_mask & q.terms[t].z_mask) & 3), 0u});
        }
        C.nrot = int(rp.size());
        tb.wtab.assign(rp.size(), -1);
        plan_circuit(q, C.T, b->prec, df_ok, unitary, fixed_point, &C, cs_of, rslot_of, &tb);
        wtab.push_back(-1);  // the energy
        wtab.insert(wtab.end(), tb.wtab.begin(), tb.wtab.end());
        C.counter_off = counters;
        counters += C.nsteps;
        b->rot_param.push_back(rp);
        state_bytes += 2 * al((size_t(1) << q.n) * amp);
        b->hcirc.push_back(C);
    }
    b->ncs = int(b->cs_param.size());
    b->ncounters = counters;
    // partial tables depend on the chunk size; size them for the smallest candidate (2^8 pairs per item)
    const int kMinChunk = 8;
    size_t part_max = 0, max_segs = 0;
    for (const BCirc& C : b->hcirc) {
        part_max += (size_t(1) << (C.n - 1 - std::min(kMinChunk, C.n - 1))) + size_t(C.nrot) * (size_t(1) << (C.n - C.T));
        max_segs += size_t(C.nsteps);
    }
    std::vector<int2> rtab;
    for (int c = 0; c < b->count; c++) {
        b->res_circ_base.push_back(int(rtab.size()));
        for (int r = 0; r <= b->hcirc[c].nrot; r++) rtab.push_back(make_int2(0, 0));
    }
    b->nres = int(rtab.size());
    // ---- arena
    const size_t o_circ = 0, o_stages = o_circ + al(sizeof(BCirc) * count + 1),
                 o_ops = o_stages + al(sizeof(BStage) * tb.stages.size() + 1),
                 o_range = o_ops + al(sizeof(BOp) * tb.ops.size() + 1),
                 o_pass = o_range + al(sizeof(SweepRange) * tb.ranges.size() + 1),
                 o_rot = o_pass + al(sizeof(SweepPass) * tb.passes.size() + 1),
                 o_fix = o_rot + al(sizeof(SweepRot) * tb.rots.size() + 1),
                 o_rslot = o_fix + al(sizeof(TileOp) * tb.fixed.size() + 1),
                 o_coef = o_rslot + al(4 * tb.rslot.size() + 1), o_wt = o_coef + al(sizeof(SweepCoef) * tb.rots.size() + 1),
                 o_sig = o_wt + al(8 * tb.rots.size() + 8), o_wtab = o_sig + al(8 * tb.ranges.size() + 8),
                 o_terms = o_wtab + al(4 * wtab.size() + 4),
                 o_cs = o_terms + al(sizeof(BPauli) * terms.size() + 1), o_first = o_cs + al(16 * (size_t(b->ncs) + 1)),
                 o_segs = o_first + al(4 * max_segs + 4), o_ctr = o_segs + al(sizeof(int4) * max_segs + 16),
                 o_part = o_ctr + al(4 * size_t(counters) + 4), o_res = o_part + al(8 * part_max + 8),
                 o_rtab = o_res + al(8 * size_t(b->nres) + 8), o_err = o_rtab + al(8 * size_t(b->nres) + 8),
                 o_tick = o_err + 256, o_states = o_tick + 256, total = o_states + state_bytes;
    cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&b->arena, total);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        give_back_memory();
        e = cudaMalloc(&b->arena, total);
    }
    if (e == cudaSuccess) e = cudaMallocHost(&b->hcs, 16 * (size_t(b->ncs) + 1));
    if (e == cudaSuccess) e = cudaMallocHost(&b->hres, 8 * (size_t(b->nres) + 1));
    if (e == cudaSuccess) e = cudaMallocHost(&b->herr, sizeof(int));
    if (e == cudaSuccess) *b->herr = 0;  // page-locked memory comes uninitialised; read even when no run precedes
    b->smem = batch_smem(b->prec, df_ok, tb.ranges);
    b->nprogs = int(tb.ranges.size());
    b->kernel = b->prec == QS_PREC_C64 ? reinterpret_cast<const void*>(k_batch<float2, false>)
                : df_ok ? (fixed_point ? reinterpret_cast<const void*>(k_batch<FxC, true>)
                                       : reinterpret_cast<const void*>(k_batch<double2, true>))
                        : (fixed_point ? reinterpret_cast<const void*>(k_batch<FxC, false>)
                                       : reinterpret_cast<const void*>(k_batch<double2, false>));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(b->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(b->smem));
    if (e != cudaSuccess) {
        release(b);
        return fail(e == cudaErrorMemoryAllocation ? QS_OUT_OF_MEMORY : QS_CUDA_ERROR,
                    std::string("batch allocation: ") + cudaGetErrorString(e));
    }
    unsigned char* A = b->arena;
    b->dcirc = reinterpret_cast<BCirc*>(A + o_circ);
    b->dstages = reinterpret_cast<BStage*>(A + o_stages);
    b->dops = reinterpret_cast<BOp*>(A + o_ops);
    b->dterms = reinterpret_cast<BPauli*>(A + o_terms);
    b->dcs = reinterpret_cast<double2*>(A + o_cs);
    b->dseg_first = reinterpret_cast<uint32_t*>(A + o_first);
    b->dsegs = reinterpret_cast<int4*>(A + o_segs);
    b->dcounters = reinterpret_cast<unsigned int*>(A + o_ctr);
    b->dpart = reinterpret_cast<double*>(A + o_part);
    b->dres = reinterpret_cast<double*>(A + o_res);
    b->drtab = reinterpret_cast<int2*>(A + o_rtab);
    b->dranges = reinterpret_cast<SweepRange*>(A + o_range);
    b->dpasses = reinterpret_cast<SweepPass*>(A + o_pass);
    b->drots = reinterpret_cast<SweepRot*>(A + o_rot);
    b->dfixed = reinterpret_cast<TileOp*>(A + o_fix);
    b->drslot = reinterpret_cast<int*>(A + o_rslot);
    b->dcoefs = reinterpret_cast<SweepCoef*>(A + o_coef);
    b->dweights = reinterpret_cast<double*>(A + o_wt);
    b->dsigmas = reinterpret_cast<double*>(A + o_sig);
    b->dwtab = reinterpret_cast<int*>(A + o_wtab);
    b->derr = reinterpret_cast<int*>(A + o_err);
    b->dticket = reinterpret_cast<unsigned int*>(A + o_tick);
    size_t off = o_states;
    for (auto& C : b->hcirc) {
        C.psi = reinterpret_cast<unsigned long long>(A + off);
        off += al((size_t(1) << C.n) * amp);
        C.lam = reinterpret_cast<unsigned long long>(A + off);
        off += al((size_t(1) << C.n) * amp);
    }
    // per chunk size (2^cl amplitude pairs per item): chunk counts, partial offsets, result table,
    // schedule
    auto layout = [&](int cl) {
        int part = 0;
        std::vector<int2> rt;
        for (auto& C : b->hcirc) {
            C.nche_log = C.n - 1 - std::min(cl, C.n - 1);
            C.ncht_log = (C.n - C.T) - std::min(C.n - C.T, std::max(0, cl + 1 - C.T));
            C.epart_off = part;
            part += 1 << C.nche_log;
            C.rpart_off = part;
            rt.push_back(make_int2(C.epart_off, 1 << C.nche_log));
            for (int r = 0; r < C.nrot; r++) rt.push_back(make_int2(C.rpart_off + (r << C.ncht_log), 1 << C.ncht_log));
            part += C.nrot << C.ncht_log;
        }
        std::vector<uint32_t> first;
        std::vector<int4> segs;
        uint64_t n = 0;
        build_schedule(b, &first, &segs, &n);
        b->nsegs = int(segs.size());
        b->nitems = uint32_t(n);
        b->chunk_log = cl;
        cudaError_t e2 = cudaMemcpy(b->dcirc, b->hcirc.data(), sizeof(BCirc) * count, cudaMemcpyHostToDevice);
        if (e2 == cudaSuccess && !rt.empty())
            e2 = cudaMemcpy(b->drtab, rt.data(), sizeof(int2) * rt.size(), cudaMemcpyHostToDevice);
        if (e2 == cudaSuccess) e2 = cudaMemcpy(b->dseg_first, first.data(), first.size() * 4, cudaMemcpyHostToDevice);
        if (e2 == cudaSuccess)
            e2 = cudaMemcpy(b->dsegs, segs.data(), segs.size() * sizeof(int4), cudaMemcpyHostToDevice);
        return e2;
    };
    auto put = [&](void* to, const void* from, size_t bytes) {
        if (e == cudaSuccess && bytes) e = cudaMemcpy(to, from, bytes, cudaMemcpyHostToDevice);
    };
    put(b->dstages, tb.stages.data(), sizeof(BStage) * tb.stages.size());
    put(b->dops, tb.ops.data(), sizeof(BOp) * tb.ops.size());
    put(b->dranges, tb.ranges.data(), sizeof(SweepRange) * tb.ranges.size());
    put(b->dpasses, tb.passes.data(), sizeof(SweepPass) * tb.passes.size());
    put(b->drots, tb.rots.data(), sizeof(SweepRot) * tb.rots.size());
    put(b->dfixed, tb.fixed.data(), sizeof(TileOp) * tb.fixed.size());
    put(b->drslot, tb.rslot.data(), 4 * tb.rslot.size());
    put(b->dwtab, wtab.data(), 4 * wtab.size());
    if (e == cudaSuccess && !terms.empty())
        e = cudaMemcpy(b->dterms, terms.data(), sizeof(BPauli) * terms.size(), cudaMemcpyHostToDevice);
    for (int i = 0; i < b->ncs; i++) b->hcs[i] = make_double2(1.0, 0.0);
    // ---- chunk size and persistence: from options, the autotune cache, or by timing candidates
    int max_per_sm = 1;
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&max_per_sm, b->kernel, kBT, b->smem);
    max_per_sm = std::max(1, max_per_sm);
    std::ostringstream key;
    // the tile type: 0 fixed point or complex64, 1 with double-float stages, 2 FP64
    const int form = df_ok ? 1 : b->prec == QS_PREC_C128 && !fixed_point ? 2 : 0;
    key << "batch3:p" << b->prec << ":a" << form << ":c" << count << ":items";
    {
        uint64_t sig = 0;
        for (size_t c = 0; c < count; c++) sig = sig * 1315423911ull + uint64_t(circuits[c].n) * 131 + circuits[c].m;
        key << sig;
    }
    int cl = o.chunk_log2, ct = o.ctas_per_sm;
    if (cl <= 0 || ct <= 0) {
        int ccl = 0, cct = 0;
        if (autotune_cache_lookup(key.str(), &ccl, &cct)) {
            if (cl <= 0) cl = ccl;
            if (ct <= 0) ct = cct;
        }
    }
    if (e == cudaSuccess && (cl <= 0 || ct <= 0)) {
        // autotune by coordinate descent: the chunk size (items of 1, 4 or 16 tiles of 2^11
        // amplitudes) at the most CTAs per SM, then the CTAs per SM at that chunk size. One timed run
        // per candidate, its graph uploaded first; one untimed run before the first (module loading).
        bool warmed = false;
        auto run = [&](int tcl, int tct, double* dt) -> cudaError_t {
            b->ctas = tct;
            cudaError_t r = layout(std::max(kMinChunk, tcl));
            if (r == cudaSuccess) r = capture(b);
            if (r == cudaSuccess) r = cudaGraphUpload(b->exec, b->stream);
            if (r == cudaSuccess && !warmed) {
                r = cudaGraphLaunch(b->exec, b->stream);
                if (r == cudaSuccess) note_launches(b->nprogs ? 4 : 3);
                warmed = true;
            }
            if (r == cudaSuccess) r = cudaStreamSynchronize(b->stream);
            if (r != cudaSuccess) return r;
            const auto t0 = std::chrono::steady_clock::now();
            r = cudaGraphLaunch(b->exec, b->stream);
            if (r == cudaSuccess) r = cudaStreamSynchronize(b->stream);
            if (r == cudaSuccess) note_launches(b->nprogs ? 4 : 3);
            *dt = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
            return r;
        };
        double best = 1e30;
        int bcl = cl > 0 ? cl : 12, bct = ct > 0 ? ct : max_per_sm;
        const int first_ct = bct;
        const std::vector<int> cls = cl > 0 ? std::vector<int>{cl} : std::vector<int>{10, 12, 14};
        for (int tcl : cls) {
            double dt = 0;
            if ((e = run(tcl, first_ct, &dt)) != cudaSuccess || *b->herr) break;
            if (dt < best) best = dt, bcl = tcl;
        }
        if (e == cudaSuccess && !*b->herr && ct <= 0) {
            for (int tct = 1; tct <= max_per_sm; tct++) {
                if (tct == first_ct) continue;
                double dt = 0;
                if ((e = run(bcl, tct, &dt)) != cudaSuccess || *b->herr) break;
                if (dt < best) best = dt, bct = tct;
            }
        }
        cl = bcl;
        ct = bct;
        if (e == cudaSuccess && !*b->herr) autotune_cache_store(key.str(), cl, ct);
    }
    b->ctas = std::max(1, std::min(ct, max_per_sm));
    if (e == cudaSuccess) e = layout(std::max(kMinChunk, cl));
    if (e == cudaSuccess) e = capture(b);
    if (e != cudaSuccess) {
        release(b);
        return fail(QS_CUDA_ERROR, std::string("batch setup: ") + cudaGetErrorString(e));
    }
    if (*b->herr) {
        release(b);
        return fail(QS_TIMEOUT, "batch setup: a dependency wait gave up");
    }
    *out = b;
    return QS_OK;
}

extern "C" int qs_batch_run(qs_batch* b, const double* params, double* energies, double* grads) {
    qs::TraceRange trace("qs_batch_run");
    if (!b || (b->total_params && !params)) {
        set_last_error_message("null argument");
        return QS_INVALID_ARGUMENT;
    }
    std::vector<char> undefined(size_t(b->count), 0);  // circuits with a rotation by an infinity or NaN
    for (int c = 0, i = 0; c < b->count; c++)
        for (size_t r = 0; r < b->rot_param[c].size(); r++, i++) {
            const double th = params[b->cs_param[i]];
            double2 cs = make_double2(std::cos(0.5 * th), std::sin(0.5 * th));
            if (!(std::isfinite(cs.x) && std::isfinite(cs.y))) {  // fixed-point tiles have no NaN: the results get it below
                undefined[c] = 1;
                cs = make_double2(1.0, 0.0);
            }
            b->hcs[i] = cs;
        }
    cudaError_t e = cudaGraphLaunch(b->exec, b->stream);
    if (e == cudaSuccess) note_launches(b->nprogs ? 4 : 3);  // the graph's coefficient, reset, persistent and reduction kernels
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
    if (e != cudaSuccess) {
        set_last_error_message(std::string("batch run: ") + cudaGetErrorString(e));
        return QS_CUDA_ERROR;
    }
    if (*b->herr) {
        set_last_error_message("batch run: a dependency wait in the persistent kernel gave up");
        return QS_TIMEOUT;
    }
    for (int c = 0; c < b->count; c++) {
        const int base = b->res_circ_base[c];
        if (undefined[c])
            std::fill(b->hres + base, b->hres + base + 1 + b->rot_param[c].size(), std::numeric_limits<double>::quiet_NaN());
        if (energies) energies[c] = b->hres[base];
        if (grads) {
            const size_t po = b->param_off[c];
            const size_t np = (size_t(c + 1) < b->param_off.size() ? b->param_off[c + 1] : b->total_params) - po;
            for (size_t p = 0; p < np; p++) grads[po + p] = 0.0;
            for (size_t r = 0; r < b->rot_param[c].size(); r++) grads[po + b->rot_param[c][r]] += b->hres[base + 1 + r];
        }
    }
    return QS_OK;
}

extern "C" int qs_batch_config(const qs_batch* b, int* chunk_log2, int* ctas_per_sm) {
    if (!b) return QS_INVALID_ARGUMENT;
    if (chunk_log2) *chunk_log2 = b->chunk_log;
    if (ctas_per_sm) *ctas_per_sm = b->ctas;
    return QS_OK;
}

extern "C" void qs_batch_free(qs_batch* b) { release(b); }
