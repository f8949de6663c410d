// qs_adjoint.cu — inner products, Pauli-sum expectation values and adjoint gradients.
//
// No counterpart in the reference (Quaru has no observables or gradients).
// The adjoint method follows Jones & Gacon, "Efficient calculation of
// gradients in classical simulations of variational quantum algorithms"
// (arXiv:2009.02823): psi = U_m...U_1 psi_0, lambda = H psi; walking the
// gates backwards, a rotation R_A(theta) = exp(-i theta A/2) contributes
// dE/dtheta = Im<lambda|A|psi> (both taken after the gate) and is then
// un-applied from both vectors, so no intermediate state is stored.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <string>
#include <vector>

#include "qs_adjoint.h"
#include "qs_circuit.h"
#include "qs_device.cuh"
#include "qs_kernels.h"
#include "qs_pass.cuh"
#include "qs_rot.cuh"
#include "qs_reduce.cuh"
#include "qs_sweep.cuh"
#include "qs_sweep.h"
#include "qs_tile.h"

namespace qs {

constexpr int kAT = 256;

__device__ __forceinline__ double2 ld2(const double2* p, uint64_t i) { return p[i]; }
__device__ __forceinline__ double2 ld2(const float2* p, uint64_t i) {  // integer-pipe conversion
    const float2 v = p[i];
    return make_double2(df_f2d(v.x), df_f2d(v.y));
}
__device__ __forceinline__ void st2(double2* p, uint64_t i, double2 v) { p[i] = v; }
__device__ __forceinline__ void st2(float2* p, uint64_t i, double2 v) { p[i] = make_float2(float(v.x), float(v.y)); }

static int grid_for_pairs(uint64_t work, int sms) {
    uint64_t b = (work + kAT - 1) / kAT;
    return int(std::max<uint64_t>(1, std::min<uint64_t>(b, uint64_t(sms) * 16)));
}

// ---------------------------------------------------------------- <a|b>
template <typename TA, typename TB>
__global__ void __launch_bounds__(kAT) k_inner(const TA* __restrict__ a, const TB* __restrict__ b, uint64_t N,
                                               double* __restrict__ partials) {
    double re = 0.0, im = 0.0;
    for (uint64_t i = uint64_t(blockIdx.x) * kAT + threadIdx.x; i < N; i += uint64_t(gridDim.x) * kAT) {
        const double2 x = ld2(a, i), y = ld2(b, i);
        re = fma(x.x, y.x, fma(x.y, y.y, re));
        im = fma(x.x, y.y, fma(-x.y, y.x, im));
    }
    rd_block_sum2<kAT>(re, im);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = re;
        partials[2 * blockIdx.x + 1] = im;
    }
}

__global__ void __launch_bounds__(kAT) k_pair_final(const double* __restrict__ partials, int nblocks,
                                                    double* __restrict__ out) {
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < nblocks; i += kAT) {
        a += partials[2 * i];
        b += partials[2 * i + 1];
    }
    rd_block_sum2<kAT>(a, b);
    if (threadIdx.x == 0) {
        out[0] = a;
        out[1] = b;
    }
}

// ---------------------------------------------------------------- H psi
struct PauliDev {
    double c;
    uint64_t x, z;
    float ch, cl;  // c as a float pair, c = ch + cl + O(2^-48 |c|)
    uint32_t cls;  // |x & z| mod 4: the term's factor i^cls
    uint32_t pad_;
};

// out_i = sum_t c_t * i^{|x&z|} * (-1)^{|z & (i^x)|} * psi_{i^x}, and the block's part of Re <psi|out> (out as
// it is stored). A pass of its own for the inner product read both vectors again: 25 us at 20 qubits, and two more
// links in the chain of launches that a gradient of a small state waits for.
template <typename T, bool DFC>
__global__ void __launch_bounds__(kAT) k_pauli_sum(const T* __restrict__ psi, T* __restrict__ out, uint64_t N,
                                                   const PauliDev* __restrict__ terms, int nt,
                                                   double* __restrict__ partials) {
    double energy = 0.0, none = 0.0;
    auto put = [&](uint64_t i, T v) {
        out[i] = v;
        const double2 a = ld2(psi, i), b = ld2(&v, 0);
        energy = fma(a.x, b.x, fma(a.y, b.y, energy));
    };
    // the parity of z & j: the qubits of most states fit one word
    const bool narrow = N <= (1ull << 32);
    auto odd = [&](uint64_t zj) { return ((narrow ? __popc(uint32_t(zj)) : __popcll(zj)) & 1) != 0; };
    static_assert(!DFC || sizeof(T) == 8, "float-pair coefficients serve complex64 states");
    if constexpr (DFC) {
        // complex64: each term's product by TwoProduct on the FP32 pipe, summed with TwoSum (DfAcc), the
        // coefficient's low float folded into the compensation; one rounding to float at the end
        for (uint64_t i = uint64_t(blockIdx.x) * kAT + threadIdx.x; i < N; i += uint64_t(gridDim.x) * kAT) {
            DfAcc re, im;
            for (int t = 0; t < nt; t++) {
                const PauliDev& p = terms[t];
                const uint64_t j = i ^ p.x;
                const float2 v = reinterpret_cast<const float2*>(psi)[j];
                const bool neg = odd(p.z & j);
                const float ch = neg ? -p.ch : p.ch, cl = neg ? -p.cl : p.cl;
                float xr, xi;  // i^cls * v
                switch (p.cls) {
                    case 0: xr = v.x; xi = v.y; break;
                    case 1: xr = -v.y; xi = v.x; break;
                    case 2: xr = -v.x; xi = -v.y; break;
                    default: xr = v.y; xi = -v.x; break;
                }
                re.add_prod(ch, xr);
                re.c = __fmaf_rn(cl, xr, re.c);
                im.add_prod(ch, xi);
                im.c = __fmaf_rn(cl, xi, im.c);
            }
            put(i, make_float2(__fadd_rn(re.s, re.c), __fadd_rn(im.s, im.c)));
        }
    } else {
        for (uint64_t i = uint64_t(blockIdx.x) * kAT + threadIdx.x; i < N; i += uint64_t(gridDim.x) * kAT) {
            double re = 0.0, im = 0.0;
            for (int t = 0; t < nt; t++) {
                const PauliDev p = terms[t];
                const uint64_t j = i ^ p.x;
                const double2 v = ld2(psi, j);
                double c = p.c;
                if (odd(p.z & j)) c = -c;
                switch (p.cls) {
                    case 0: re = fma(c, v.x, re); im = fma(c, v.y, im); break;
                    case 1: re = fma(-c, v.y, re); im = fma(c, v.x, im); break;  // i * v
                    case 2: re = fma(-c, v.x, re); im = fma(-c, v.y, im); break;
                    default: re = fma(c, v.y, re); im = fma(-c, v.x, im); break;  // -i * v
                }
            }
            T v;
            st2(&v, 0, make_double2(re, im));
            put(i, v);
        }
    }
    rd_block_sum2<kAT>(energy, none);
    if (threadIdx.x == 0) partials[blockIdx.x] = energy;
}

// Block 0 sums the nenergy partials of the energy into out[0]; block g + 1 sums partials[g * nblocks ..
// (g + 1) * nblocks) into out[g + 1], times weights[at[g]] (at[g] < 0: 1).
__global__ void __launch_bounds__(kAT) k_grad_final(const double* __restrict__ energy, int nenergy,
                                                    const double* __restrict__ partials, int nblocks,
                                                    const double* __restrict__ weights, const int* __restrict__ at,
                                                    double* __restrict__ out) {
    const int g = int(blockIdx.x) - 1, count = g < 0 ? nenergy : nblocks;
    const double* p = g < 0 ? energy : partials + size_t(g) * nblocks;
    double a = 0.0, b = 0.0;
    for (int i = threadIdx.x; i < count; i += kAT) a += p[i];
    rd_block_sum2<kAT>(a, b);
    if (threadIdx.x == 0) out[blockIdx.x] = g < 0 || at[g] < 0 ? a : a * weights[at[g]];
}

// ---------------------------------------------------------------- tiled sweeps
// The forward run and the reverse walk as launches of stage programs (qs_sweep.h): a block takes its
// tiles of 2^T amplitudes (psi; in the reverse walk psi and lambda side by side) through the program's
// passes in shared memory. The reverse walk takes the gates backwards, a rotation adding
// Im<lambda|A|psi> over the tile to its slot before it is un-applied from both vectors. Gates were
// reordered only past gates on disjoint qubits, with which they commute, so every inner product equals
// the one of the gate-by-gate walk.
struct SweepArgs {
    int RH, pass0, coef0, prog;   // 2^RH tile rows; first pass, first coefficient and index of the program
    SweepTile t;
    IndexMap outer;
    uint8_t rhigh[kTileMaxHigh];
    int slot[kSwMaxRot];          // global slot of each program-local rotation
};

template <int RB>
constexpr int sweep_threads() {
    return RB == 3 ? 256 : 128;  // the largest tile that takes RB register bits
}
// src: psi as the launch finds it (the register's own state in the first launch, which is not written; psi itself in
// the others, so neither is __restrict__).
// Blocks per SM: two complex128 tile pairs fill the shared memory; complex64 tiles gain more from a third
// block's warps (80 registers) than from free registers (20-qubit gradient 1.81 against 1.89 ms).
template <typename T, int RB, bool REV>
__global__ void __launch_bounds__(sweep_threads<RB>(), RB < 3 ? 4 : sizeof(T) == 16 ? 2 : REV ? 3 : 4)
    k_sweep(const typename Sw<T>::Glob* src, typename Sw<T>::Glob* psi, typename Sw<T>::Glob* lam, uint64_t ntiles,
            const __grid_constant__ SweepArgs a, const SweepPass* __restrict__ passes,
            const TileOp* __restrict__ fixed, const SweepCoef* __restrict__ coef, const double* __restrict__ sigmas,
            double* __restrict__ partials) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nt = blockDim.x;
    SweepTile t = a.t;
    t.sigma = sigmas[a.prog];
    T* sp = reinterpret_cast<T*>(smem_raw);
    T* sl = sp + (REV ? 1u << t.T : 0u);
    const SweepSide<T> side(reinterpret_cast<unsigned char*>(sl + (1u << t.T)), t.npass, t.nrot, t.ndiag, REV);
    for (int r = threadIdx.x; r < (1 << a.RH); r += nt) {
        uint64_t o = 0;
        for (int b = 0; b < a.RH; b++)
            if (r >> b & 1) o |= 1ull << a.rhigh[b];
        side.rowoff[r] = o;
    }
    sw_begin<T>(side, passes + a.pass0, t.npass, coef + a.coef0, t.nrot, t.T, REV, t.sigma, nt);
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
        sw_tile<T, RB, REV, false>(src, psi, lam, expand_index(tile, a.outer), t, sp, sl, side, fixed, nt);
    if (REV)
        for (int r = threadIdx.x; r < t.nrot; r += nt)
            partials[size_t(a.slot[r]) * gridDim.x + blockIdx.x] = sw_total<T>(side, r, nt);
}

// ---------------------------------------------------------------- double-float reverse sweep
// Stages of rotations and pure moves on complex128 registers in QS_ARITH_DF64: psi and lambda tiles as
// double-float values, one gate after another.
constexpr int kAdjT = 11;           // tile qubits of the sweeps (largest; see adj_tile_qubits)
constexpr int kAdjThreads = 256;
constexpr int kAdjMaxOps = 32;      // gates per stage: the op table is staged in shared memory

struct AdjOpDev {
    TileOp t;      // tile-local form (target bit, tuple expansion, controls)
    int rot;       // stage-local rotation slot, or -1 for a fixed gate
    int axis;      // QS_GATE_RX / RY / RZ
    double c, s;   // cos(theta/2), -sin(theta/2): the inverse rotation
};

static_assert(sizeof(AdjOpDev) % 16 == 0, "the op table is copied to shared memory in 16-byte words");

struct AdjStageArgs {
    int T, RL, RH;
    int nops, nrot;
    IndexMap outer;
    uint8_t rhigh[kTileMaxHigh];
    int slot[kAdjMaxOps];  // global rotation slot of each stage-local slot
};

template <int AXIS>
__device__ __forceinline__ DfAcc adj_rot_tile_df(float4* sp, float4* sl, const AdjOpDev& op, uint32_t tsize) {
    const TileOp& t = op.t;
    uint32_t seg[5];
#pragma unroll
    for (int j = 0; j < 5; j++) seg[j] = t.seg[j];
    const uint32_t tb = 1u << t.tb[0];
    float ch, cl, sh, sl_;
    df_split(op.c, ch, cl);
    df_split(op.s, sh, sl_);
    DfAcc acc;
    for (uint32_t p = threadIdx.x; p < (tsize >> 1); p += kAdjThreads) {
        const uint32_t i0 = tuple_index(p, t.npos, seg, t.pos, 0u), i1 = i0 | tb;
        float4 a = sp[i0], b = sp[i1], l0 = sl[i0], l1 = sl[i1];
        adj_im_df_acc<AXIS>(acc, l0, l1, a, b);
        df_rot_pair<AXIS>(ch, cl, sh, sl_, a, b);
        df_rot_pair<AXIS>(ch, cl, sh, sl_, l0, l1);
        sp[i0] = a;
        sp[i1] = b;
        sl[i0] = l0;
        sl[i1] = l1;
    }
    return acc;
}

// pure moves (permutations with factors 1, -1, i, -i) on double-float amplitudes
__device__ __forceinline__ float4 df_pf(float4 x, uint8_t c) {
    if (c == 1) return make_float4(-x.x, -x.y, -x.z, -x.w);
    if (c == 2) return make_float4(-x.z, -x.w, x.x, x.y);
    if (c == 3) return make_float4(x.z, x.w, -x.x, -x.y);
    return x;
}

__device__ __forceinline__ void adj_move_df(float4* s, const TileOp& op, uint32_t tsize) {
    const uint32_t ntup = tsize >> op.npos;
    uint32_t seg[5];
#pragma unroll
    for (int j = 0; j < 5; j++) seg[j] = op.seg[j];
    const int D = 1 << op.k;
    for (uint32_t p = threadIdx.x; p < ntup; p += kAdjThreads) {
        const uint32_t i0 = tuple_index(p, op.npos, seg, op.pos, op.lfixval);
        float4 y[8];
#pragma unroll
        for (int r = 0; r < 8; r++)
            if (r < D && op.pf[r] != PF_SKIP_DEV) y[r] = s[i0 + op.offsrc[r]];
#pragma unroll
        for (int r = 0; r < 8; r++)
            if (r < D && op.pf[r] != PF_SKIP_DEV) s[i0 + op.off[r]] = df_pf(y[r], op.pf[r]);
    }
}

__global__ void __launch_bounds__(kAdjThreads) k_adj_stage_df(double2* __restrict__ psi, double2* __restrict__ lam,
                                                              uint64_t ntiles, const __grid_constant__ AdjStageArgs a,
                                                              const AdjOpDev* __restrict__ ops,
                                                              double* __restrict__ partials) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t tsize = 1u << a.T;
    float4* fp = reinterpret_cast<float4*>(smem_raw);
    float4* fl = fp + tsize;
    double* sacc = reinterpret_cast<double*>(fl + tsize);  // [nrot][8 warps]
    AdjOpDev* sops = reinterpret_cast<AdjOpDev*>(sacc + size_t(a.nrot) * (kAdjThreads / 32));
    uint64_t* rowoff = reinterpret_cast<uint64_t*>(sops + a.nops);
    const int nrows = 1 << a.RH, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < a.nrot * (kAdjThreads / 32); i += kAdjThreads) sacc[i] = 0.0;
    {  // the launch's op table, read by every thread for every gate of every tile
        const uint4* src = reinterpret_cast<const uint4*>(ops);
        uint4* dst = reinterpret_cast<uint4*>(sops);
        const int words = a.nops * int(sizeof(AdjOpDev) / 16);
        for (int w = threadIdx.x; w < words; w += kAdjThreads) dst[w] = src[w];
    }
    for (int r = threadIdx.x; r < nrows; r += kAdjThreads) {
        uint64_t o = 0;
        for (int b = 0; b < a.RH; b++)
            if (r >> b & 1) o |= 1ull << a.rhigh[b];
        rowoff[r] = o;
    }
    __syncthreads();
    const uint32_t rmask = (1u << a.RL) - 1u;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const uint64_t base = expand_index(tile, a.outer);
        for (uint32_t i = threadIdx.x; i < tsize; i += kAdjThreads) {
            const uint64_t g = base + rowoff[i >> a.RL] + (i & rmask);
            const double2 v = psi[g], w = lam[g];
            float4 f;
            df_split(v.x, f.x, f.y);
            df_split(v.y, f.z, f.w);
            fp[i] = f;
            df_split(w.x, f.x, f.y);
            df_split(w.y, f.z, f.w);
            fl[i] = f;
        }
        __syncthreads();
        for (int o = 0; o < a.nops; o++) {
            const AdjOpDev& op = sops[o];
            if ((base & op.t.omask) != op.t.oval) continue;  // the same for the whole block
            if (op.rot >= 0) {  // the warp's float pairs reduced on the FP32 pipe, one FP64 rejoin
                DfAcc f;
                if (op.axis == QS_GATE_RX)
                    f = adj_rot_tile_df<QS_GATE_RX>(fp, fl, op, tsize);
                else if (op.axis == QS_GATE_RY)
                    f = adj_rot_tile_df<QS_GATE_RY>(fp, fl, op, tsize);
                else
                    f = adj_rot_tile_df<QS_GATE_RZ>(fp, fl, op, tsize);
                f.warp_reduce();
                const double v = __dadd_rn(df_f2d(f.s), df_f2d(f.c));
                if (lane == 0) sacc[op.rot * (kAdjThreads / 32) + warp] += v;
            } else {
                adj_move_df(fp, op.t, tsize);
                adj_move_df(fl, op.t, tsize);
            }
            __syncthreads();
        }
        for (uint32_t i = threadIdx.x; i < tsize; i += kAdjThreads) {
            const uint64_t g = base + rowoff[i >> a.RL] + (i & rmask);
            const float4 f = fp[i], h = fl[i];
            psi[g] = make_double2(__dadd_rn(df_f2d(f.x), df_f2d(f.y)), __dadd_rn(df_f2d(f.z), df_f2d(f.w)));
            lam[g] = make_double2(__dadd_rn(df_f2d(h.x), df_f2d(h.y)), __dadd_rn(df_f2d(h.z), df_f2d(h.w)));
        }
        __syncthreads();
    }
    for (int r = threadIdx.x; r < a.nrot; r += kAdjThreads) {
        double v = 0.0;
        for (int w = 0; w < kAdjThreads / 32; w++) v += sacc[r * (kAdjThreads / 32) + w];
        partials[size_t(a.slot[r]) * gridDim.x + blockIdx.x] = v;
    }
}

// ---------------------------------------------------------------- host side
static int fail(cudaError_t e, const char* what, std::string* msg) {
    if (msg) *msg = std::string(what) + ": " + cudaGetErrorString(e);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return QS_OUT_OF_MEMORY;
    }
    return QS_CUDA_ERROR;
}

#define AJ_CHECK(call, what)                            \
    do {                                                \
        cudaError_t e_ = (call);                        \
        if (e_ != cudaSuccess) { rc = fail(e_, what, msg); goto done; } \
    } while (0)

int inner_product(const void* a, int pa, const void* b, int pb, int n, cudaStream_t s, int sms, double* scratch,
                  double* out2) {
    const uint64_t N = 1ull << n;
    const int grid = std::min(grid_for_pairs(N, sms), 4096);
    if (pa == QS_PREC_C128 && pb == QS_PREC_C128)
        k_inner<double2, double2><<<grid, kAT, 0, s>>>((const double2*)a, (const double2*)b, N, scratch);
    else if (pa == QS_PREC_C128)
        k_inner<double2, float2><<<grid, kAT, 0, s>>>((const double2*)a, (const float2*)b, N, scratch);
    else if (pb == QS_PREC_C128)
        k_inner<float2, double2><<<grid, kAT, 0, s>>>((const float2*)a, (const double2*)b, N, scratch);
    else
        k_inner<float2, float2><<<grid, kAT, 0, s>>>((const float2*)a, (const float2*)b, N, scratch);
    k_pair_final<<<1, kAT, 0, s>>>(scratch, grid, out2);
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) note_launches(2);
    return e == cudaSuccess ? QS_OK : QS_CUDA_ERROR;
}

static std::vector<PauliDev> pauli_table(const qs_pauli_term* terms, size_t nt) {
    std::vector<PauliDev> v(nt);
    for (size_t t = 0; t < nt; t++) {
        const double c = terms[t].coeff;
        const float ch = float(c);
        v[t] = {c, terms[t].x_mask, terms[t].z_mask, ch, float(c - double(ch)),
                uint32_t(__builtin_popcountll(terms[t].x_mask & terms[t].z_mask) & 3), 0u};
    }
    return v;
}

// Whether every coefficient lies where its float pair carries it to FP64 accuracy.
static bool pauli_df_ok(const std::vector<PauliDev>& ht) {
    for (const PauliDev& p : ht) {
        const double a = std::fabs(p.c);
        if (a != 0.0 && !(a >= 0x1p-90 && a <= 0x1p90)) return false;
    }
    return true;
}

// Returns the number of blocks: partials of the energy written (at most 16 per SM).
template <typename T>
static int launch_pauli_sum(const void* psi, void* out, int n, const PauliDev* dterms, int nt, bool df_ok,
                            double* partials, cudaStream_t s, int sms) {
    const uint64_t N = 1ull << n;
    const int grid = grid_for_pairs(N, sms);
    if (sizeof(T) == 8 && df_ok)
        k_pauli_sum<float2, true>
            <<<grid, kAT, 0, s>>>((const float2*)psi, (float2*)out, N, dterms, nt, partials);
    else
        k_pauli_sum<T, false><<<grid, kAT, 0, s>>>((const T*)psi, (T*)out, N, dterms, nt, partials);
    note_launches(1);
    return grid;
}

int expval_pauli(const void* psi, int prec, int n, const qs_pauli_term* terms, size_t nt, cudaStream_t s, int sms,
                 double* value, std::string* msg) {
    const size_t amp = prec == QS_PREC_C64 ? 8 : 16;
    const uint64_t N = 1ull << n;
    int rc = QS_OK;
    unsigned char* blob = nullptr;
    const size_t o_terms = 0, o_part = ((nt * sizeof(PauliDev) + 255) / 256) * 256, o_res = o_part + 4096 * 16,
                 o_lam = o_res + 256, total = o_lam + N * amp;
    std::vector<PauliDev> ht = pauli_table(terms, nt);
    double res = 0.0;
    int blocks = 0;
    AJ_CHECK(device_alloc((void**)&blob, total, s), "expval buffers");
    if (nt) AJ_CHECK(cudaMemcpyAsync(blob + o_terms, ht.data(), nt * sizeof(PauliDev), cudaMemcpyHostToDevice, s),
                     "terms upload");
    if (prec == QS_PREC_C64)
        blocks = launch_pauli_sum<float2>(psi, blob + o_lam, n, (const PauliDev*)(blob + o_terms), int(nt),
                                          pauli_df_ok(ht), (double*)(blob + o_part), s, sms);
    else
        blocks = launch_pauli_sum<double2>(psi, blob + o_lam, n, (const PauliDev*)(blob + o_terms), int(nt), false,
                                           (double*)(blob + o_part), s, sms);
    AJ_CHECK(cudaGetLastError(), "pauli sum");
    k_grad_final<<<1, kAT, 0, s>>>((const double*)(blob + o_part), blocks, nullptr, 0, nullptr, nullptr,
                                   (double*)(blob + o_res));
    note_launches(1);
    AJ_CHECK(cudaGetLastError(), "energy");
    AJ_CHECK(cudaMemcpyAsync(&res, blob + o_res, sizeof(res), cudaMemcpyDeviceToHost, s), "expval readback");
    AJ_CHECK(cudaStreamSynchronize(s), "expval sync");
    *value = res;
done:
    if (blob) cudaFreeAsync(blob, s);
    return rc;
}

// R_A(theta) as a row-major interleaved 2x2 matrix.
static std::vector<double> rotation_matrix(int axis, double c, double s) {
    if (axis == QS_GATE_RX) return {c, 0, 0, -s, 0, -s, c, 0};
    if (axis == QS_GATE_RY) return {c, 0, -s, 0, s, 0, c, 0};
    return {c, -s, 0, 0, 0, 0, c, s};
}

// Tile qubits for an n-qubit state: `cap` for large states, fewer below n = cap + 7 so that 128
// tiles (blocks) share the work of mid-size states, never fewer than `floor`: 8 (16 tiles at 12 qubits),
// and the whole state in one tile up to 8 qubits (one block runs every gate without a launch each). Complex64
// sweeps take 10: their tiles are cheap and the launches saved count for more (gradients of 10, 12, 14 qubits
// 323, 423, 486 us at 8 and 285, 367, 444 us at 10; in complex128 the larger tiles lose).
static int adj_tile_qubits(int n, int cap, int floor = 8) {
    return std::min(n, std::max(floor, std::min(cap, n - 7)));
}

constexpr int kAdjDfMin = 6;  // from this many qubits QS_ARITH_DF64 runs double-float tiles

// The tile types of qs_sweep.cuh.
enum SweepType { SW_C64, SW_FX, SW_F64 };

template <typename T, int RB>
static int sweep_per_sm(int tq) {
    const size_t smem = 2 * (sizeof(T) << tq) + SweepSide<T>::bytes(kSwMaxPass, kSwMaxRot, kSwMaxDiag, true, kTileMaxHigh);
    int per_sm = 1;
    resident_blocks(reinterpret_cast<const void*>(k_sweep<T, RB, false>), sweep_threads<RB>(), smem, &per_sm);  // raises its limit
    resident_blocks(reinterpret_cast<const void*>(k_sweep<T, RB, true>), sweep_threads<RB>(), smem, &per_sm);
    return std::max(1, per_sm);
}

// Calls F<T, RB>() for a tile type and tile size.
#define QS_SWEEP(type, tq, F)                                  \
    [&] {                                                      \
        const int rb_ = sw_register_bits(tq);                  \
        if ((type) == SW_C64) {                                \
            if (rb_ == 3) return F(float2, 3);                 \
            if (rb_ == 2) return F(float2, 2);                 \
            return F(float2, 1);                               \
        }                                                      \
        if ((type) == SW_FX) {                                 \
            if (rb_ == 3) return F(FxC, 3);                    \
            if (rb_ == 2) return F(FxC, 2);                    \
            return F(FxC, 1);                                  \
        }                                                      \
        if (rb_ == 3) return F(double2, 3);                    \
        if (rb_ == 2) return F(double2, 2);                    \
        return F(double2, 1);                                  \
    }()

// Blocks of a launch over 2^n amplitudes in tiles of tq qubits (the same for every launch of a gradient,
// so that partials line up).
static int sweep_grid(int n, int tq, SweepType type, bool df, int sms) {
#define QS_F(T, RB) sweep_per_sm<T, RB>(tq)
    int per_sm = QS_SWEEP(type, tq, QS_F);
#undef QS_F
    if (df) {
        int k = 1;
        const size_t smem = 2 * (sizeof(float4) << kAdjT) + size_t(kAdjMaxOps) * (kAdjThreads / 32) * 8 +
                            size_t(kAdjMaxOps) * sizeof(AdjOpDev) + (8u << kTileMaxHigh);
        resident_blocks(reinterpret_cast<const void*>(k_adj_stage_df), kAdjThreads, smem, &k);
        per_sm = std::max(1, std::min(per_sm, k));
    }
    return int(std::min<uint64_t>(1ull << (n - tq), uint64_t(sms) * uint64_t(per_sm)));
}

// The circuit as sweeps: the gates in order of execution, their stages, and the launches with their
// tables. A launch is a program, a double-float stage (df) or a gate no tile holds (single).
struct SweepPlan {
    struct Launch {
        int stage = 0, single = -1, prog = -1;
        bool df = false;
        int first = 0, count = 0;            // df: entries of df_ops
        SweepProgram program;
        std::vector<int> slots;              // df: global slots
    };
    SweepType type = SW_F64;
    std::vector<OpDesc> ops;                 // planning form, in order of execution
    std::vector<int> src;                    // gate index of each op
    std::vector<TileStage> stages;
    std::vector<Launch> launches;
    std::vector<SweepRange> ranges;          // per program
    std::vector<SweepPass> passes;
    std::vector<SweepRot> rots;
    std::vector<TileOp> fixed;
    std::vector<AdjOpDev> df_ops;
    std::vector<int> weight_at;              // per rotation slot: its coefficient, -1: none
};

// gates in order (reverse: backwards), fixed gates as `fixed` classifies them (moved out).
static void plan_sweep(const qs_param_gate* gates, size_t m, const double2* angles, const std::vector<int>& rot_slot,
                       int nrot, std::vector<OpDesc>& fixed, int n, int tq, bool reverse, SweepType type, bool df,
                       bool ordered, SweepPlan* P) {
    P->type = type;
    P->ops.reserve(m);
    P->src.reserve(m);
    for (size_t k = 0; k < m; k++) {
        const size_t g = reverse ? m - 1 - k : k;
        if (rot_slot[g] >= 0) {  // planning form: a dense 1-qubit gate on the rotation's target
            OpDesc d;
            d.kind = OP_DENSE;
            d.k = d.orig_k = 1;
            d.tq[0] = int(gates[g].targets[0]);
            d.m.assign(8, 0.0);
            d.touched_rows = 2;
            P->ops.push_back(std::move(d));
        } else {
            P->ops.push_back(std::move(fixed[g]));
        }
        P->src.push_back(int(g));
    }
    P->weight_at.assign(std::max(1, nrot), -1);
    // rows of 128 bytes: more of the tile's qubits are free to choose
    const int low = df || ordered ? 5 : type == SW_C64 ? 4 : 3;
    P->stages = plan_tiles(P->ops, n, tq, std::min(low, tq), false, df || ordered ? kAdjMaxOps : kSwMaxRot, false,
                           !df && !ordered);
    for (size_t si = 0; si < P->stages.size(); si++) {
        const TileStage& st = P->stages[si];
        SweepPlan::Launch L;
        L.stage = int(si);
        if (!st.tiled) {
            L.single = st.single;
            P->launches.push_back(L);
            continue;
        }
        bool moves_only = true;  // double-float tiles take rotations and pure moves
        for (int idx : st.ops)
            if (rot_slot[P->src[idx]] < 0 && P->ops[idx].kind != OP_MONO_PF) moves_only = false;
        if (df && moves_only) {
            L.df = true;
            L.first = int(P->df_ops.size());
            for (int idx : st.ops) {
                const int g = P->src[idx];
                AdjOpDev e;
                std::memset(&e, 0, sizeof(e));
                e.t = make_tile_op(P->ops[idx], st);
                e.rot = -1;
                if (rot_slot[g] >= 0) {
                    e.rot = int(L.slots.size());
                    L.slots.push_back(rot_slot[g]);
                    e.axis = gates[g].kind;
                    e.c = angles[g].x;
                    e.s = -angles[g].y;
                }
                P->df_ops.push_back(e);
            }
            L.count = int(P->df_ops.size()) - L.first;
            P->launches.push_back(L);
            continue;
        }
        std::vector<SweepGate> sg;
        for (int idx : st.ops) {
            const int g = P->src[idx];
            SweepGate e;
            e.gate = g;
            if (rot_slot[g] >= 0) {
                e.axis = gates[g].kind;
                e.target = int(gates[g].targets[0]);
            } else {
                e.fixed = &P->ops[idx];
            }
            sg.push_back(e);
        }
        for (SweepProgram& prog : build_sweep(sg, st, type == SW_FX, reverse, ordered, &P->fixed)) {
            L.prog = int(P->ranges.size());
            P->ranges.push_back(SweepRange{int(P->passes.size()), int(prog.passes.size()), int(P->rots.size()),
                                           int(prog.rots.size()), prog.ndiag, type != SW_FX, type == SW_C64, 0});
            for (int g : prog.rots) {
                P->weight_at[rot_slot[g]] = int(P->rots.size());
                P->rots.push_back(SweepRot{g, gates[g].kind});
            }
            P->passes.insert(P->passes.end(), prog.passes.begin(), prog.passes.end());
            L.program = std::move(prog);
            P->launches.push_back(L);
        }
    }
}

// Copy rows and tuple expansion of a stage's tiles.
template <typename A>
static void tile_geometry(const TileStage& st, A* a, int* T, int* RL) {
    *T = st.T;
    const int H = int(st.high.size());
    int run = 0;
    while (run < H && st.high[run] == st.L + run) run++;
    *RL = st.L + run;
    a->RH = H - run;
    for (int b = 0; b < a->RH; b++) a->rhigh[b] = uint8_t(st.high[run + b]);
    std::vector<int> qpos;
    for (int q = 0; q < st.L; q++) qpos.push_back(q);
    for (int q : st.high) qpos.push_back(q);
    std::sort(qpos.begin(), qpos.end());
    a->outer.npos = int(qpos.size());
    for (size_t i = 0; i < qpos.size(); i++) a->outer.pos[i] = uint8_t(qpos[i]);
}

// A plan's tables on the device.
struct SweepTables {
    unsigned char* dev = nullptr;
    const SweepRange* ranges = nullptr;
    const SweepPass* passes = nullptr;
    const SweepRot* rots = nullptr;
    const TileOp* fixed = nullptr;
    const AdjOpDev* df_ops = nullptr;
    const int* weight_at = nullptr;
    const double2* angles = nullptr;
    SweepCoef* coefs = nullptr;
    double* weights = nullptr;
    double* sigmas = nullptr;
};

template <typename T, int RB>
static void launch_sweep(bool reverse, const void* src, void* psi, void* lam, uint64_t ntiles, const SweepArgs& a,
                         const SweepTables& tb, double* part, int grid, cudaStream_t s) {
    using G = typename Sw<T>::Glob;
    const size_t smem = size_t(reverse ? 2 : 1) * (sizeof(T) << a.t.T) +
                        SweepSide<T>::bytes(a.t.npass, a.t.nrot, a.t.ndiag, reverse, a.RH);
    const int threads = std::max(32, (1 << a.t.T) >> RB);
    if (reverse)
        k_sweep<T, RB, true><<<grid, threads, smem, s>>>((const G*)src, (G*)psi, (G*)lam, ntiles, a, tb.passes, tb.fixed,
                                                         tb.coefs, tb.sigmas, part);
    else
        k_sweep<T, RB, false><<<grid, threads, smem, s>>>((const G*)src, (G*)psi, (G*)lam, ntiles, a, tb.passes,
                                                          tb.fixed, tb.coefs, tb.sigmas, part);
}

// Uploads a plan's tables (through page-locked staging buffer `staging`, so that the upload does not wait
// for work queued before it) and forms its coefficients. tb->dev is the caller's to free.
static int upload_sweep(const SweepPlan& P, const std::vector<double2>& angles, int staging, cudaStream_t s,
                        SweepTables* tb, std::string* msg) {
    auto al = [](size_t x) { return ((x + 255) / 256) * 256; };
    const size_t o_range = 0, o_pass = o_range + al(P.ranges.size() * sizeof(SweepRange)),
                 o_rot = o_pass + al(P.passes.size() * sizeof(SweepPass)), o_fix = o_rot + al(P.rots.size() * sizeof(SweepRot)),
                 o_df = o_fix + al(P.fixed.size() * sizeof(TileOp)), o_at = o_df + al(P.df_ops.size() * sizeof(AdjOpDev)),
                 o_ang = o_at + al(P.weight_at.size() * sizeof(int)), up = o_ang + al(angles.size() * sizeof(double2)),
                 o_coef = up, o_wt = o_coef + al(P.rots.size() * sizeof(SweepCoef)), o_sig = o_wt + al(P.rots.size() * 8 + 8),
                 total = o_sig + al(P.ranges.size() * 8 + 8);
    cudaError_t e = device_alloc((void**)&tb->dev, total, s);
    if (e != cudaSuccess) {
        tb->dev = nullptr;
        return fail(e, "sweep tables", msg);
    }
    std::vector<unsigned char> pageable;
    unsigned char* host = static_cast<unsigned char*>(pinned_staging(staging, up));
    if (!host) {
        pageable.resize(up);
        host = pageable.data();
    }
    auto put = [&](size_t at, const void* p, size_t bytes) {
        if (bytes) std::memcpy(host + at, p, bytes);
    };
    put(o_range, P.ranges.data(), P.ranges.size() * sizeof(SweepRange));
    put(o_pass, P.passes.data(), P.passes.size() * sizeof(SweepPass));
    put(o_rot, P.rots.data(), P.rots.size() * sizeof(SweepRot));
    put(o_fix, P.fixed.data(), P.fixed.size() * sizeof(TileOp));
    put(o_df, P.df_ops.data(), P.df_ops.size() * sizeof(AdjOpDev));
    put(o_at, P.weight_at.data(), P.weight_at.size() * sizeof(int));
    put(o_ang, angles.data(), angles.size() * sizeof(double2));
    e = cudaMemcpyAsync(tb->dev, host, up, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return fail(e, "sweep tables", msg);
    tb->ranges = reinterpret_cast<const SweepRange*>(tb->dev + o_range);
    tb->passes = reinterpret_cast<const SweepPass*>(tb->dev + o_pass);
    tb->rots = reinterpret_cast<const SweepRot*>(tb->dev + o_rot);
    tb->fixed = reinterpret_cast<const TileOp*>(tb->dev + o_fix);
    tb->df_ops = reinterpret_cast<const AdjOpDev*>(tb->dev + o_df);
    tb->weight_at = reinterpret_cast<const int*>(tb->dev + o_at);
    tb->angles = reinterpret_cast<const double2*>(tb->dev + o_ang);
    tb->coefs = reinterpret_cast<SweepCoef*>(tb->dev + o_coef);
    tb->weights = reinterpret_cast<double*>(tb->dev + o_wt);
    tb->sigmas = reinterpret_cast<double*>(tb->dev + o_sig);
    if (!P.ranges.empty()) {
        k_sweep_coefs<<<int(P.ranges.size()), 64, 0, s>>>(tb->ranges, tb->passes, tb->rots, tb->angles, tb->coefs,
                                                         tb->weights, tb->sigmas);
        e = cudaGetLastError();
        if (e != cudaSuccess) return fail(e, "sweep coefficients", msg);
        note_launches(1);
    }
    return QS_OK;
}

// Runs a plan: psi (and lam in the reverse walk) hold the vectors; src, when not null, is where the
// first launch finds psi. Partials of rotation slot r land in part[r * grid .. + grid).
static int run_sweep(const SweepPlan& P, const SweepTables& tb, const void* src, void* psi, void* lam, int n, int prec,
                     int arith, bool reverse, const std::vector<int>& rot_slot, double* part, int grid, cudaStream_t s,
                     int sms, std::string* msg) {
    const size_t amp = prec == QS_PREC_C64 ? 8 : 16;
    cudaError_t e = cudaSuccess;
    for (size_t li = 0; li < P.launches.size(); li++) {
        const SweepPlan::Launch& L = P.launches[li];
        const TileStage& st = P.stages[L.stage];
        if (src && (L.single >= 0 || L.df)) {  // works in place
            e = cudaMemcpyAsync(psi, src, (size_t(1) << n) * amp, cudaMemcpyDeviceToDevice, s);
            if (e != cudaSuccess) return fail(e, "state copy", msg);
            src = nullptr;
        }
        if (L.single >= 0) {  // a gate no tile holds: one sweep each
            int rc = apply_op(psi, n, prec, arith, P.ops[L.single], s, sms, msg);
            if (rc == QS_OK && reverse) rc = apply_op(lam, n, prec, arith, P.ops[L.single], s, sms, msg);
            if (rc != QS_OK) return rc;
            continue;
        }
        const uint64_t ntiles = 1ull << (n - st.T);
        if (L.df) {
            AdjStageArgs a;
            std::memset(&a, 0, sizeof(a));
            tile_geometry(st, &a, &a.T, &a.RL);
            a.nops = L.count;
            a.nrot = int(L.slots.size());
            for (int r = 0; r < a.nrot; r++) a.slot[r] = L.slots[r];
            const size_t smem = 2 * (sizeof(float4) << st.T) + size_t(a.nrot) * (kAdjThreads / 32) * 8 +
                                size_t(a.nops) * sizeof(AdjOpDev) + (8u << a.RH);
            k_adj_stage_df<<<grid, kAdjThreads, smem, s>>>((double2*)psi, (double2*)lam, ntiles, a, tb.df_ops + L.first,
                                                           part);
        } else {
            SweepArgs a;
            std::memset(&a, 0, sizeof(a));
            tile_geometry(st, &a, &a.t.T, &a.t.RL);
            const SweepRange& R = P.ranges[L.prog];
            a.t.npass = R.npass;
            a.t.nrot = R.nrot;
            a.t.ndiag = R.ndiag;
            a.t.store = !reverse || li + 1 < P.launches.size();
            a.pass0 = R.pass0;
            a.coef0 = R.coef0;
            a.prog = L.prog;
            for (int r = 0; r < R.nrot; r++) a.slot[r] = rot_slot[L.program.rots[r]];
            const void* from = src ? src : psi;
#define QS_F(T, RB) launch_sweep<T, RB>(reverse, from, psi, lam, ntiles, a, tb, part, grid, s)
            QS_SWEEP(P.type, st.T, QS_F);
#undef QS_F
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) return fail(e, "sweep", msg);
        note_launches(1);
        src = nullptr;
    }
    if (src) {  // no launch took the state over
        e = cudaMemcpyAsync(psi, src, (size_t(1) << n) * amp, cudaMemcpyDeviceToDevice, s);
        if (e != cudaSuccess) return fail(e, "state copy", msg);
    }
    return QS_OK;
}

int adjoint_gradient(void* state, int n, int prec, int arith, const qs_param_gate* gates, size_t m,
                     const double* params, size_t np, const qs_pauli_term* terms, size_t nt, cudaStream_t s, int sms,
                     double* energy, double* grad, size_t* err, std::string* msg) {
    // ---- validation (nothing is launched before every gate checks out)
    std::vector<OpDesc> fwd(m), inv(m);
    std::vector<int> rot_slot(m, -1);
    int nrot = 0;
    for (size_t g = 0; g < m; g++) {
        const qs_param_gate& G = gates[g];
        if (G.kind == QS_GATE_FIXED) {
            const size_t dim = G.k < 64 ? (size_t(1) << G.k) : 0;
            int rc = validate_gate(size_t(n), dim, dim, G.targets, G.k, err, msg);
            if (!rc && !G.matrix) rc = QS_INVALID_ARGUMENT, *msg = "matrix is null";
            if (rc) {
                if (err) err[2] = g;
                return rc;
            }
            classify_gate(G.matrix, G.k, G.targets, &fwd[g]);
            std::vector<double> h(2 * dim * dim);
            for (size_t r = 0; r < dim; r++)
                for (size_t c = 0; c < dim; c++) {  // conjugate transpose
                    h[2 * (r * dim + c)] = G.matrix[2 * (c * dim + r)];
                    h[2 * (r * dim + c) + 1] = -G.matrix[2 * (c * dim + r) + 1];
                }
            classify_gate(h.data(), G.k, G.targets, &inv[g]);
        } else if (G.kind == QS_GATE_RX || G.kind == QS_GATE_RY || G.kind == QS_GATE_RZ) {
            if (G.k != 1 || !G.targets) {
                if (err) err[0] = G.k, err[2] = g;
                *msg = "rotation gates take exactly one target";
                return QS_INVALID_ARITY;
            }
            if (G.targets[0] >= size_t(n)) {
                if (err) err[0] = G.targets[0], err[2] = g;
                *msg = "InvalidTarget(" + std::to_string(G.targets[0]) + ")";
                return QS_INVALID_TARGET;
            }
            if (G.param < 0 || size_t(G.param) >= np) {
                if (err) err[2] = g;
                *msg = "rotation parameter index out of range";
                return QS_INVALID_ARGUMENT;
            }
            rot_slot[g] = nrot++;
        } else {
            if (err) err[2] = g;
            *msg = "unknown gate kind";
            return QS_INVALID_ARGUMENT;
        }
    }
    // ---- tables
    std::vector<PauliDev> ht = pauli_table(terms, nt);
    const size_t amp = prec == QS_PREC_C64 ? 8 : 16;
    const uint64_t N = 1ull << n;
    const bool df = prec == QS_PREC_C128 && arith == QS_ARITH_DF64 && n >= kAdjDfMin;
    const int tq = adj_tile_qubits(n, kAdjT, prec == QS_PREC_C64 ? 10 : 8);
    bool unitary = true;
    for (size_t g = 0; g < m && unitary; g++)
        if (gates[g].kind == QS_GATE_FIXED) unitary = is_unitary(gates[g].matrix, gates[g].k);
    const SweepType type = prec == QS_PREC_C64 ? SW_C64 : sweep_fixed_point(arith, unitary) ? SW_FX : SW_F64;
    const int pgrid = sweep_grid(n, tq, type, df, sms);
    auto al = [](size_t x) { return ((x + 255) / 256) * 256; };
    const size_t o_terms = 0, o_part = o_terms + al(nt * sizeof(PauliDev) + 1),
                 o_res = o_part + al(size_t(std::max(nrot, 1)) * pgrid * 8 + 4096 * 16),
                 o_lam = o_res + al((2 + size_t(nrot)) * 8), o_psi = o_lam + al(N * amp), total = o_psi + N * amp;
    unsigned char* blob = nullptr;
    std::vector<double> res(2 + nrot, 0.0);  // the energy, the rotations' terms, the status: one readback
    std::vector<double2> angles(std::max<size_t>(m, 1), make_double2(1.0, 0.0));  // per gate: cos, sin of theta / 2
    bool finite = true;
    for (size_t g = 0; g < m; g++)
        if (rot_slot[g] >= 0) {
            const double th = params[gates[g].param];
            angles[g] = make_double2(std::cos(0.5 * th), std::sin(0.5 * th));
            finite = finite && std::isfinite(angles[g].x) && std::isfinite(angles[g].y);
        }
    if (!finite) {
        // A rotation by an infinity or NaN leaves NaN in every amplitude, so the energy and every rotation's
        // derivative are NaN. Said here: the tiles' fixed-point coefficients and phases have no NaN.
        const double nan = std::numeric_limits<double>::quiet_NaN();
        if (energy) *energy = nan;
        for (size_t p = 0; grad && p < np; p++) grad[p] = 0.0;
        for (size_t g = 0; grad && g < m; g++)
            if (rot_slot[g] >= 0) grad[gates[g].param] = nan;
        return QS_OK;
    }
    SweepPlan fplan, rplan;
    SweepTables ftab, rtab;
    int rc = QS_OK;
    AJ_CHECK(device_alloc((void**)&blob, total, s), "adjoint buffers");
    {
        void* lam = blob + o_lam;
        void* psi = blob + o_psi;  // the register's own state is only read
        double* part = (double*)(blob + o_part);
        double* dres = (double*)(blob + o_res);
        if (nt)
            AJ_CHECK(cudaMemcpyAsync(blob + o_terms, ht.data(), nt * sizeof(PauliDev), cudaMemcpyHostToDevice, s),
                     "terms upload");
        int* derr = reinterpret_cast<int*>(dres + 1 + nrot);  // raised by a forward tile kernel's bounded wait
        int blocks = 0;  // of the energy's partials
        double* epart = part + size_t(std::max(nrot, 1)) * pgrid;
        // forward
        if (df) {
            AJ_CHECK(cudaMemsetAsync(derr, 0, sizeof(double), s), "status flag");
            AJ_CHECK(cudaMemcpyAsync(psi, state, N * amp, cudaMemcpyDeviceToDevice, s), "state copy");
            std::vector<OpDesc> fops(m);
            std::vector<double> rmat(8 * m);  // the rotations' matrices, in gate order
            for (size_t g = 0; g < m; g++) {
                if (rot_slot[g] >= 0) {
                    const std::vector<double> R = rotation_matrix(gates[g].kind, angles[g].x, angles[g].y);
                    std::copy(R.begin(), R.end(), rmat.begin() + 8 * g);
                    classify_gate(R.data(), 1, gates[g].targets, &fops[g]);
                } else {
                    fops[g] = std::move(fwd[g]);
                }
            }
            if (n >= 18) {
                // double-float dense blocks (3 qubits, the automatic width): the fastest complex128
                // double-float form of a circuit of 1-qubit rotations and CNOTs at 11-qubit tiles (1.85x
                // the stages at 20 qubits; below 18 qubits the smaller stage tiles win); the blocks are
                // products of the gates' FP64 matrices
                std::vector<qs_gate> qg(m);
                for (size_t g = 0; g < m; g++)
                    qg[g] = rot_slot[g] >= 0 ? qs_gate{1, gates[g].targets, rmat.data() + 8 * g}
                                             : qs_gate{gates[g].k, gates[g].targets, gates[g].matrix};
                const qs_circuit_options fo{2, 0, 0, 0};
                if ((rc = run_circuit(psi, n, prec, arith, fops, qg.data(), fo, s, sms, msg, derr)) != QS_OK)
                    goto done;
            } else {
                // tiles as in the reverse sweep: below 18 qubits smaller than the default so that smaller
                // states still spread over many blocks
                const qs_circuit_options fo{1, 5, adj_tile_qubits(n, 11), 0};
                // queued without waiting: the reverse sweep is planned while the forward runs
                if ((rc = run_circuit(psi, n, prec, arith, fops, nullptr, fo, s, sms, msg, derr)) != QS_OK)
                    goto done;
            }
        } else {
            plan_sweep(gates, m, angles.data(), rot_slot, nrot, fwd, n, tq, false, type, false, !unitary, &fplan);
            if ((rc = upload_sweep(fplan, angles, 0, s, &ftab, msg)) != QS_OK) goto done;
            if ((rc = run_sweep(fplan, ftab, state, psi, nullptr, n, prec, arith, false, rot_slot, part, pgrid, s, sms,
                                msg)) != QS_OK)
                goto done;
        }
        // lambda = H psi, E = Re<psi|lambda>
        if (prec == QS_PREC_C64)
            blocks = launch_pauli_sum<float2>(psi, lam, n, (const PauliDev*)(blob + o_terms), int(nt), pauli_df_ok(ht),
                                              epart, s, sms);
        else
            blocks = launch_pauli_sum<double2>(psi, lam, n, (const PauliDev*)(blob + o_terms), int(nt), false, epart, s,
                                               sms);
        AJ_CHECK(cudaGetLastError(), "pauli sum");
        // reverse
        plan_sweep(gates, m, angles.data(), rot_slot, nrot, inv, n, tq, true, type, df, !unitary, &rplan);
        if ((rc = upload_sweep(rplan, angles, 1, s, &rtab, msg)) != QS_OK) goto done;
        if ((rc = run_sweep(rplan, rtab, nullptr, psi, lam, n, prec, arith, true, rot_slot, part, pgrid, s, sms, msg)) !=
            QS_OK)
            goto done;
        k_grad_final<<<1 + nrot, kAT, 0, s>>>(epart, blocks, part, pgrid, rtab.weights, rtab.weight_at, dres);
        note_launches(1);
        AJ_CHECK(cudaGetLastError(), "gradient reduction");
        AJ_CHECK(cudaMemcpyAsync(res.data(), dres, (1 + size_t(nrot) + (df ? 1 : 0)) * 8, cudaMemcpyDeviceToHost, s),
                 "readback");
        AJ_CHECK(cudaStreamSynchronize(s), "adjoint sync");
        int herr = 0;
        std::memcpy(&herr, &res[1 + nrot], sizeof(herr));
        if (df && herr) {
            *msg = "a tile kernel's bounded wait for its bulk copies gave up";
            rc = QS_TIMEOUT;
            goto done;
        }
        if (energy) *energy = res[0];
        if (grad) {
            for (size_t p = 0; p < np; p++) grad[p] = 0.0;
            for (size_t g = 0; g < m; g++)
                if (rot_slot[g] >= 0) grad[gates[g].param] += res[1 + rot_slot[g]];
        }
    }
done:
    if (rc != QS_OK) cudaStreamSynchronize(s);  // the staging buffers are free again
    if (ftab.dev) cudaFreeAsync(ftab.dev, s);
    if (rtab.dev) cudaFreeAsync(rtab.dev, s);
    if (blob) cudaFreeAsync(blob, s);
    return rc;
}

}  // namespace qs
