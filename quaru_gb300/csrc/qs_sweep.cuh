// qs_sweep.cuh — the passes of the gradient sweeps over a tile in shared memory (see qs_sweep.h).
//
// Tile types: float2 (complex64), FxC (complex128 as 64-bit fixed point), double2 (complex128 in
// QS_ARITH_EXACT, or where a fixed gate is not unitary, so that fixed point has no bound to scale by).
//
// sm_103a issues about 2 FP64 operations per clock and SM, 64 integer and 128 FP32 ones, so double2
// tiles are bound by the FP64 pipe and the others by instruction issue. Hence
//   * complex128 tiles in fixed point: every component is an integer on the scale of the tile's own
//     norm, 2^60, which unitary gates keep, and rotations are three shears of integer multiply-adds
//     (4 wide ones and 3 other instructions each; an FP64 multiply-add takes the time of 32);
//     an operation's rounding, 2^-60 of the tile's norm on each of up to 2^12 components, is a
//     quarter of what FP64 leaves on the tile's vector;
//   * a floating rotation leaves out its common factor (two multiply-adds per real pair instead of
//     four operations), which the phases of the program carry as one number;
//   * a run of RZ gates is one multiplication by a phase from two small tables, and its inner products
//     are signed sums of one product per amplitude, split over register, warp and lane bits (a
//     Walsh-Hadamard butterfly);
//   * a run of CNOTs is one gather;
//   * a pass holds 2^RB amplitudes of each vector in registers for up to four rotations, whose partial
//     sums cross the warp together.
// Tiles are XOR-swizzled so that the register bits {0,1,2}, {3,4,5}, ... are free of bank conflicts.
#pragma once

#include <cuda_runtime.h>

#include "qs_device.cuh"
#include "qs_pass.cuh"
#include "qs_reduce.cuh"
#include "qs_rot.cuh"
#include "qs_sweep.h"

namespace qs {

constexpr int kSwThreads = 256;  // most threads of a block: 2^8 tuples of eight amplitudes
constexpr int kSwWarps = kSwThreads / 32;
constexpr int kSwTable = 32 + (1 << (kSwMaxT - 5));  // factor table: low five tile bits, then the others

template <int V>
struct SwInt {
    static constexpr int value = V;
};

// ---- per element type: swizzle, packed updates, partial sums
// ---- fixed point: 2^60 ths of a scale; products by 30-bit limbs
struct alignas(16) FxC {
    long long x, y;
};
constexpr double kFxOne = 1152921504606846976.0;  // 2^60

// C as limbs ch 2^30 + cl with cl in [-2^29, 2^29), and what is added before the low products are cut off:
// half a unit, and the mean of the dropped product of low limbs.
struct FxLimb {
    int h, l;
    long long k;
    int one;  // 1, as a value the compiler does not know
};
__host__ __device__ __forceinline__ FxLimb fx_limb(long long C) {
    FxLimb r;
    r.l = int(static_cast<long long>(static_cast<unsigned long long>(C) << 34) >> 34);
    r.h = int((C - r.l) >> 30);
    r.k = (1ll << 29) + (r.l >> 1);
    r.one = 1;
    return r;
}
__device__ __forceinline__ int fx_one() {
    int r;
    asm("mov.u32 %0, 1;" : "=r"(r));
    return r;
}
__device__ __forceinline__ FxLimb fx_neg(FxLimb c) {
    c.h = -c.h;
    c.l = -c.l;
    c.k = (1ll << 30) - c.k;
    return c;
}
struct FxVal {  // x = h 2^30 + l, 0 <= l < 2^30
    int h, l;
};
__device__ __forceinline__ FxVal fx_val(long long x) {
    FxVal r;
    r.h = int(__funnelshift_r(uint32_t(x), uint32_t(static_cast<unsigned long long>(x) >> 32), 30));
    r.l = int(uint32_t(x) & 0x3fffffffu);
    return r;
}
// acc + v C / 2^60 for |v|, |C| <= 2^60: four wide multiply-adds
__device__ __forceinline__ long long fx_mac(long long acc, FxVal v, const FxLimb& c) {
    long long b = fx_mad(v.h, c.l, c.k);
    b = fx_mad(v.l, c.h, b);
    acc = fx_mad(v.h, c.h, acc);
    const int cut = int(__funnelshift_r(uint32_t(b), uint32_t(static_cast<unsigned long long>(b) >> 32), 30));
    return fx_mad(cut, c.one, acc);  // one wide multiply-add instead of a sign extension and two additions
}
__device__ __forceinline__ long long fx_mac(long long acc, long long v, const FxLimb& c) {
    return fx_mac(acc, fx_val(v), c);
}

template <typename T>
struct Sw;

template <>
struct Sw<double2> {
    using Acc = double;  // a partial sum of inner products
    using Glob = double2;
    using Coef = double2;   // RX, RY: t, form
    using Phase = double2;  // entry of a factor table
    static __device__ __forceinline__ Coef coef(const SweepCoef& c) { return make_double2(c.c, c.s); }
    static __device__ __forceinline__ uint32_t at(uint32_t x) { return x ^ ((x >> 3) & 7u); }
    static __device__ __forceinline__ Acc zero() { return 0.0; }
    static __device__ __forceinline__ Acc add(Acc a, Acc b) { return a + b; }
    static __device__ __forceinline__ Acc neg(Acc a) {
        return __hiloint2double(__double2hiint(a) ^ int(0x80000000u), __double2loint(a));
    }
    static __device__ __forceinline__ Acc shfl_xor(Acc a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
    static __device__ __forceinline__ Acc shfl(Acc a, int l) { return __shfl_sync(0xffffffffu, a, l); }
    using Cell = double;  // a warp's sum in shared memory
    static __device__ __forceinline__ void gather(Cell& c, Acc a) { c += a; }
    static __device__ __forceinline__ double value(Cell c) { return c; }
};

template <>
struct Sw<FxC> {
    using Acc = long long;  // 2^60 ths of the product of the two vectors' scales
    using Glob = double2;
    using Coef = SweepCoef;
    using Phase = int4;     // limbs of the real and the imaginary part
    static __device__ __forceinline__ Coef coef(const SweepCoef& c) { return c; }
    static __device__ __forceinline__ Phase phase(const FxC& v) {
        const FxLimb r = fx_limb(v.x), i = fx_limb(v.y);
        return make_int4(r.h, r.l, i.h, i.l);
    }
    static __device__ __forceinline__ uint32_t at(uint32_t x) { return x ^ ((x >> 3) & 7u); }
    static __device__ __forceinline__ Acc zero() { return 0; }
    static __device__ __forceinline__ Acc add(Acc a, Acc b) { return a + b; }
    static __device__ __forceinline__ Acc neg(Acc a) { return -a; }
    static __device__ __forceinline__ Acc shfl_xor(Acc a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
    static __device__ __forceinline__ Acc shfl(Acc a, int l) { return __shfl_sync(0xffffffffu, a, l); }
    using Cell = long long;  // one tile's
    static __device__ __forceinline__ void gather(Cell& c, Acc a) { c += a; }
};

template <>
struct Sw<float2> {
    using Acc = DfAcc;
    using Glob = float2;
    using Coef = float2;
    using Phase = float2;
    static __device__ __forceinline__ Coef coef(const SweepCoef& c) { return make_float2(float(c.c), float(c.s)); }
    static __device__ __forceinline__ uint32_t at(uint32_t x) { return x ^ ((x >> 4) & 7u) ^ ((x >> 3) & 8u); }
    static __device__ __forceinline__ Acc zero() { return Acc(); }
    static __device__ __forceinline__ Acc add(Acc a, Acc b) {
        a.add(b.s);
        a.c = __fadd_rn(a.c, b.c);
        return a;
    }
    static __device__ __forceinline__ Acc neg(Acc a) {
        a.s = -a.s;
        a.c = -a.c;
        return a;
    }
    static __device__ __forceinline__ Acc shfl_xor(Acc a, int o) {
        Acc r;
        r.s = __shfl_xor_sync(0xffffffffu, a.s, o);
        r.c = __shfl_xor_sync(0xffffffffu, a.c, o);
        return r;
    }
    static __device__ __forceinline__ Acc shfl(Acc a, int l) {
        Acc r;
        r.s = __shfl_sync(0xffffffffu, a.s, l);
        r.c = __shfl_sync(0xffffffffu, a.c, l);
        return r;
    }
    using Cell = DfAcc;
    static __device__ __forceinline__ void gather(Cell& c, Acc a) { c = add(c, a); }
    static __device__ __forceinline__ double value(Cell a) { return __dadd_rn(df_f2d(a.s), df_f2d(a.c)); }
};

__device__ __forceinline__ double sw_neg(double x) {
    return __hiloint2double(__double2hiint(x) ^ int(0x80000000u), __double2loint(x));
}
__device__ __forceinline__ float sw_neg(float x) { return -x; }
__device__ __forceinline__ long long sw_neg(long long x) { return -x; }

// a + t b, both components (packed on float2)
__device__ __forceinline__ double2 sw_axpy(double t, double2 b, double2 a) {
    return make_double2(fma(t, b.x, a.x), fma(t, b.y, a.y));
}
__device__ __forceinline__ uint64_t sw_pack(float2 v) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v.x), "f"(v.y));
    return r;
}
__device__ __forceinline__ float2 sw_unpack(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ float2 sw_fma2(float2 a, float2 b, float2 c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(sw_pack(a)), "l"(sw_pack(b)), "l"(sw_pack(c)));
    return sw_unpack(r);
}
__device__ __forceinline__ float2 sw_mul2(float2 a, float2 b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(sw_pack(a)), "l"(sw_pack(b)));
    return sw_unpack(r);
}
__device__ __forceinline__ float2 sw_add2(float2 a, float2 b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(sw_pack(a)), "l"(sw_pack(b)));
    return sw_unpack(r);
}
__device__ __forceinline__ float2 sw_sub2(float2 a, float2 b) { return sw_fma2(b, make_float2(-1.0f, -1.0f), a); }
// (x + y) of d as a compensated pair (TwoSum)
__device__ __forceinline__ DfAcc sw_across(float2 d) {
    DfAcc a;
    a.s = __fadd_rn(d.x, d.y);
    const float bb = __fsub_rn(a.s, d.x);
    a.c = __fadd_rn(__fsub_rn(d.x, __fsub_rn(a.s, bb)), __fsub_rn(d.y, bb));
    return a;
}
// d + f, both components, then across (TwoSum on both at once)
__device__ __forceinline__ DfAcc sw_across(float2 d, float2 f) {
    const float2 s = sw_add2(d, f), bb = sw_sub2(s, d);
    const float2 e = sw_add2(sw_sub2(d, sw_sub2(s, bb)), sw_sub2(f, bb));
    DfAcc a = sw_across(s);
    a.c = __fadd_rn(a.c, __fadd_rn(e.x, e.y));
    return a;
}
__device__ __forceinline__ float2 sw_axpy(float t, float2 b, float2 a) { return sw_fma2(make_float2(t, t), b, a); }

template <typename T>
__device__ __forceinline__ T sw_minus(T v) {
    T r;
    r.x = sw_neg(v.x);
    r.y = sw_neg(v.y);
    return r;
}

// A rotations pass turns every pair like RY: R_X acts on (a, -i b) as R_Y(-theta) does on (a, b), so an RX
// runs between two changes of b (sw_frame), which leave the other bits' inner products as they are. A
// quarter turn (SweepCoef's exchanged form) comes first: the sign it leaves out is common to every
// amplitude of both vectors.
template <int J, int N, typename T>
__device__ __forceinline__ void sw_frame(bool back, T (&x)[N]) {  // b <- -i b, or back
#pragma unroll
    for (int r = 0; r < N; r++)
        if (r & (1 << J)) {
            const T v = x[r];
            x[r].x = back ? sw_neg(v.y) : v.y;
            x[r].y = back ? v.x : sw_neg(v.x);
        }
}
template <int N, typename T>
__device__ __forceinline__ void sw_frames(uint32_t rx, bool back, T (&x)[N]) {
    if (rx & 1u) sw_frame<0>(back, x);
    if (N > 2 && (rx & 2u)) sw_frame<1>(back, x);
    if (N > 4 && (rx & 4u)) sw_frame<2>(back, x);
}
template <int J, int N, typename T>
__device__ __forceinline__ void sw_quarter(T (&x)[N]) {  // (a, b) <- (-b, a)
#pragma unroll
    for (int r = 0; r < N; r++) {
        if (r & (1 << J)) continue;
        const T a = x[r];
        x[r] = sw_minus(x[r | (1 << J)]);
        x[r | (1 << J)] = a;
    }
}
// (a - t b, b + t a): R_Y without its common factor.
template <int J, int N, typename T>
__device__ __forceinline__ void sw_update(T cf, bool inverse, T (&x)[N]) {
    const auto t = inverse ? sw_neg(cf.x) : cf.x, nt = sw_neg(t);
#pragma unroll
    for (int r = 0; r < N; r++) {
        if (r & (1 << J)) continue;
        const T a = x[r], b = x[r | (1 << J)];
        x[r] = sw_axpy(nt, b, a);
        x[r | (1 << J)] = sw_axpy(t, a, b);
    }
}
// (x, y) turned by the angle whose shears are p = -tan(a / 2), s = sin(a)
__device__ __forceinline__ void fx_turn(long long& x, long long& y, const FxLimb& p, const FxLimb& s) {
    x = fx_mac(x, y, p);
    y = fx_mac(y, x, s);
    x = fx_mac(x, y, p);
}
template <int J, int N>
__device__ __forceinline__ void sw_update(const SweepCoef& cf, bool inverse, FxC (&x)[N]) {
    const int one = fx_one();
    FxLimb p{cf.ph, cf.pl, cf.pk, one}, s{cf.sh, cf.sl, cf.sk, one};
    if (inverse) p = fx_neg(p), s = fx_neg(s);
#pragma unroll
    for (int r = 0; r < N; r++) {
        if (r & (1 << J)) continue;
        fx_turn(x[r].x, x[r | (1 << J)].x, p, s);
        fx_turn(x[r].y, x[r | (1 << J)].y, p, s);
    }
}
template <typename T>
__device__ __forceinline__ bool sw_exchanged(T cf) { return cf.y != decltype(cf.y)(0); }
__device__ __forceinline__ bool sw_exchanged(const SweepCoef& cf) { return cf.quarter != 0; }

// This thread's share of Im<lambda|Y|psi> on register bit J: sum of Re(conj(l_b) p_a) - Re(conj(l_a) p_b)
// (for an RX, behind the change of b, minus Im<lambda|X|psi>).
template <int J, int N>
__device__ __forceinline__ double sw_inner(const double2 (&p)[N], const double2 (&l)[N]) {
    double s = 0.0;
#pragma unroll
    for (int r = 0; r < N; r++) {
        if (r & (1 << J)) continue;
        const int k = r | (1 << J);
        s = fma(l[k].x, p[r].x, s);
        s = fma(l[k].y, p[r].y, s);
        s = fma(sw_neg(l[r].x), p[k].x, s);
        s = fma(sw_neg(l[r].y), p[k].y, s);
    }
    return s;
}
// complex64: real and imaginary parts side by side (packed operations); chains of at most four products, as
// one pair's four products take, then compensated sums.
template <int J, int N>
__device__ __forceinline__ DfAcc sw_inner(const float2 (&p)[N], const float2 (&l)[N]) {
    float2 d[2];
#pragma unroll
    for (int h = 0; h < (N > 4 ? 2 : 1); h++) {
        float2 plus = make_float2(0.0f, 0.0f), minus = plus;
        bool first = true;
#pragma unroll
        for (int i = 0; i < (N > 2 ? 2 : 1); i++) {
            const int q = 2 * h + i, r = ((q >> J) << (J + 1)) | (q & ((1 << J) - 1)), k = r | (1 << J);
            plus = first ? sw_mul2(l[k], p[r]) : sw_fma2(l[k], p[r], plus);
            minus = first ? sw_mul2(l[r], p[k]) : sw_fma2(l[r], p[k], minus);
            first = false;
        }
        d[h] = sw_sub2(plus, minus);
    }
    if constexpr (N > 4) return sw_across(d[0], d[1]);
    else return sw_across(d[0]);
}
// fixed point: positive and negative products apart (each sum of 8 stays below 2^63 by the norms)
struct FxSum {
    long long a = 0, b = 0;
    __device__ __forceinline__ void add(long long u, long long v) {
        const FxVal p = fx_val(u), q = fx_val(v);
        a = fx_mad(p.h, q.h, a);
        b = fx_mad(p.h, q.l, b);
        b = fx_mad(p.l, q.h, b);
    }
};
template <int J, int N>
__device__ __forceinline__ long long sw_inner(const FxC (&p)[N], const FxC (&l)[N]) {
    FxSum plus, minus;
#pragma unroll
    for (int r = 0; r < N; r++) {
        if (r & (1 << J)) continue;
        const int k = r | (1 << J);
        plus.add(l[k].x, p[r].x);
        plus.add(l[k].y, p[r].y);
        minus.add(l[r].x, p[k].x);
        minus.add(l[r].y, p[k].y);
    }
    return (plus.a - minus.a) + (plus.b >> 30) - (minus.b >> 30);
}

// Sums of four values over the warp: lane 8 k returns (and so do its seven neighbours) value k's.
// Two exchanging steps, then three of one value each: 6 additions instead of 20.
template <typename T>
__device__ __forceinline__ typename Sw<T>::Acc sw_warp_sum4(typename Sw<T>::Acc a0, typename Sw<T>::Acc a1,
                                                            typename Sw<T>::Acc a2, typename Sw<T>::Acc a3) {
    using S = Sw<T>;
    using A = typename S::Acc;
    const bool h = threadIdx.x & 16u, g = threadIdx.x & 8u;
    A k0 = h ? a2 : a0, k1 = h ? a3 : a1;  // kept: values 0, 1 below lane 16, 2, 3 from there
    const A g0 = h ? a0 : a2, g1 = h ? a1 : a3;
    k0 = S::add(k0, S::shfl_xor(g0, 16));
    k1 = S::add(k1, S::shfl_xor(g1, 16));
    A k = g ? k1 : k0;
    const A give = g ? k0 : k1;
    k = S::add(k, S::shfl_xor(give, 8));
    k = S::add(k, S::shfl_xor(k, 4));
    k = S::add(k, S::shfl_xor(k, 2));
    return S::add(k, S::shfl_xor(k, 1));
}

// ---- a rotations pass. The rotations are on different bits and commute, so every inner product is taken
// from the vectors as the pass finds them; then one vector after the other is turned, by the same code.
// Warps without a tuple return at once; in the last one, lanes without a tuple take part with zeros.
template <typename T, int RB, bool REV>
__device__ __forceinline__ void sw_rotations(T* sp, T* sl, uint32_t tsize, const SweepPass& P,
                                             const typename Sw<T>::Coef* coef, typename Sw<T>::Cell* sacc) {
    using S = Sw<T>;
    using A = typename S::Acc;
    constexpr int N = 1 << RB;
    const uint32_t ntup = tsize >> RB, p = threadIdx.x;
    if ((p & ~31u) >= ntup) return;
    uint32_t base = p & P.seg[0];
    base |= (p << 1) & P.seg[1];
    if (RB > 1) base |= (p << 2) & P.seg[2];
    if (RB > 2) base |= (p << 3) & P.seg[3];
    uint32_t at[N];  // byte offsets
    at[0] = S::at(base) * uint32_t(sizeof(T));
#pragma unroll
    for (int j = 0; j < RB; j++) {
        const uint32_t w = S::at(1u << P.rbit[j]) * uint32_t(sizeof(T));
#pragma unroll
        for (int r = 0; r < (1 << j); r++) at[r | (1 << j)] = at[r] ^ w;
    }
    const uint32_t rx = P.rx;
    const bool on = p < ntup;  // false only in the one warp of a tile of fewer than 32 tuples
    auto load = [&](const T* s, T (&x)[N]) {
        if (ntup >= 32u) {
#pragma unroll
            for (int r = 0; r < N; r++) x[r] = *reinterpret_cast<const T*>(reinterpret_cast<const char*>(s) + at[r]);
        } else {
#pragma unroll
            for (int r = 0; r < N; r++)
                x[r] = on ? *reinterpret_cast<const T*>(reinterpret_cast<const char*>(s) + at[r]) : T{0, 0};
        }
        if (rx) sw_frames(rx, false, x);
    };
    if (REV) {
        T x[N], l[N];
        load(sp, x);
        load(sl, l);
        A v[4] = {S::zero(), S::zero(), S::zero(), S::zero()};
        v[0] = sw_inner<0>(x, l);
        if constexpr (RB > 1) v[1] = sw_inner<1>(x, l);
        if constexpr (RB > 2) v[2] = sw_inner<2>(x, l);
        const A t = sw_warp_sum4<T>(v[0], v[1], v[2], v[3]);
        const int lane = threadIdx.x & 31, k = lane >> 3;
        if ((lane & 7) == 0 && k < RB && P.rot[k] >= 0)
            S::gather(sacc[P.rot[k] * kSwWarps + (threadIdx.x >> 5)], (rx >> k & 1u) ? S::neg(t) : t);
    }
#pragma unroll 1
    for (int h = 0; h < (REV ? 2 : 1); h++) {
        T* s = h ? sl : sp;
        T x[N];
        load(s, x);
        auto turn = [&](auto bit) {
            constexpr int J = decltype(bit)::value;
            if constexpr (J < RB) {
                if (P.rot[J] < 0) return;
                const typename S::Coef& cf = coef[P.rot[J]];
                if (sw_exchanged(cf)) sw_quarter<J>(x);
                sw_update<J>(cf, REV != bool(rx >> J & 1u), x);
            }
        };
        turn(SwInt<0>());
        turn(SwInt<1>());
        turn(SwInt<2>());
        if (rx) sw_frames(rx, true, x);
        if (on) {
#pragma unroll
            for (int r = 0; r < N; r++) *reinterpret_cast<T*>(reinterpret_cast<char*>(s) + at[r]) = x[r];
        }
    }
}

// Im(conj(l) p)
__device__ __forceinline__ double sw_cross(double2 l, double2 p) { return fma(l.x, p.y, -(l.y * p.x)); }
__device__ __forceinline__ long long sw_cross(const FxC& l, const FxC& p) {
    FxSum plus, minus;
    plus.add(l.x, p.y);
    minus.add(l.y, p.x);
    return (plus.a - minus.a) + (plus.b >> 30) - (minus.b >> 30);
}

// ---- a moves pass: amplitude x takes what f(x) held, times its phase. The register bits are the top
// RB tile bits. Two barriers inside (every thread of the block calls this).
template <typename T>
__device__ __forceinline__ T sw_phase(T ph, T v) {
    return cfma(ph.x, ph.y, v, czero<T>());
}
__device__ __forceinline__ FxC sw_phase(int4 ph, FxC v) {
    const int one = fx_one();
    const FxLimb re = {ph.x, ph.y, (1ll << 29) + (ph.y >> 1), one}, im = {ph.z, ph.w, (1ll << 29) + (ph.w >> 1), one};
    const FxVal x = fx_val(v.x), y = fx_val(v.y);
    return FxC{fx_mac(fx_mac(0, x, re), y, fx_neg(im)), fx_mac(fx_mac(0, y, re), x, im)};
}
// the product of two table entries
template <typename T>
__device__ __forceinline__ T sw_phase2(T a, T b) {
    return cfma(a.x, a.y, b, czero<T>());
}
__device__ __forceinline__ int4 sw_phase2(int4 a, int4 b) {
    const FxC v = sw_phase(a, FxC{(static_cast<long long>(b.x) << 30) + b.y, (static_cast<long long>(b.z) << 30) + b.w});
    const FxLimb re = fx_limb(v.x), im = fx_limb(v.y);
    return make_int4(re.h, re.l, im.h, im.l);
}

template <typename T, int RB, bool REV>
__device__ __forceinline__ void sw_moves(T* sp, T* sl, uint32_t tsize, int tq, uint64_t tile_base, const SweepPass& P,
                                         const typename Sw<T>::Phase* tables, typename Sw<T>::Cell* sacc) {
    using S = Sw<T>;
    using A = typename S::Acc;
    constexpr int N = 1 << RB;
    const uint32_t ntup = tsize >> RB, p = threadIdx.x;
    const bool warp_on = (p & ~31u) < ntup, on = p < ntup;
    const int TB = tq - RB;  // thread bits
    T x[N], l[N];
    uint32_t f = p, c[RB];  // f(x) = f ^ (c[j] for every set bit j of r), x = p | r << TB
#pragma unroll
    for (int j = 0; j < RB; j++) c[j] = 1u << (TB + j);
    if (P.moves && on) {
        f = P.flip;
        for (int i = 0; i < P.nout; i++)
            if (tile_base >> P.oq[i] & 1ull) f ^= P.om[i];
        for (int b = 0; b < TB; b++) f ^= (p >> b & 1u) ? uint32_t(P.col[b]) : 0u;
#pragma unroll
        for (int j = 0; j < RB; j++) c[j] = P.col[TB + j];
    }
    auto from = [&](int r) {
        uint32_t y = f;
#pragma unroll
        for (int j = 0; j < RB; j++)
            if (r >> j & 1) y ^= c[j];
        return y;
    };
    if (on) {
#pragma unroll
        for (int r = 0; r < N; r++) {
            uint32_t y = S::at(f);
#pragma unroll
            for (int j = 0; j < RB; j++)
                if (r >> j & 1) y ^= S::at(c[j]);
            x[r] = sp[y];
            if (REV) l[r] = sl[y];
        }
    } else {
#pragma unroll
        for (int r = 0; r < N; r++) {
            x[r] = T{0, 0};
            if (REV) l[r] = T{0, 0};
        }
    }
    if (P.moves) __syncthreads();  // everything read before anything is written
    if (P.diag >= 0 && warp_on) {
        const typename S::Phase* tab = tables + size_t(P.diag) * kSwTable;
        const int lane = p & 31, warp = p >> 5;
        if (REV) {
            // w = Im(conj(lambda) psi); the sum over the tile with the sign of each tile bit
            A sum = S::zero(), sj[3] = {S::zero(), S::zero(), S::zero()};
            if constexpr (sizeof(T) == 16) {
                A w[N];
#pragma unroll
                for (int r = 0; r < N; r++) w[r] = sw_cross(l[r], x[r]);
#pragma unroll
                for (int j = RB - 1; j >= 0; j--) {  // halve: sums over bit j stay, differences are its signed sum
                    A d = 0;
#pragma unroll
                    for (int r = 0; r < (1 << j); r++) {
                        const A lo = w[r], hi = w[r | (1 << j)];
                        d = r == 0 ? lo - hi : d + (lo - hi);
                        w[r] = lo + hi;
                    }
                    sj[j] = d;
                }
                sum = w[0];
            } else {
                // chains of four products across the top register bit, then compensated sums
                constexpr int H = N / 2;
#pragma unroll
                for (int r = 0; r < H; r++) {
                    const float2 a = x[r], b = x[r + H], u = l[r], v = l[r + H];
                    const float w0 = __fmaf_rn(u.x, a.y, __fmul_rn(-u.y, a.x));
                    const float s = __fmaf_rn(v.x, b.y, __fmaf_rn(-v.y, b.x, w0));
                    const float d = __fmaf_rn(-v.x, b.y, __fmaf_rn(v.y, b.x, w0));
                    sum.add(s);
                    sj[RB - 1].add(d);
                    if (RB > 1) sj[0].add((r & 1) ? -s : s);
                    if (RB > 2) sj[1].add((r & 2) ? -s : s);
                }
            }
            // lane m of the butterfly ends with the sum over lanes signed by parity(lane & m)
            A v = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const A q = S::shfl_xor(v, o);
                v = (lane & o) ? S::add(q, S::neg(v)) : S::add(v, q);
            }
            const A all = S::shfl(v, 0);
            const A rs = sw_warp_sum4<T>(sj[0], sj[1], sj[2], S::zero());  // register bit j on lanes 8 j ..
            // one lane per tile bit adds its sum: lanes 1, 2, 4, 8, 16 the lane bits, 3, 5, 6, 7 the warp
            // bits (the whole warp's sum, by the warp's sign), 9, 17, 25 register bits 0, 1, 2
            int bit = -1;
            A mine = v;
            if (lane && !(lane & (lane - 1))) {
                bit = __ffs(lane) - 1;
                if (bit >= TB) bit = -1;
            } else if (lane == 3 || (lane >= 5 && lane <= 7)) {
                const int k = lane == 3 ? 0 : lane - 4;
                mine = (warp >> k & 1) ? S::neg(all) : all;
                bit = 5 + k < TB ? 5 + k : -1;
            }
            const A reg = S::shfl(rs, lane == 9 ? 0 : lane == 17 ? 8 : 16);
            if (lane == 9 || lane == 17 || lane == 25) {
                const int j = lane == 9 ? 0 : lane == 17 ? 1 : 2;
                mine = reg;
                bit = j < RB ? TB + j : -1;
            }
            const int slot = bit >= 0 ? int(P.zrot[bit]) : -1;
            if (slot >= 0) S::gather(sacc[slot * kSwWarps + warp], mine);
        }
        const uint32_t tmask = (1u << (tq < 5 ? tq : 5)) - 1u;
        if (P.phase_first) {  // never in the reverse walk; without the branch there it spills more (complex64 batches +1 %)
#pragma unroll
            for (int r = 0; r < N; r++) {
                const uint32_t y = from(r);
                const typename S::Phase ph = sw_phase2(tab[y & tmask], tab[32 + (y >> 5)]);
                x[r] = sw_phase(ph, x[r]);
            }
        } else {
#pragma unroll
            for (int r = 0; r < N; r++) {
                const uint32_t i = p | (uint32_t(r) << TB);
                const typename S::Phase ph = sw_phase2(tab[i & tmask], tab[32 + (i >> 5)]);
                x[r] = sw_phase(ph, x[r]);
                if (REV) l[r] = sw_phase(ph, l[r]);
            }
        }
    }
    if (on) {
#pragma unroll
        for (int r = 0; r < N; r++) {
            const uint32_t i = S::at(p) ^ S::at(uint32_t(r) << TB);
            sp[i] = x[r];
            if (REV) sl[i] = l[r];
        }
    }
}

// ---- a fixed gate on one tile. A dense gate takes pairs; a monomial one is a gather like a moves pass,
// amplitude x taking its source row's value times its row's factor.
template <typename T>
struct SwEntry {  // entry i of a fixed gate, times a value, on top of an accumulator
    using R = decltype(T().x);
    const TileOp& op;
    __device__ __forceinline__ T mac(T acc, int i, T v) const {
        if constexpr (sizeof(R) == 4)  // the host-rounded float copy: no FP64-pipe conversions per thread
            return cfma(op.mf[2 * i], op.mf[2 * i + 1], v, acc);
        else
            return cfma(op.m[2 * i], op.m[2 * i + 1], v, acc);
    }
};
template <>
struct SwEntry<FxC> {  // the builder leaves the entries' limbs in dfh (high) and dfl (low)
    const TileOp& op;
    __device__ __forceinline__ FxLimb limb(int i) const {
        const int h = __float_as_int(op.dfh[i]), l = __float_as_int(op.dfl[i]);
        return FxLimb{h, l, (1ll << 29) + (l >> 1), fx_one()};
    }
    __device__ __forceinline__ FxC mac(FxC acc, int i, FxC v) const {
        const FxLimb re = limb(2 * i), im = limb(2 * i + 1);
        return FxC{fx_mac(fx_mac(acc.x, v.x, re), v.y, fx_neg(im)), fx_mac(fx_mac(acc.y, v.y, re), v.x, im)};
    }
};

template <typename T, int RB>
__device__ __noinline__ void sw_fixed(T* s, const TileOp& op, uint32_t tsize, int tq, int nthreads) {
    using S = Sw<T>;
    const SwEntry<T> e{op};
    const T nil{0, 0};
    if (op.kind == OP_DENSE || op.kind == OP_DENSE_REAL) {
        uint32_t seg[5];
#pragma unroll
        for (int j = 0; j < 5; j++) seg[j] = op.seg[j];
        const uint32_t tb = op.off[1], ntup = tsize >> op.npos;
        for (uint32_t p = threadIdx.x; p < ntup; p += nthreads) {
            const uint32_t i = tuple_index(p, op.npos, seg, op.pos, op.lfixval);
            const uint32_t i0 = S::at(i), i1 = S::at(i | tb);
            const T a = s[i0], b = s[i1];
            s[i0] = e.mac(e.mac(nil, 1, b), 0, a);
            s[i1] = e.mac(e.mac(nil, 3, b), 2, a);
        }
        return;  // the caller's barrier follows
    }
    constexpr int N = 1 << RB;
    const int TB = tq - RB, k = op.k;
    const uint32_t p = threadIdx.x;
    const bool on = p < (tsize >> RB);
    uint32_t fix = 0;  // controls inside the tile
    for (int i = 0; i < op.npos; i++) fix |= 1u << op.pos[i];
    for (int j = 0; j < k; j++) fix &= ~(1u << op.tb[j]);
    T x[N];
    int row[N];
#pragma unroll
    for (int r = 0; r < N; r++) {
        const uint32_t i = p | (uint32_t(r) << TB);
        int q = 0;
        for (int j = 0; j < k; j++) q |= int(i >> op.tb[j] & 1u) << j;
        row[r] = on && (i & fix) == op.lfixval && op.pf[q] != PF_SKIP_DEV ? q : -1;
        if (row[r] >= 0) x[r] = s[S::at(i ^ op.off[q] ^ op.offsrc[q])];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < N; r++) {
        if (row[r] < 0) continue;
        s[S::at(p | (uint32_t(r) << TB))] =
            op.pf[row[r]] == 255 ? e.mac(nil, row[r], x[r]) : apply_pf(x[r], op.pf[row[r]]);
    }
}

// The factor tables of a program: entry i of the low part is the product of the phases of tile bits
// 0..4 at i, entry j of the high part that of the bits from 5 on; sigma goes into the first table.
// RZ(theta) multiplies bit 0 by c - i s and bit 1 by c + i s; the inverse the other way. Formed in fixed
// point for fixed-point tiles: an entry's error is common to every amplitude that it multiplies, and
// FP64 products (2^-53 each) left three times the error on a gradient, in ten times the time. Complex64 tables
// are formed in float pairs, right to 2^-44 of each part however small it is, and rounded to floats once.
template <typename T>
__device__ __forceinline__ void sw_tables(typename Sw<T>::Phase* tables, const SweepPass* passes, int npass, int tq,
                                          bool rev, const SweepCoef* __restrict__ coef, double sigma, int nthreads) {
    constexpr bool F64 = sizeof(typename Sw<T>::Coef) == 16;
    for (int k = 0; k < npass; k++) {
        const SweepPass& P = passes[k];
        if (P.kind != SW_MOVE || P.diag < 0) continue;
        for (int e = threadIdx.x; e < kSwTable; e += nthreads) {
            const bool high = e >= 32;
            const int lo = high ? 5 : 0, hi = high ? tq : (tq < 5 ? tq : 5), i = high ? e - 32 : e;
            const double start = high && P.diag == 0 ? sigma : 1.0;
            typename Sw<T>::Phase& out = tables[size_t(P.diag) * kSwTable + e];
            if constexpr (F64) {
                double re = start, im = 0.0;
                for (int b = lo; b < hi; b++) {
                    if (P.zrot[b] < 0) continue;
                    const SweepCoef& c = coef[P.zrot[b]];
                    const bool plus = ((i >> (b - lo) & 1) != 0) != rev;
                    const double s = plus ? c.s : sw_neg(c.s);
                    const double r = fma(re, c.c, -(im * s));
                    im = fma(re, s, im * c.c);
                    re = r;
                }
                out = make_double2(re, im);
            } else if constexpr (sizeof(T) == 8) {
                float rh = 1.0f, rl = 0.0f, ih = 0.0f, il = 0.0f;
                if (start != 1.0) df_split(start, rh, rl);
                for (int b = lo; b < hi; b++) {
                    if (P.zrot[b] < 0) continue;
                    const SweepCoef& c = coef[P.zrot[b]];
                    const bool plus = ((i >> (b - lo) & 1) != 0) != rev;
                    const float ch = __int_as_float(c.ph), cl = __int_as_float(c.pl);
                    float sh = __int_as_float(c.sh), sl = __int_as_float(c.sl);
                    if (!plus) sh = -sh, sl = -sl;
                    float th, tl;
                    df_lin2(ch, cl, rh, rl, -sh, -sl, ih, il, th, tl);
                    df_lin2(ch, cl, ih, il, sh, sl, rh, rl, ih, il);
                    rh = th, rl = tl;
                }
                out = make_float2(__fadd_rn(rh, rl), __fadd_rn(ih, il));
            } else {
                FxC v{start == 1.0 ? 1ll << 60 : __double2ll_rn(start * kFxOne), 0};
                for (int b = lo; b < hi; b++) {
                    if (P.zrot[b] < 0) continue;
                    const SweepCoef& c = coef[P.zrot[b]];
                    const bool plus = ((i >> (b - lo) & 1) != 0) != rev;
                    v = sw_phase(make_int4(c.ph, c.pl, plus ? c.sh : -c.sh, plus ? c.sl : -c.sl), v);
                }
                out = Sw<T>::phase(v);
            }
        }
    }
}

// A program on one tile; ends behind a barrier. Every thread of the block calls it.
template <typename T, int RB, bool REV>
__device__ __forceinline__ void sw_program(T* sp, T* sl, int tq, uint64_t tile_base, const SweepPass* passes, int npass,
                                           const TileOp* __restrict__ fixed, const typename Sw<T>::Coef* coef,
                                           const typename Sw<T>::Phase* tables, typename Sw<T>::Cell* sacc,
                                           int nthreads) {
    const uint32_t tsize = 1u << tq;
#pragma unroll 1
    for (int k = 0; k < npass; k++) {
        const SweepPass& P = passes[k];
        if (P.kind == SW_ROT) {
            sw_rotations<T, RB, REV>(sp, sl, tsize, P, coef, sacc);
        } else if (P.kind == SW_MOVE) {
            sw_moves<T, RB, REV>(sp, sl, tsize, tq, tile_base, P, tables, sacc);
        } else {
            const TileOp& op = fixed[P.op];
            if ((tile_base & op.omask) == op.oval) {
                sw_fixed<T, RB>(sp, op, tsize, tq, nthreads);
                if (REV) sw_fixed<T, RB>(sl, op, tsize, tq, nthreads);
            }
        }
        __syncthreads();
    }
}

// ---- tiles in and out
// A double on the scale 2^k, |x| 2^k <= 2^60, rounded to an integer (integer instructions only).
__device__ __forceinline__ long long fx_from(double v, int k) {
    const long long bits = __double_as_longlong(v);
    const int e = int(bits >> 52) & 0x7ff;
    const long long m = ((bits & 0xfffffffffffffll) | (1ll << 52)) << 7;  // bit 59
    const int d = 1082 - k - e;                                            // v 2^k = m 2^-d
    long long r = d > 60 || e == 0 ? 0ll : d > 0 ? (m + (1ll << (d - 1))) >> d : m << -d;
    return bits < 0 ? -r : r;
}
// X 2^-k as a double, rounded once.
__device__ __forceinline__ double fx_to(long long X, int k) {
    const double d = __ll2double_rn(X);
    const int hi = __double2hiint(d), e = ((hi >> 20) & 0x7ff) - k;
    if (X == 0) return 0.0;
    if (e < 1 || e > 2046) return fx_to_double_any(X, -k);  // out of line: inlined, its FP64 operations issue for every X
    return __hiloint2double(hi - (k << 20), __double2loint(d));
}

// A tile's scale from the raw doubles its threads hold in shared memory: per warp the largest exponent
// field and the sum of squares relative to it, combined over the block through `box` (kSwWarps entries).
// k: the tile's norm times 2^k is at most 2^60. Returns false when a component is infinite or NaN.
struct FxWarpNorm {
    int e;
    float sum;
};
__device__ __forceinline__ uint32_t fx_field(double v) { return (uint32_t(__double2hiint(v)) >> 20) & 0x7ffu; }
__device__ __forceinline__ float fx_relative(double v, uint32_t e) {  // |v| 2^(1023 - e), truncated to 24 bits
    const uint32_t hi = uint32_t(__double2hiint(v)), lo = uint32_t(__double2loint(v));
    const uint32_t f = (hi >> 20) & 0x7ffu;
    if (f + 60u < e || f == 0u) return 0.0f;
    return __uint_as_float(((f + 127u - e) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
}
__device__ __forceinline__ void fx_warp_norm(const double2* raw, uint32_t tsize, int nt, FxWarpNorm* box) {
    uint32_t e = 0;
    const uint32_t ap = Sw<FxC>::at(threadIdx.x);
    for (uint32_t i = 0; i + threadIdx.x < tsize; i += nt) {
        const double2 v = raw[ap ^ Sw<FxC>::at(i)];
        e = max(e, max(fx_field(v.x), fx_field(v.y)));
    }
    e = __reduce_max_sync(0xffffffffu, e);
    float s = 0.0f;
    if (e != 0u && e != 0x7ffu)
        for (uint32_t i = 0; i + threadIdx.x < tsize; i += nt) {
            const double2 v = raw[ap ^ Sw<FxC>::at(i)];
            const float a = fx_relative(v.x, e), b = fx_relative(v.y, e);
            s = fmaf(a, a, fmaf(b, b, s));
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) box[threadIdx.x >> 5] = FxWarpNorm{int(e), s};
}
// Returns the tile's largest exponent field: 0 without a normal number, 0x7ff with an infinity or NaN.
__device__ __forceinline__ int fx_scale(const FxWarpNorm* box, int nwarps, int* k) {
    int e = 0;
    for (int w = 0; w < nwarps; w++) e = max(e, box[w].e);
    if (e == 0x7ff) return e;
    float sum = 0.0f;
    for (int w = 0; w < nwarps; w++) {
        const int d = 2 * (e - box[w].e);
        if (d < 100) sum = fmaf(box[w].sum, __uint_as_float(uint32_t(127 - d) << 23), sum);
    }
    // squares of truncated values: a margin of 2^-18; norm^2 < 2^(h + 1) 2^(2 (e - 1023))
    const int h = int(__float_as_uint(sum * 1.000004f) >> 23) - 127;
    *k = sum > 0.0f ? 60 - ((h + 2) >> 1) - (e - 1023) : 0;
    return e;
}

// Shared memory of a program beside its tiles, in this order.
template <typename T>
struct SweepSide {
    typename Sw<T>::Phase* tables;
    typename Sw<T>::Coef* coef;
    typename Sw<T>::Cell* sacc;  // [rotation][warp]
    double* total;           // [rotation]: fixed-point tiles' sums so far
    SweepPass* passes;
    FxWarpNorm* box;         // 2 * kSwWarps
    uint64_t* rowoff;        // 2^RH row offsets
    static __host__ __device__ constexpr size_t up(size_t x) { return (x + 15) / 16 * 16; }
    static __host__ __device__ constexpr size_t bytes(int npass, int nrot, int ndiag, bool rev, int rh) {
        return up(size_t(ndiag) * kSwTable * sizeof(typename Sw<T>::Phase)) + up(size_t(nrot) * sizeof(typename Sw<T>::Coef)) +
               (rev ? up(size_t(nrot) * (kSwWarps + 1) * sizeof(double)) : 0) + size_t(npass) * sizeof(SweepPass) +
               2 * kSwWarps * sizeof(FxWarpNorm) + (size_t(8) << rh);
    }
    __device__ __forceinline__ SweepSide(unsigned char* p, int npass, int nrot, int ndiag, bool rev) {
        tables = reinterpret_cast<typename Sw<T>::Phase*>(p);
        p += up(size_t(ndiag) * kSwTable * sizeof(typename Sw<T>::Phase));
        coef = reinterpret_cast<typename Sw<T>::Coef*>(p);
        p += up(size_t(nrot) * sizeof(typename Sw<T>::Coef));
        sacc = reinterpret_cast<typename Sw<T>::Cell*>(p);
        total = reinterpret_cast<double*>(p) + size_t(nrot) * kSwWarps;
        p += rev ? up(size_t(nrot) * (kSwWarps + 1) * sizeof(double)) : 0;
        passes = reinterpret_cast<SweepPass*>(p);
        p += size_t(npass) * sizeof(SweepPass);
        box = reinterpret_cast<FxWarpNorm*>(p);
        rowoff = reinterpret_cast<uint64_t*>(p + 2 * kSwWarps * sizeof(FxWarpNorm));
    }
};

// Fills a program's side tables; a barrier follows.
template <typename T>
__device__ __forceinline__ void sw_begin(const SweepSide<T>& side, const SweepPass* __restrict__ passes, int npass,
                                         const SweepCoef* __restrict__ coef, int nrot, int tq, bool rev, double sigma,
                                         int nt) {
    const uint4* from = reinterpret_cast<const uint4*>(passes);
    uint4* to = reinterpret_cast<uint4*>(side.passes);
    for (int w = threadIdx.x; w < npass * int(sizeof(SweepPass) / 16); w += nt) to[w] = from[w];
    if (rev)
        for (int i = threadIdx.x; i < nrot * (kSwWarps + 1); i += nt) reinterpret_cast<uint64_t*>(side.sacc)[i] = 0ull;
    for (int i = threadIdx.x; i < nrot; i += nt) side.coef[i] = Sw<T>::coef(coef[i]);
    __syncthreads();
    sw_tables<T>(side.tables, side.passes, npass, tq, rev, coef, sigma, nt);
    __syncthreads();
}

// ---- coefficients from angles
struct SweepRot {
    int angle;  // index of (cos, sin) of theta / 2
    int axis;
};
struct SweepRange {
    int pass0, npass, coef0, nrot;
    int ndiag, floating, single, pad;
};

// One block per program: the coefficients of its rotations from (cos, sin) of half their angles and, for
// floating tiles, the common factors they leave out: *sigma is their product, which the phases of the
// first factor table carry (without one, the tile is scaled as it is written back), and an inner
// product comes out of the tile 1 / weight times its value (psi and lambda both lack what was left
// out so far). Fixed-point tiles leave nothing out.
__device__ __forceinline__ void sw_times(double& hi, double& lo, double bh, double bl) {  // an unevaluated sum
    const double p = hi * bh;
    const double e = fma(hi, bh, -p) + fma(hi, bl, lo * bh);
    hi = p + e;
    lo = e - (hi - p);
}
static __global__ void __launch_bounds__(64) k_sweep_coefs(const SweepRange* __restrict__ ranges,
                                                           const SweepPass* __restrict__ passes,
                                                           const SweepRot* __restrict__ rots,
                                                           const double2* __restrict__ angles,
                                                           SweepCoef* __restrict__ coefs, double* __restrict__ weights,
                                                           double* __restrict__ sigmas) {
    __shared__ double fh[kSwMaxRot], fl[kSwMaxRot];
    const SweepRange R = ranges[blockIdx.x];
    for (int r = threadIdx.x; r < R.nrot; r += blockDim.x) {
        const SweepRot rot = rots[R.coef0 + r];
        const double2 cs = angles[rot.angle];
        SweepCoef o{};
        o.c = cs.x;
        o.s = cs.y;
        fh[r] = 1.0;
        fl[r] = 0.0;
        const bool cot = fabs(cs.y) > fabs(cs.x);
        if (rot.axis != QS_GATE_RZ && R.floating) {
            double t = cot ? -cs.x / cs.y : cs.y / cs.x;
            if (R.single) t = double(float(t));
            // the factor follows the rounded t: 1 / sqrt(1 + t^2) with a correction step, its residual by
            // exact products, so that a whole program's product is right to double accuracy
            const double u = t * t, ue = fma(t, t, -u), a = 1.0 + u, ae = u - (a - 1.0);
            double g = 1.0 / sqrt(a);
            const double g2 = g * g, g2e = fma(g, g, -g2);
            double lo = 0.5 * g * (fma(-g2, a, 1.0) - g2e * a - g2 * (ae + ue));
            if ((cot ? cs.y : cs.x) < 0.0) g = -g, lo = -lo;
            o.c = t;
            o.s = cot ? 1.0 : 0.0;
            fh[r] = g;
            fl[r] = lo;
        } else if (rot.axis != QS_GATE_RZ) {
            // theta / 2 = a + k pi / 2: sin a and cos a > 0 are the pair, exchanged or not, up to sign
            double s0 = cot ? -cs.x : cs.y, c0 = cot ? cs.y : cs.x;
            if (c0 < 0.0) s0 = -s0, c0 = -c0;
            const double d = 1.0 + c0, p = s0 / d, rest = (fma(-p, d, s0) - p * (c0 - (d - 1.0))) / d;
            const FxLimb lp = fx_limb(-(__double2ll_rn(p * kFxOne) + __double2ll_rn(rest * kFxOne)));
            const FxLimb ls = fx_limb(__double2ll_rn(s0 * kFxOne));
            o.ph = lp.h, o.pl = lp.l, o.pk = lp.k;
            o.sh = ls.h, o.sl = ls.l, o.sk = ls.k;
            o.quarter = cot ? 1 : 0;
        } else {
            const FxLimb lc = fx_limb(__double2ll_rn(cs.x * kFxOne)), ls = fx_limb(__double2ll_rn(cs.y * kFxOne));
            o.ph = lc.h, o.pl = lc.l;
            o.sh = ls.h, o.sl = ls.l;
            if (R.single) {
                float h, l;
                df_split(cs.x, h, l);
                o.ph = __float_as_int(h), o.pl = __float_as_int(l);
                df_split(cs.y, h, l);
                o.sh = __float_as_int(h), o.sl = __float_as_int(l);
            }
        }
        coefs[R.coef0 + r] = o;
        weights[R.coef0 + r] = 1.0;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    double th = 1.0, tl = 0.0;
    if (R.floating && R.single) {
        for (int r = 0; r < R.nrot; r++) th *= fh[r];
        double sh = 1.0;
        for (int k = 0; k < R.npass; k++) {
            const SweepPass& q = passes[R.pass0 + k];
            if (q.kind == SW_ROT) {
                for (int j = 0; j < 3; j++)
                    if (q.rot[j] >= 0) weights[R.coef0 + q.rot[j]] = sh * sh;
                for (int j = 0; j < 3; j++)
                    if (q.rot[j] >= 0) sh *= fh[q.rot[j]];
            }
            if (q.kind == SW_MOVE && q.diag >= 0) {
                for (int b = 0; b < kSwMaxT; b++)
                    if (q.zrot[b] >= 0) weights[R.coef0 + q.zrot[b]] = sh * sh;
                if (q.diag == 0) sh /= th;
            }
        }
    } else if (R.floating) {
        for (int r = 0; r < R.nrot; r++) sw_times(th, tl, fh[r], fl[r]);
        double sh = 1.0, sl = 0.0;  // true amplitudes over those in the tile
        for (int k = 0; k < R.npass; k++) {
            const SweepPass& q = passes[R.pass0 + k];
            if (q.kind == SW_ROT) {
                for (int j = 0; j < 3; j++)
                    if (q.rot[j] >= 0) weights[R.coef0 + q.rot[j]] = sh * sh;
                for (int j = 0; j < 3; j++)
                    if (q.rot[j] >= 0) sw_times(sh, sl, fh[q.rot[j]], fl[q.rot[j]]);
            }
            if (q.kind == SW_MOVE && q.diag >= 0) {
                for (int b = 0; b < kSwMaxT; b++)
                    if (q.zrot[b] >= 0) weights[R.coef0 + q.zrot[b]] = sh * sh;
                if (q.diag == 0) {
                    const double back = 1.0 / th;
                    sw_times(sh, sl, back, fma(-th, back, 1.0) * back - tl * back * back);
                }
            }
        }
    }
    sigmas[blockIdx.x] = th;
}

// A program's sum of rotation r over the block's tiles.
template <typename T>
__device__ __forceinline__ double sw_total(const SweepSide<T>& side, int r, int nt) {
    if constexpr (sizeof(T) == 16 && sizeof(typename Sw<T>::Coef) != 16) {
        return side.total[r];
    } else {
        double v = 0.0;
        for (int w = 0; w < (nt + 31) / 32; w++) v += Sw<T>::value(side.sacc[r * kSwWarps + w]);
        return v;
    }
}

// ---- a range of tiles of one stage through a program, by one block: what the single-circuit launches
// and the batched kernel share. LD reads global memory (the batched kernel bypasses L1).
struct SweepTile {
    int T, RL, npass, nrot, ndiag;
    bool store;           // false: nothing reads the vectors afterwards
    double sigma;
};

template <typename T, int RB, bool REV, bool CG>
__device__ __forceinline__ void sw_tile(const typename Sw<T>::Glob* src, typename Sw<T>::Glob* psi,
                                        typename Sw<T>::Glob* lam, uint64_t base, const SweepTile& t, T* sp, T* sl,
                                        const SweepSide<T>& side, const TileOp* __restrict__ fixed, int nt) {
    using S = Sw<T>;
    using G = typename S::Glob;
    constexpr bool FX = sizeof(T) == 16 && sizeof(typename S::Coef) != 16;
    const uint32_t tsize = 1u << t.T, rmask = (1u << t.RL) - 1u, p = threadIdx.x;
    G* rp = reinterpret_cast<G*>(sp);
    G* rl = reinterpret_cast<G*>(sl);
    // element k of a thread is p | k nt: its place in memory and in the tile are those of p and of k nt put
    // together (disjoint bits), the latter the same for the whole block
    const uint64_t gp = base + side.rowoff[(p & (tsize - 1u)) >> t.RL] + (p & rmask);
    const uint32_t ap = S::at(p);
    auto place = [&](uint32_t i, uint64_t* g, uint32_t* at) {  // i = k nt
        *g = gp + (side.rowoff[i >> t.RL] + (i & rmask));
        *at = ap ^ S::at(i);
    };
    // A tile of zeros goes through no program (from a basis state most tiles of a forward run's first stages are:
    // 20 qubits, 12 stages). Fixed-point tiles know from their norm; complex64 tiles OR their bits, and a program
    // with a dense fixed gate runs all the same: its entries may overflow a float.
    uint32_t any = 0;
#pragma unroll 8
    for (uint32_t i = 0; i + p < tsize; i += nt) {
        uint64_t g;
        uint32_t at;
        place(i, &g, &at);
        const G v = CG ? __ldcg(src + g) : src[g];
        rp[at] = v;
        if constexpr (sizeof(T) == 8) any |= (__float_as_uint(v.x) | __float_as_uint(v.y)) << 1;
        if (REV) {
            const G w = CG ? __ldcg(lam + g) : lam[g];
            rl[at] = w;
            if constexpr (sizeof(T) == 8) any |= (__float_as_uint(w.x) | __float_as_uint(w.y)) << 1;
        }
    }
    int kp = 0, kl = 0;
    double unit = 1.0;
    bool finite = true, live = true;
    if constexpr (FX) {  // each thread converts the elements it loaded
        const int nw = (nt + 31) / 32;
        fx_warp_norm(rp, tsize, nt, side.box);
        if (REV) fx_warp_norm(rl, tsize, nt, side.box + kSwWarps);
        __syncthreads();
        const int ep = fx_scale(side.box, nw, &kp), el = REV ? fx_scale(side.box + kSwWarps, nw, &kl) : 0;
        finite = ep != 0x7ff && el != 0x7ff;
        live = finite && (ep | el) != 0;
        if (finite) {
            const int eu = 1023 + 60 - kp - kl;
            unit = eu > 0 && eu < 2047 ? __hiloint2double(eu << 20, 0) : fx_to_double_any(1, eu - 1023);
            for (uint32_t i = 0; i + p < tsize; i += nt) {
                const uint32_t at = ap ^ S::at(i);
                const double2 v = rp[at];
                sp[at] = T{fx_from(v.x, kp), fx_from(v.y, kp)};
                if (REV) {
                    const double2 w = rl[at];
                    sl[at] = T{fx_from(w.x, kl), fx_from(w.y, kl)};
                }
            }
        }
    }
    if constexpr (sizeof(T) == 8) {
        live = __syncthreads_or(any != 0);
        for (int k = 0; k < t.npass && !live; k++) live = side.passes[k].kind == SW_FIXED;
    } else {
        __syncthreads();
    }
    if (live) {
        sw_program<T, RB, REV>(sp, sl, t.T, base, side.passes, t.npass, fixed, side.coef, side.tables, side.sacc, nt);
    }
    if constexpr (FX && REV) {  // the tile's sums on its own scale (undefined with an infinity or NaN in it)
        for (int r = threadIdx.x; r < t.nrot; r += nt) {
            long long v = 0;
            for (int w = 0; w < (nt + 31) / 32; w++) {
                v += side.sacc[r * kSwWarps + w];
                side.sacc[r * kSwWarps + w] = 0;
            }
            side.total[r] = finite ? fma(double(v), unit, side.total[r]) : __longlong_as_double(0x7ff8ll << 48);
        }
    }
    if (t.store) {
        const bool scaled = !FX && t.ndiag == 0;
        for (uint32_t i = 0; i + p < tsize; i += nt) {
            uint64_t g;
            uint32_t at;
            place(i, &g, &at);
            auto out = [&](const T* s, int k) {
                G v;
                if constexpr (FX) {
                    const T a = s[at];
                    if (finite) v = G{fx_to(a.x, k), fx_to(a.y, k)};
                    else v.x = v.y = __longlong_as_double(0x7ff8ll << 48);
                } else {
                    v = s[at];
                    if (scaled) v.x *= decltype(v.x)(t.sigma), v.y *= decltype(v.y)(t.sigma);
                }
                return v;
            };
            const G v = out(sp, kp);
            if (CG) __stcg(psi + g, v);
            else psi[g] = v;
            if (REV) {
                const G w = out(sl, kl);
                if (CG) __stcg(lam + g, w);
                else lam[g] = w;
            }
        }
    }
    __syncthreads();
}

}  // namespace qs
