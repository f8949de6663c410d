// qs_rot.cuh — double-float rotation arithmetic (FP32 pipe) shared by the adjoint and the batch kernel for
// complex128 states in QS_ARITH_DF64: R_A(theta) = cos(theta/2) I - i sin(theta/2) A on an amplitude pair
// (a, b) = (bit 0, bit 1), and the pair's term of Im<lambda|A|psi>.
#pragma once

#include <cuda_runtime.h>

#include "qs_device.cuh"
#include "qs_reduce.cuh"

namespace qs {

// ---- double-float forms. Amplitudes as float4 (re_hi, re_lo, im_hi, im_lo); each pair's
// Im<lambda|A|psi> is a double-float dot product (df_dot_pair), added to a compensated float-pair
// accumulator: no FP64 operation per pair.
template <int AXIS>
__device__ __forceinline__ void adj_im_df_acc(DfAcc& acc, float4 l0, float4 l1, float4 a, float4 b) {
    // terms u * x of Im<lambda|A|psi> (rows with the target bit 0: a, l0; 1: b, l1):
    // u from lambda, x from psi
    float uh[4], ul[4], xh[4], xl[4];
    auto set = [&](int k, float vh, float vl, float wh, float wl, bool neg) {
        uh[k] = neg ? -vh : vh;
        ul[k] = neg ? -vl : vl;
        xh[k] = wh;
        xl[k] = wl;
    };
    if (AXIS == QS_GATE_RX) {  // l0.re*b.im - l0.im*b.re + l1.re*a.im - l1.im*a.re
        set(0, l0.x, l0.y, b.z, b.w, false); set(1, l0.z, l0.w, b.x, b.y, true);
        set(2, l1.x, l1.y, a.z, a.w, false); set(3, l1.z, l1.w, a.x, a.y, true);
    } else if (AXIS == QS_GATE_RY) {  // l1.re*a.re + l1.im*a.im - l0.re*b.re - l0.im*b.im
        set(0, l1.x, l1.y, a.x, a.y, false); set(1, l1.z, l1.w, a.z, a.w, false);
        set(2, l0.x, l0.y, b.x, b.y, true); set(3, l0.z, l0.w, b.z, b.w, true);
    } else {  // l0.re*a.im - l0.im*a.re - l1.re*b.im + l1.im*b.re
        set(0, l0.x, l0.y, a.z, a.w, false); set(1, l0.z, l0.w, a.x, a.y, true);
        set(2, l1.x, l1.y, b.z, b.w, true); set(3, l1.z, l1.w, b.x, b.y, false);
    }
    float h, l;
    df_dot_pair<4>(uh, ul, xh, xl, h, l);
    acc.add(h);
    acc.c = __fadd_rn(acc.c, l);
}

// c * p + q2 * r in double-float, with (c, s) = (ch + cl, sh + sl).
__device__ __forceinline__ void df_lin2(float ch, float cl, float p_h, float p_l, float dh, float dl, float q_h,
                                        float q_l, float& oh, float& ol) {
    const float uh[2] = {ch, dh}, ul[2] = {cl, dl}, xh[2] = {p_h, q_h}, xl[2] = {p_l, q_l};
    df_dot_pair<2>(uh, ul, xh, xl, oh, ol);
}

template <int AXIS>
__device__ __forceinline__ void df_rot_pair(float ch, float cl, float sh, float sl, float4& a, float4& b) {
    float4 na, nb;
    if (AXIS == QS_GATE_RY) {  // [[c, -s], [s, c]]
        df_lin2(ch, cl, a.x, a.y, -sh, -sl, b.x, b.y, na.x, na.y);
        df_lin2(ch, cl, a.z, a.w, -sh, -sl, b.z, b.w, na.z, na.w);
        df_lin2(sh, sl, a.x, a.y, ch, cl, b.x, b.y, nb.x, nb.y);
        df_lin2(sh, sl, a.z, a.w, ch, cl, b.z, b.w, nb.z, nb.w);
    } else if (AXIS == QS_GATE_RZ) {  // diag(c - i s, c + i s)
        df_lin2(ch, cl, a.x, a.y, sh, sl, a.z, a.w, na.x, na.y);
        df_lin2(ch, cl, a.z, a.w, -sh, -sl, a.x, a.y, na.z, na.w);
        df_lin2(ch, cl, b.x, b.y, -sh, -sl, b.z, b.w, nb.x, nb.y);
        df_lin2(ch, cl, b.z, b.w, sh, sl, b.x, b.y, nb.z, nb.w);
    } else {  // RX: [[c, -i s], [-i s, c]]
        df_lin2(ch, cl, a.x, a.y, sh, sl, b.z, b.w, na.x, na.y);
        df_lin2(ch, cl, a.z, a.w, -sh, -sl, b.x, b.y, na.z, na.w);
        df_lin2(ch, cl, b.x, b.y, sh, sl, a.z, a.w, nb.x, nb.y);
        df_lin2(ch, cl, b.z, b.w, -sh, -sl, a.x, a.y, nb.z, nb.w);
    }
    a = na;
    b = nb;
}

}  // namespace qs
