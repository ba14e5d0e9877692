// wf_kw_ff.cuh -- the split form's solve of the surface kinematic wave, in double-FP32.
#pragma once

#include "wf_ff.cuh"

namespace wfk {

constexpr double KIN_WAVE_MIN_FLOW_QROOT = 0x1.0c6f7a0b5ed8ap-20;  // 1e-30^0.2 (routing/utils.jl:2)

// Root of dt_dx u^5 + alpha u^3 = cterm for the kinematic wave in u = Q^0.2 (the reference's
// Newton-Raphson on Q, surface_process.jl:24-70, written for u), in double-FP32: Newton
// iterations in FP32 from the previous u, held below the upper bound min((cterm/alpha)^(1/3),
// (cterm/dt_dx)^(1/5)) (computed beside the first iteration; the start without a previous u), until
// |du| <= 1e-4 u (an error below 2 du^2 / u, less than the rounding of FP32), then one Newton
// correction with the residual evaluated in double-FP32. Q = u^5 is formed from the correction du as
// v^5 - 5 v^4 du (the dropped terms are of relative size 10 (du/v)^2). Results below the
// reference's floor (u = QROOT) are raised to it, as the reference does.
//
// Error of Q (tests/test_split_solve_gpu.py): v is within 2e-7 of the root, the FP32 derivative and
// division put the correction off by 3e-7 of it and its own Newton error is below 2 (2e-7)^2, 1.4e-13 of
// u or 7e-13 of Q. Measured over 4 million roots: at most 2.1e-13, 1.4e-14 in the mean square, the
// same as with iterations until |du| <= 3e-7 u.
//
// The floor discharge QROOT^5 is 9.999999999999968e-31, just below KIN_WAVE_MIN_FLOW, so a cell
// whose solve ended at the floor does not count as flowing in the Courant quantile of adaptive
// sub-stepping; a floored cell whose next solve stops at once (kw_node_ff) keeps
// pow(q, 0.2)^5 = 1.000000000000002e-30, just above it, and counts from then on. Both values
// are held exactly as double-FP32 pairs (the low parts are FP32 subnormals).
__device__ __forceinline__ wff::ff q_floor() { return {__uint_as_float(0x0da24260u), __uint_as_float(0x802287aeu)}; }
__device__ __forceinline__ wff::ff q_rest() { return {__uint_as_float(0x0da24260u), __uint_as_float(0x802287abu)}; }

__device__ __forceinline__ void kw_solve_ff(wff::ff cterm, wff::ff dt_dx, float alpha, float u_prev, wff::ff& u_out,
                                            wff::ff& q_out) {
    const float QR = (float)KIN_WAVE_MIN_FLOW_QROOT;
    const float floor_c = alpha * (QR * QR * QR);
    if (!(cterm.hi > floor_c)) {
        u_out = {QR, 0.0f};
        q_out = q_floor();
        return;
    }
    const float a = dt_dx.hi, b = alpha, c = cterm.hi;
    const float ub = 1.00001f * fminf(__powf(__fdividef(c, b), 1.0f / 3.0f), __powf(__fdividef(c, a), 0.2f));
    float v = u_prev > 0.0f ? u_prev : ub;
    const float a5 = 5.0f * a, b3 = 3.0f * b;
#pragma unroll 1
    for (int it = 0; it < 12; ++it) {
        const float v2 = v * v;
        const float g = v2 * v * fmaf(a, v2, b) - c;
        const float dg = v2 * fmaf(a5, v2, b3);
        const float dv = __fdividef(g, dg);
        v = fminf(v - dv, ub);
        if (!(fabsf(dv) > 1e-4f * v)) break;
    }
    const wff::ff v2 = wff::two_prod(v, v);
    const wff::ff v3 = wff::mul(v2, v);
    const wff::ff v5 = wff::mul(v3, v2);
    const wff::ff f = wff::add(wff::add(wff::mul(dt_dx, v5), wff::mul(v3, b)), wff::neg(cterm));
    const float dv = __fdividef(f.hi, v2.hi * fmaf(a5, v2.hi, b3));
    wff::ff u = wff::two_sum(v, -dv);
    wff::ff q = wff::add(v5, wff::mul(wff::mul(v2, v2), -5.0f * dv));
    if (!(u.hi > QR)) {
        u = {QR, 0.0f};
        q = q_floor();
    }
    u_out = u;
    q_out = q;
}

}  // namespace wfk
