// tce_orders.cuh -- which Bessel orders the node sums of a periodic direction
// need, and with what stride.
//
// For a primitive quartet and a node t the sum is, over all integers n,
//     I(phi) = sum_n V^bra_n V^ket_n e^{-C} I_n(C) e^{i n phi},  C = 2 t^2 / a^2,
// the Fourier series of a function on the circle: the convolution of three von
// Mises densities of concentrations A_bra, A_ket and C (times polynomials in
// sin, cos for p and d functions), evaluated at phi.  Its width is that of one
// density of concentration
//     A_c = 1 / (1/A_bra + 1/A_ket + 1/C).
// Two facts bound the work:
//  * decay in n: with f(n, A) = n asinh(n/A) + A - sqrt(n^2 + A^2) each factor
//    falls like e^{-f(n, A)} (I_n(A)/I_0(A) <= e^{-f}), f(n, 1/u) is concave in
//    u and zero at u = 0, so the three add up to at least f(n, A_c): orders with
//    f(n, A_c) > E are below e^{-E} of the sum of the terms' magnitudes;
//  * decay on the circle: at the distance x the function is below
//    e^{-A_c (1 - cos x)} of its peak.  A sum over the multiples of h only,
//    times h, adds the function's values at phi + 2 pi m / h (m = 1..h-1): they
//    are below e^{-E} of the peak when 2 pi / h >= |phi| + x_E,
//    A_c (1 - cos x_E) = E.  Where |phi| itself is past x_E, the sum is below
//    e^{-E} of the peak and is not evaluated.
// So about E (1 + |phi| / x_E) / pi orders do, at most 2 E / pi, instead of the
// 20 + 9 sqrt(min(A_bra, A_ket)) orders of the reference's truncation
// (clifford_tools.f90:566-572): about 13 to 27 instead of 170 on the 64-cell
// chain.  With E = 40 the error is 4e-18 of the peak, below the rounding of
// the sum over every order (the terms cancel from the peak's size).  A p or
// d function's vector is smaller than the s one by A^{-1/2} per power and
// grows by at most (n / A) per power, so E grows by 2.5 > ln(9) per power; at
// small A its orders are shifted by the power, hence `shift`.
#pragma once
#include "tce_device.cuh"

__host__ __device__ constexpr float tce_order_exponent(int powers) { return 40.0f + 2.5f * (float)powers; }

struct OrderPlan {
    int h;      // stride; 0: every sum is negligible
    int last;   // largest order
};

// The stride and last order that serve every row (u = 1/A_bra + 1/A_ket in
// [umin, umax], |phi| in [pmin, pmax] within [0, pi]) and every node
// (v = 1/C in [vmin, vmax]); nlast: the last order with a stored term.
__device__ __forceinline__ OrderPlan tce_order_plan(float E, int shift, float umin, float umax, float pmin, float pmax,
                                                    float vmin, float vmax, int nlast)
{
    OrderPlan p;
    const float qw = E * (umax + vmax);          // E / (smallest A_c)
    const float sp = sinf(0.5f * pmin);
    p.h = 1;
    if (2.0f * sp * sp >= qw) {
        p.h = 0;
    } else if (qw < 2.0f) {
        const float x = 2.0f * asinf(sqrtf(0.5f * qw));
        const int h = (int)(6.2831f / (pmax + x));
        p.h = h > 1 ? h : 1;
    }
    const float un = umin + vmin;                // 1 / (largest A_c)
    if (un < 1e9f) {
        // A_c x asinh(x) + ... = E by Newton's method from the Gaussian estimate,
        // which lies below the root of a convex function: every step stays above it
        const float q = E * un;
        float x = sqrtf(2.0f * q);
#pragma unroll
        for (int it = 0; it < 2; ++it) {
            const float w = sqrtf(1.0f + x * x), as = logf(x + w);
            const float g = x * as - x * x / (1.0f + w);
            x += fmaxf((q - g) / as, -0.5f * x);
        }
        const float n = 1.001f * x / un + 2.0f;
        if (n < (float)nlast) p.last = min(nlast, (int)n + shift);
        else p.last = nlast;
    } else {
        p.last = min(nlast, 4 + shift);
    }
    return p;
}

// |phi| reduced to [0, pi]
__device__ __forceinline__ float tce_fold_phase(double phi)
{
    const double t = phi * 0.15915494309189535;   // 1 / (2 pi)
    return fabsf((float)(t - rint(t))) * 6.2831853f;
}

// e^{i q phi} (q = 0..3: a lane's first order) and e^{4 i phi} (the rotation per
// step of four orders) from (c, s) = e^{i phi}, phi the stride's phase; cosines of
// doubled angles by 1 - 2 sin^2
__device__ __forceinline__ void tce_phase_start(double c, double s, int q, double &cc, double &sc, double &c4, double &s4)
{
    const double c2 = fma(-2.0 * s, s, 1.0), s2 = 2.0 * s * c;
    cc = q == 0 ? 1.0 : q == 1 ? c : q == 2 ? c2 : fma(c2, c, -s2 * s);
    sc = q == 0 ? 0.0 : q == 1 ? s : q == 2 ? s2 : fma(s2, c, c2 * s);
    c4 = fma(-2.0 * s2, s2, 1.0);
    s4 = 2.0 * s2 * c2;
}

// the next step: one rounding per step, so errors grow linearly with the few steps taken
__device__ __forceinline__ void tce_phase_step(double &cc, double &sc, double c4, double s4)
{
    const double t = cc;
    cc = fma(t, c4, -sc * s4);
    sc = fma(sc, c4, t * s4);
}
