// tce_onee.cu -- nuclear attraction matrix on the device.
//
// NA(i, j) = -sum_atoms Z_C <i| 1/|r - C| |j> for i in the unit cell, j in
// the supercell: nuclear_attraction_integral_toroidal_{1,2,3}D
// (1D_Nuclear_attraction_toroidal.f90:26-163, 3D_Nuclear_attraction_toroidal.f90
// :18-111) with the handle's t-rule and T table, then |NA| < 1e-14 set to
// zero and the other cells' rows by translation (nuclear_attraction_matrix_
// toroidal_1D, :169-276; fill_with_symmetry, symmetric_matrix.f90:1-52).
//
// Per primitive pair the integral is
//   (2/sqrt(pi)) c1 c2 prod_periodic[e^{-2(p - pe)/a^2} L / a^M] prod_real e^{-mu R^2}
//   x sum_k w_k prod_d X_d(t_k),
// periodic d: X_d = sum_n F_n T[n][k], F_n = Re[(G_n) e^{i n phi_C}], G_n the
// pair's Fourier-Bessel vector sum_j d_j e^{-A} I_{|n+j|}(A), phi_C = a (P - C);
// real d: X_d = e^{-p eta (P - C)^2} S_1D(l1, l2, p + t^2, PA - eta PC, PB - eta PC),
// eta = t^2 / (p + t^2).
//
// One warp per function pair (i, j).  Lane 0 runs the Miller recurrence of
// e^{-A} I_n(A) (bessel_scaled_vector_fast, clifford_tools.f90:429-461) into
// shared memory; the lanes build G_n over n, then per atom F_n over n (a
// rotation by e^{32 i phi} per step of the lane's n) and finally the node
// sums over k (lanes over nodes, F broadcast from shared memory, T rows
// coalesced), reduced over the warp.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "tce_handle.h"
#include "tce_orders.cuh"

namespace {

constexpr double PI_D = 3.14159265358979323846;
constexpr int NA_WARPS_MAX = 8;
constexpr int NA_MEXTRA = 4 * TCE_LMAX + 4;   // Bessel orders past N for the Fourier product

// 1D overlap of (x + pa)^j (x + pb)^m with e^{-p x^2}, over sqrt(pi / p): the
// polynomial's even coefficients times the moments (n-1)!! / (2p)^{n/2}
// (overlap_1D_real, :336-361); inv = 1 / p
__device__ __forceinline__ double na_overlap_1d(int j, int m, double inv, double pa, double pb)
{
    if (j + m == 0) return 1.0;
    double c[2 * TCE_LMAX + 1];
    c[0] = 1.0;
#pragma unroll
    for (int x = 1; x <= 2 * TCE_LMAX; ++x) c[x] = 0.0;
    for (int f = 0; f < j + m; ++f) {
        const double r = f < j ? pa : pb;
#pragma unroll
        for (int x = 2 * TCE_LMAX; x > 0; --x) c[x] = fma(r, c[x], c[x - 1]);
        c[0] *= r;
    }
    return fma(0.75 * inv * inv, c[4], fma(0.5 * inv, c[2], c[0]));
}

struct NaArgs {
    const int2 *fsh;     // per function: shell, component
    const int2 *plist;   // (i, j) of each element, or null: every i < nfuc, j < nbas
    long long npairs;
    int natoms;
    const double *geo;   // [natoms + natoms * d] (Fortran geometry(natoms, 3))
    const int *Z;
    double *V;           // rows of the unit cell V[i + nfuc * j], or V[p] for a pair list
    int wdoubles;        // shared doubles per warp
    double zsum;         // sum of |Z|
};

__global__ void __launch_bounds__(NA_WARPS_MAX * 32) k_nuclear(DevSys S, NaArgs A)
{
    extern __shared__ double smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const long long pair = (long long)blockIdx.x * (blockDim.x >> 5) + wib;
    if (pair >= A.npairs) return;
    const int fi = A.plist ? A.plist[pair].x : (int)(pair % S.nfuc);
    const int fj = A.plist ? A.plist[pair].y : (int)(pair / S.nfuc);
    const int NW = S.ncap + 1;
    double *Iv = smem + (size_t)wib * A.wdoubles;            // NW + NA_MEXTRA
    double *Gre = Iv + NW + NA_MEXTRA;                        // [ndp][NW] each
    double *Gim = Gre + S.ndp * NW;
    double *F = Gim + S.ndp * NW;
    const int2 a1 = A.fsh[fi], a2 = A.fsh[fj];
    const int S1 = a1.x, S2 = a2.x;
    int l1[3], l2[3], M[3];
    for (int d = 0; d < 3; ++d) {
        l1[d] = S.fn_pw[3 * fi + d];
        l2[d] = S.fn_pw[3 * fj + d];
        M[d] = l1[d] + l2[d];
    }
    const double *r1 = S.sh_r + 3 * S1, *r2 = S.sh_r + 3 * S2;
    const int n1 = S.sh_np[S1], n2 = S.sh_np[S2];
    double V = 0.0;
    for (int pi = 0; pi < n1; ++pi)
        for (int pj = 0; pj < n2; ++pj) {
            const double al = S.sh_exp[S.sh_eoff[S1] + pi], be = S.sh_exp[S.sh_eoff[S2] + pj];
            const double es = al + be, mu = al * be / es;
            double pref = S.sh_coef[S.sh_coff[S1] + a1.y * n1 + pi] * S.sh_coef[S.sh_coff[S2] + a2.y * n2 + pj] * 2.0 /
                          sqrt(PI_D);
            double cen[3];
            int Np[3] = {0, 0, 0};
            for (int d = 0; d < 3; ++d) {
                if (d < S.ndp) {
                    const double a = S.a[d];
                    double pe;
                    tce_bary(al, be, r1[d], r2[d], S.L[d], a, pe, cen[d]);
                    const double Aa = 2.0 * pe / (a * a);
                    pref *= exp(-2.0 * (es - pe) / (a * a)) * S.L[d] / pow(a, (double)M[d]);
                    const int est = tce_nmax_estimate(Aa);
                    Np[d] = est < S.ncap ? est : S.ncap;
                    const int N = Np[d] + M[d];
                    if (lane == 0) {   // e^{-A} I_n(A), n = 0..N, Miller from N
                        if (Aa < 1e-10) {
                            for (int k = 0; k <= N; ++k) Iv[k] = 0.0;
                            Iv[0] = 1.0;
                        } else if (N < 2) {
                            for (int k = 0; k <= N; ++k) Iv[k] = 0.0;
                            Iv[0] = tce_iv0_scaled(Aa);
                        } else {
                            const double inv_A2 = 2.0 / Aa;
                            Iv[N] = 1e-280;
                            Iv[N - 1] = Iv[N] * (double)N * inv_A2;
                            for (int k = N - 1; k >= 1; --k) {
                                Iv[k - 1] = Iv[k + 1] + (double)k * inv_A2 * Iv[k];
                                if (Iv[k - 1] > 1e250)
                                    for (int m = k - 1; m <= N; ++m) Iv[m] *= 1e-250;
                            }
                            const double s = tce_iv0_scaled(Aa) / Iv[0];
                            for (int k = 0; k <= N; ++k) Iv[k] *= s;
                        }
                    }
                    __syncwarp();
                    double dre[4 * TCE_LMAX + 1], dim[4 * TCE_LMAX + 1];
                    if (M[d] > 0) tce_fourier_sin(l1[d], l2[d], a * (cen[d] - r1[d]), a * (cen[d] - r2[d]), dre, dim);
                    for (int n = lane; n <= Np[d]; n += 32) {
                        double gr = 0.0, gi = 0.0;
                        if (M[d] == 0) {
                            gr = Iv[n];
                        } else {
                            for (int kk = -M[d]; kk <= M[d]; ++kk) {
                                const int idx = n + kk;
                                const double b = Iv[idx < 0 ? -idx : idx];
                                gr += dre[kk + M[d]] * b;
                                gi += dim[kk + M[d]] * b;
                            }
                        }
                        Gre[d * NW + n] = gr;
                        Gim[d * NW + n] = gi;
                    }
                    __syncwarp();
                } else {
                    cen[d] = (al * r1[d] + be * r2[d]) / es;
                    pref *= exp(-mu * (r1[d] - r2[d]) * (r1[d] - r2[d]));
                }
            }
            for (int at = 0; at < A.natoms; ++at) {
                double Cc[3];
                for (int d = 0; d < 3; ++d) Cc[d] = A.geo[at + (size_t)A.natoms * d];
                for (int d = 0; d < S.ndp; ++d) {
                    const double phi = S.a[d] * (cen[d] - Cc[d]);
                    double sn, cn, s32, c32;
                    sincos((double)lane * phi, &sn, &cn);
                    sincos(32.0 * phi, &s32, &c32);
                    for (int n = lane; n <= Np[d]; n += 32) {
                        F[d * NW + n] = Gre[d * NW + n] * cn - Gim[d * NW + n] * sn;
                        const double t = cn * c32 - sn * s32;
                        sn = sn * c32 + cn * s32;
                        cn = t;
                    }
                }
                __syncwarp();
                double res = 0.0;
                for (int k = lane; k < S.nq; k += 32) {
                    const double t2 = S.tnode[k] * S.tnode[k];
                    double prod = 1.0;
                    for (int d = 0; d < 3; ++d) {
                        if (d < S.ndp) {
                            const double *Tk = S.Tt + (size_t)d * NW * S.nq + k;
                            const double *Fd = F + d * NW;
                            double d0 = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0;   // four chains
                            int n = 0;
                            for (; n + 3 <= Np[d]; n += 4) {
                                d0 = fma(Fd[n], Tk[(size_t)n * S.nq], d0);
                                d1 = fma(Fd[n + 1], Tk[(size_t)(n + 1) * S.nq], d1);
                                d2 = fma(Fd[n + 2], Tk[(size_t)(n + 2) * S.nq], d2);
                                d3 = fma(Fd[n + 3], Tk[(size_t)(n + 3) * S.nq], d3);
                            }
                            for (; n <= Np[d]; ++n) d0 = fma(Fd[n], Tk[(size_t)n * S.nq], d0);
                            prod *= (d0 + d1) + (d2 + d3);
                        } else {
                            const double ppt = es + t2, eta = t2 / ppt, pc = cen[d] - Cc[d];
                            const double ed = exp(-es * eta * pc * pc);
                            prod *= ed * sqrt(PI_D / ppt) * na_overlap_1d(l1[d], l2[d], 1.0 / ppt, (cen[d] - r1[d]) - eta * pc,
                                                                          (cen[d] - r2[d]) - eta * pc);
                        }
                    }
                    res = fma(S.tweight[k], prod, res);
                }
                res = tce_warp_sum(res);
                V -= (double)A.Z[at] * pref * res;
                __syncwarp();
            }
        }
    if (lane == 0) A.V[A.plist ? pair : fi + (long long)S.nfuc * fj] = fabs(V) < 1e-14 ? 0.0 : V;
}

// One periodic direction: a block per function pair, its warps over the
// primitive pairs.  Per primitive pair the node sums of every atom,
//     X(atom, k) = h sum_j F_{h j}(atom) T[h j][k],
// run over the orders of tce_order_plan (tce_orders.cuh: two densities here, A of
// the pair and C of the node) as (atoms x orders) x (orders x nodes) products,
// FP64 mma.sync.m8n8k4 tiles of 16 atoms x 16 nodes: lane l owns atom rows
// 8 m + l/4 and orders h (4 s + l%4), e^{i n phi_atom} by rotation; B fragments
// T[n][8 g + l/4].  Atoms whose distance makes the 16 nodes' sums negligible
// are skipped by the plan.
// What bounds it: with every order (about 250) and powers by pow() it was the
// epilogue, then the order loop, and 576 of 2304 warps had a 16-fold share.
// 1 / (p + t^2) is found once per node and primitive pair, the powers are
// multiplied out.  64-cell chain, 32 nodes: kernel 15 -> 0.48 ms, call 15.5 -> 0.66.
// A primitive pair whose prefactor times the charges is below 1e-36 is skipped:
// with powers of distances up to 1e8 it adds less than 1e-28, and elements below
// 1e-14 are set to zero.
constexpr int NA_TC_WARPS = 4;
__global__ void __launch_bounds__(NA_TC_WARPS * 32) k_nuclear_tc(DevSys S, NaArgs A)
{
    constexpr int MT = 2;
    extern __shared__ double smem[];
    __shared__ double vpart[NA_TC_WARPS];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int rq = lane >> 2, cq = lane & 3;
    const long long pair = blockIdx.x;
    const int fi = A.plist ? A.plist[pair].x : (int)(pair % S.nfuc);
    const int fj = A.plist ? A.plist[pair].y : (int)(pair / S.nfuc);
    const int NW = S.ncap + 1, nq = S.nq, nhalf = (nq + 15) / 16;
    double *Iv = smem + (size_t)wib * A.wdoubles;            // NW + NA_MEXTRA
    double2 *G = reinterpret_cast<double2 *>(Iv + ((NW + NA_MEXTRA + 1) & ~1));   // [NW]
    double2 *nd = G + NW;                                    // [nq]: 1 / (p + t^2), w pi / (p + t^2)
    const int2 a1 = A.fsh[fi], a2 = A.fsh[fj];
    const int S1 = a1.x, S2 = a2.x;
    int l1[3], l2[3];
    for (int d = 0; d < 3; ++d) {
        l1[d] = S.fn_pw[3 * fi + d];
        l2[d] = S.fn_pw[3 * fj + d];
    }
    const int M = l1[0] + l2[0];
    const bool powers = l1[1] + l2[1] + l1[2] + l2[2] > 0;
    const double *r1 = S.sh_r + 3 * S1, *r2 = S.sh_r + 3 * S2;
    const int n1 = S.sh_np[S1], n2 = S.sh_np[S2];
    const double a = S.a[0];
    const float E = tce_order_exponent(M);
    // half `lane`: 1/C range and last stored order
    float vmin, vmax;
    int glast = -1;
    {
        float lo = __int_as_float(0x7f800000), hi = -lo;
        for (int t = 0; t < 2; ++t) {
            const int g = 2 * lane + t;
            if (g < nq / 8) {
                const float2 w = S.rule_t2[g];
                lo = fminf(lo, w.x);
                hi = fmaxf(hi, w.y);
                glast = max(glast, S.rule_gmax[g]);
            }
        }
        const float h2 = 0.5f * (float)(a * a);
        vmin = h2 / hi;
        vmax = h2 / lo;
    }
    double V = 0.0;
    for (int pp = wib; pp < n1 * n2; pp += NA_TC_WARPS) {
        const int pi = pp / n2, pj = pp - pi * n2;
        const double al = S.sh_exp[S.sh_eoff[S1] + pi], be = S.sh_exp[S.sh_eoff[S2] + pj];
        const double es = al + be, mu = al * be / es;
        double pref = S.sh_coef[S.sh_coff[S1] + a1.y * n1 + pi] * S.sh_coef[S.sh_coff[S2] + a2.y * n2 + pj] * 2.0 /
                      sqrt(PI_D);
        double cen[3], pe;
        tce_bary(al, be, r1[0], r2[0], S.L[0], a, pe, cen[0]);
        const double Aa = 2.0 * pe / (a * a);
        pref *= exp(-2.0 * (es - pe) / (a * a)) * S.L[0];
        for (int i = 0; i < M; ++i) pref /= a;
        const int est = tce_nmax_estimate(Aa);
        const int Np = est < S.ncap ? est : S.ncap;
        const int N = Np + M;
        for (int d = 1; d < 3; ++d) {
            cen[d] = (al * r1[d] + be * r2[d]) / es;
            pref *= exp(-mu * (r1[d] - r2[d]) * (r1[d] - r2[d]));
        }
        if (fabs(pref) * A.zsum < 1e-36) continue;   // |P - A|, |P - C| to the fourth stay below 1e8
        __syncwarp();
        if (lane == 0) {   // e^{-A} I_n(A), n = 0..N
            if (Aa < 1e-10) {
                for (int k = 0; k <= N; ++k) Iv[k] = 0.0;
                Iv[0] = 1.0;
            } else if (N < 2) {
                for (int k = 0; k <= N; ++k) Iv[k] = 0.0;
                Iv[0] = tce_iv0_scaled(Aa);
            } else {
                const double inv_A2 = 2.0 / Aa;
                double hi = 1e-280, lo = hi * (double)N * inv_A2;
                Iv[N] = hi;
                Iv[N - 1] = lo;
                for (int k = N - 1; k >= 1; --k) {
                    const double nx = hi + (double)k * inv_A2 * lo;
                    hi = lo;
                    lo = nx;
                    Iv[k - 1] = nx;
                    if (nx > 1e250) {
                        for (int m = k - 1; m <= N; ++m) Iv[m] *= 1e-250;
                        hi *= 1e-250;
                        lo *= 1e-250;
                    }
                }
            }
        }
        __syncwarp();
        const double sc = Aa < 1e-10 || N < 2 ? 1.0 : tce_iv0_scaled(Aa) / Iv[0];
        __syncwarp();
        for (int k = lane; k <= N; k += 32) Iv[k] *= sc;
        for (int k = lane; k < nq; k += 32) {
            const double t = S.tnode[k], inv = 1.0 / fma(t, t, es);
            nd[k] = make_double2(inv, S.tweight[k] * PI_D * inv);
        }
        __syncwarp();
        if (M == 0) {
            for (int n = lane; n <= Np; n += 32) G[n] = make_double2(Iv[n], 0.0);
        } else if (Aa >= 4.0) {
            PowerSeries ps;   // the vectors sum_k d_k I_{n+k} are the ones of sign -1
            tce_power_series(l1[0], l2[0], a * (cen[0] - r1[0]), a * (cen[0] - r2[0]), ps);
            const double inv_A = 1.0 / Aa;
            for (int n = lane; n <= Np; n += 32) G[n] = tce_power_coef(ps, Iv, -n, inv_A);
        } else {
            double dre[4 * TCE_LMAX + 1], dim[4 * TCE_LMAX + 1];
            tce_fourier_sin(l1[0], l2[0], a * (cen[0] - r1[0]), a * (cen[0] - r2[0]), dre, dim);
            for (int n = lane; n <= Np; n += 32) {
                double gr = 0.0, gi = 0.0;
                for (int kk = -M; kk <= M; ++kk) {
                    const int idx = n + kk;
                    const double bv = Iv[idx < 0 ? -idx : idx];
                    gr += dre[kk + M] * bv;
                    gi += dim[kk + M] * bv;
                }
                G[n] = make_double2(gr, gi);
            }
        }
        __syncwarp();
        const float u = 1.0f / (float)Aa;
        double vsum = 0.0;
        for (int at0 = 0; at0 < A.natoms; at0 += 8 * MT) {
            double phr[MT], cy[MT], cz[MT], zc[MT];
            float pmin = 0.0f, pmax = 0.0f;
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const int at = at0 + 8 * m + rq, ar = at < A.natoms ? at : A.natoms - 1;
                zc[m] = at < A.natoms ? (double)A.Z[ar] : 0.0;
                phr[m] = a * (cen[0] - A.geo[ar]);
                cy[m] = cen[1] - A.geo[ar + (size_t)A.natoms];
                cz[m] = cen[2] - A.geo[ar + (size_t)A.natoms * 2];
                const float ap = tce_fold_phase(phr[m]);
                pmin = m == 0 ? ap : fminf(pmin, ap);
                pmax = m == 0 ? ap : fmaxf(pmax, ap);
            }
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) {
                pmin = fminf(pmin, __shfl_xor_sync(0xffffffffu, pmin, o));
                pmax = fmaxf(pmax, __shfl_xor_sync(0xffffffffu, pmax, o));
            }
            OrderPlan plan = tce_order_plan(E, M, u, u, pmin, pmax, vmin, vmax, min(glast, Np));
            if (glast < 0) plan.h = 0;
            double cs = 1.0, sn = 0.0;
#pragma unroll 1
            for (int hf = 0; hf < nhalf; ++hf) {
                if ((hf & 1) == 0)   // lane column cq: row 8 (cq / 2) + rq, half hf + cq % 2
                    sincos((double)__shfl_sync(0xffffffffu, plan.h, hf + (cq & 1)) * ((cq >> 1) ? phr[1] : phr[0]), &sn, &cs);
                const int h = __shfl_sync(0xffffffffu, plan.h, hf), last = __shfl_sync(0xffffffffu, plan.last, hf);
                if (h == 0) continue;
                const int ntile = nq / 8 - 2 * hf > 1 ? 2 : 1;
                double acc[2][MT][2];
#pragma unroll
                for (int t = 0; t < 2; ++t)
#pragma unroll
                    for (int m = 0; m < MT; ++m) acc[t][m][0] = acc[t][m][1] = 0.0;
                double cc[MT], ss[MT], c4[MT], s4[MT];
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const int src = (lane & ~3) | (2 * m + (hf & 1));
                    const double c = __shfl_sync(0xffffffffu, cs, src), s = __shfl_sync(0xffffffffu, sn, src);
                    tce_phase_start(c, s, cq, cc[m], ss[m], c4[m], s4[m]);
                }
                const double *T = S.Tt + 16 * hf + rq;
                const int t1 = ntile > 1 ? 8 : 0;
#pragma unroll 2
                for (int n0 = 0; n0 <= last; n0 += 4 * h) {
                    const int n = n0 + h * cq, nn = min(n, last);
                    double2 g = G[nn];
                    if (n > last) g = make_double2(0.0, 0.0);
                    const double T0 = __ldg(T + (size_t)nn * nq), T1 = __ldg(T + (size_t)nn * nq + t1);
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        const double F = g.x * cc[m] - g.y * ss[m];
                        tce_phase_step(cc[m], ss[m], c4[m], s4[m]);
                        tce_dmma(acc[0][m][0], acc[0][m][1], F, T0);
                        tce_dmma(acc[1][m][0], acc[1][m][1], F, T1);
                    }
                }
                // epilogue: acc[t][m][i] = X(atom 8 m + rq, node 16 hf + 8 t + 2 cq + i) / h
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    if (t >= ntile) continue;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int k = 16 * hf + 8 * t + 2 * cq + i;
                        const double2 w = nd[k];
                        const double tk = __ldg(S.tnode + k), eta = tk * tk * w.x;   // t^2 / (p + t^2)
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
                            const double R2 = cy[m] * cy[m] + cz[m] * cz[m];
                            double v = acc[t][m][i] * w.y;
                            if (R2 != 0.0) v *= exp(-es * eta * R2);
                            if (powers)
                                v *= na_overlap_1d(l1[1], l2[1], w.x, (cen[1] - r1[1]) - eta * cy[m], (cen[1] - r2[1]) - eta * cy[m]) *
                                     na_overlap_1d(l1[2], l2[2], w.x, (cen[2] - r1[2]) - eta * cz[m], (cen[2] - r2[2]) - eta * cz[m]);
                            vsum = fma(zc[m] * (double)h, v, vsum);
                        }
                    }
                }
            }
        }
        vsum = tce_warp_sum(vsum);
        V -= pref * vsum;
    }
    if (lane == 0) vpart[wib] = V;
    __syncthreads();
    if (threadIdx.x == 0) {
        V = 0.0;
        for (int w = 0; w < NA_TC_WARPS; ++w) V += vpart[w];
        A.V[A.plist ? pair : fi + (long long)S.nfuc * fj] = fabs(V) < 1e-14 ? 0.0 : V;
    }
}

}  // namespace

using namespace tcehost;

// Elements of the nuclear attraction matrix on the device: every i < nfuc,
// j < nbas (plist empty; out[i + nfuc j]) or the listed (i, j) (out[p]).
static int nuclear_elements(Handle *h, int natoms, const double *geo, const int32_t *Z, const std::vector<int2> &plist,
                            std::vector<double> &out)
{
    const int nbas = h->nbas, nfuc = h->nfuc;
    std::vector<int2> fsh((size_t)nbas, make_int2(-1, 0));
    for (int s = 0; s < (int)h->sh_first.size(); ++s)
        for (int c = 0; c < h->sh_n[s]; ++c) fsh[(size_t)h->sh_first[s] + c] = make_int2(s, c);
    for (int f = 0; f < nbas; ++f)
        if (fsh[(size_t)f].x < 0) return fail(h, TCE_ERR_STATE, "function without a shell");
    for (const int2 &p : plist)
        if (p.x < 0 || p.x >= nfuc || p.y < 0 || p.y >= nbas) return fail(h, TCE_ERR_ARG, "element outside the unit-cell rows");
    const long long npairs = plist.empty() ? (long long)nfuc * nbas : (long long)plist.size();
    std::vector<double> g(geo, geo + (size_t)natoms * 3);
    std::vector<int> z(Z, Z + natoms);
    // one buffer, one copy: out[npairs] | geometry | function table | pairs | charges
    const size_t np = (size_t)npairs, ng = g.size(), nf = fsh.size(), npl = plist.size();
    std::vector<double> in(ng + nf + npl + (z.size() + 1) / 2);
    static_assert(sizeof(int2) == sizeof(double), "tables packed as doubles");
    std::memcpy(in.data(), g.data(), sizeof(double) * ng);
    std::memcpy(in.data() + ng, fsh.data(), sizeof(int2) * nf);
    if (npl) std::memcpy(in.data() + ng + nf, plist.data(), sizeof(int2) * npl);
    std::memcpy(in.data() + ng + nf + npl, z.data(), sizeof(int) * z.size());
    double *d_V = nullptr;
    int s;
    if ((s = dalloc(h, &d_V, np + in.size()))) return s;
    double *d_geo = d_V + np;
    int2 *d_fsh = reinterpret_cast<int2 *>(d_geo + ng), *d_pl = d_fsh + nf;
    int *d_Z = reinterpret_cast<int *>(d_pl + npl);
    cudaError_t e = cudaMemcpyAsync(d_geo, in.data(), sizeof(double) * in.size(), cudaMemcpyHostToDevice, h->st);
    if (e != cudaSuccess) {
        dfree(h, d_V);
        return fail(h, TCE_ERR_CUDA, std::string("nuclear attraction: ") + cudaGetErrorString(e));
    }
    NaArgs A;
    A.fsh = d_fsh;
    A.plist = plist.empty() ? nullptr : d_pl;
    A.npairs = npairs;
    A.natoms = natoms;
    A.geo = d_geo;
    A.Z = d_Z;
    A.V = d_V;
    A.zsum = 1.0;
    for (int x : z) A.zsum += std::abs((double)x);
    const int NW = h->ncap + 1;
    // one periodic direction: the tensor-core form, where its buffers fit
    A.wdoubles = ((NW + NA_MEXTRA + 1) & ~1) + 2 * NW + 2 * h->nq;
    const size_t tbytes = (size_t)A.wdoubles * sizeof(double) * NA_TC_WARPS;
    if (h->use_tc && h->ndp == 1 && tbytes <= 200 * 1024 && npairs < 0x7fffffffLL) {
        cudaFuncSetAttribute(k_nuclear_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tbytes);
        k_nuclear_tc<<<(unsigned)npairs, 32 * NA_TC_WARPS, tbytes, h->st>>>(h->S, A);
    } else {
        A.wdoubles = (NW + NA_MEXTRA + 3 * h->ndp * NW + 31) / 32 * 32;
        const size_t wbytes = (size_t)A.wdoubles * sizeof(double);
        int warps = NA_WARPS_MAX;
        while (warps > 1 && wbytes * warps > 200 * 1024) --warps;
        if (wbytes > 200 * 1024) {
            dfree(h, d_V);
            return fail(h, TCE_ERR_UNSUPPORTED, "truncation order too large for the nuclear-attraction kernel");
        }
        const size_t smem = wbytes * (size_t)warps;
        const unsigned grid = (unsigned)((npairs + warps - 1) / warps);
        cudaFuncSetAttribute(k_nuclear, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k_nuclear<<<grid, 32 * warps, smem, h->st>>>(h->S, A);
    }
    e = cudaGetLastError();
    out.assign((size_t)npairs, 0.0);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out.data(), d_V, sizeof(double) * out.size(), cudaMemcpyDeviceToHost, h->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->st);
    dfree(h, d_V);
    if (e != cudaSuccess) return fail(h, TCE_ERR_CUDA, std::string("nuclear attraction: ") + cudaGetErrorString(e));
    return TCE_OK;
}

extern "C" int tce_nuclear_attraction(void *handle, int32_t natoms, const double *geo, const int32_t *Z, double *V)
{
    Handle *h = static_cast<Handle *>(handle);
    if (!h || !geo || !Z || !V || natoms < 1) return fail(h, TCE_ERR_ARG, "bad argument");
    const int nbas = h->nbas, nfuc = h->nfuc;
    std::vector<double> rows;
    int s = nuclear_elements(h, natoms, geo, Z, {}, rows);
    if (s) return s;
    // rows of the unit cell, the rest by translation (fill_with_symmetry)
    const int nx = h->ncl[0], ny = h->ncl[1], nz = h->ncl[2];
    for (int Rj = 0; Rj < nbas / nfuc; ++Rj)
        for (int Ri = 0; Ri < nbas / nfuc; ++Ri) {   // one cell block at a time: its source cell is the same for all of it
            const int dx = (Rj % nx - Ri % nx + nx) % nx, dy = ((Rj / nx) % ny - (Ri / nx) % ny + ny) % ny;
            const int dz = (Rj / (nx * ny) - Ri / (nx * ny) + nz) % nz;
            const double *src = rows.data() + (size_t)nfuc * nfuc * ((size_t)(dz * ny + dy) * nx + dx);
            for (int b = 0; b < nfuc; ++b)
                std::copy(src + (size_t)nfuc * b, src + (size_t)nfuc * (b + 1), V + (size_t)Ri * nfuc + (size_t)nbas * (Rj * nfuc + b));
        }
    return TCE_OK;
}

// The nuclear-attraction half of fast_quad_self_check (fast_quad_self_check.f90
// :135-172, 189): after the ERI sample (tce_quad_self_check, whose 50 random
// quartets take 200 draws of the generator next() :228-231, seed 12345), the
// diagonal V(i,i) of the first function of every unit-cell shell, 20 random
// pairs inside the unit cell and 20 with j anywhere, each with both handles'
// rules; the fast rule stays when both largest differences are <= 1e-10.
extern "C" int tce_quad_self_check_nuc(void *fast, void *full, int32_t natoms, const double *geo, const int32_t *Z,
                                       double *dmax, double *dV, int32_t *nq, int32_t *nv)
{
    Handle *hf = static_cast<Handle *>(fast), *hg = static_cast<Handle *>(full);
    if (!hf || !hg || !geo || !Z || !dmax || !dV || !nq || !nv || natoms < 1) return fail(hf, TCE_ERR_ARG, "bad argument");
    if (hf->nbas != hg->nbas || hf->nfuc != hg->nfuc) return fail(hf, TCE_ERR_ARG, "handles of different systems");
    int s = tce_quad_self_check(fast, full, dmax, nq);
    if (s) return s;
    const int nfuc = hf->nfuc, nbas = hf->nbas;
    long long seed = 12345;
    auto next = [&]() {
        seed = (seed * 1103515245LL + 12345LL) % 2147483648LL;
        return seed / 16;
    };
    for (int k = 0; k < 4 * 50; ++k) next();   // the ERI sample's draws
    std::vector<int2> pl;
    for (size_t sh = 0; sh < hf->sh_first.size(); ++sh)
        if (hf->sh_first[sh] < nfuc) pl.push_back(make_int2(hf->sh_first[sh], hf->sh_first[sh]));
    if (pl.empty()) pl.push_back(make_int2(0, 0));
    for (int r = 0; r < 40; ++r) {
        const int i = (int)(next() % nfuc);
        const int j = (int)(next() % (r < 20 ? nfuc : nbas));
        pl.push_back(make_int2(i, j));
    }
    std::vector<double> v1, v2;
    if ((s = nuclear_elements(hf, natoms, geo, Z, pl, v1))) return s;
    if ((s = nuclear_elements(hg, natoms, geo, Z, pl, v2))) return fail(hf, s, hg->err);
    double m = 0.0;
    for (size_t p = 0; p < pl.size(); ++p) m = std::max(m, std::fabs(v1[p] - v2[p]));
    *dV = m;
    *nv = (int32_t)pl.size();
    return TCE_OK;
}
