// tce_kernels_tc.cu -- all-s shell quartets, the node sums on the FP64 tensor
// cores, with per-quartet learned-grid rules (LG) or the system's rule.
//
// The quartet is the one k_quartets_s evaluates (ERI_shell_block_toroidal.f90
// :28-366 for s functions, scattered like direct_JK, eri_direct.f90:331-357).
// A batch of 8 MT primitive quartets pq, sorted by concentration, needs per
// periodic direction and node k of the rule
//     I[pq][k] = h sum_j F[pq][h j] T[h j][k],   F[pq][n] = G_n H_n cos(n phi_pq),
// with the stride h and last order that tce_order_plan finds for the batch and
// a pass of NT node tiles of 8 (T[n][k] = c_n e^{-C_k} I_n(C_k)): an (8 MT x J)
// x (J x 8 NT) product per pass, mma.sync.m8n8k4 (FP64) per 8 x 8 tile and step
// of four orders.  Lane l builds the A fragments (F) of rows 8 m + l/4 at order
// h (4 s + l%4), e^{i n phi} by rotation; the B fragments are T[h (4 s + l%4)][8 g + l/4].
// The G, H and T of four steps are loaded together before their mma.
//
// What bounds it: with every order summed (about 170 per node on the 64-cell
// chain) the mma instructions did; with 13 to 27 orders per tile the epilogue
// (one reciprocal per two nodes), the plans and the loads' latency weigh as
// much.  The node with the smallest C sets a pass's stride, the largest its last
// order: passes of 8 nodes need half the tile products of passes of 16 on the
// 64-cell chain, 32-node passes twice as many (tce_tc_shape_s).
// 64-cell chain: all-s 64-node list 16.4 -> 6.4 ms, 32-node list 6.5 -> 2.9 ms;
// fixed 32-node rule, whole pass 72.7 -> 14.4 ms.  (With one step's loads ahead
// and 16-node passes it was 8.2, 4.8 and 16.7 ms.)
//
// Also here: the launch of the s/p tensor-core kernel (k_quartets_sp_tc,
// tce_kernels_tc.cuh) for the classes with one p shell; those with two are
// instantiated in tce_kernels_sp2.cu.
#include "tce_kernels_tc.cuh"

// A batch is 8 MT primitive quartets, a pass NT node tiles of 8 for one set of
// orders; (MT, NT) are template parameters, chosen per work list by
// tce_lg_autotune (tce_tc_shapes_s, tce_tc_shapes_sp).
template <int NDP, int MT, int NT, bool LG>
__global__ void __launch_bounds__(256, 2) k_quartets_s_tc(DevSys S, SArgs A)
{
    constexpr int BT = 8 * MT, US = 4, RW = 3 + NDP;
    static_assert(MT <= 2, "the epilogue's shared reciprocal takes two row tiles");
    constexpr float E = tce_order_exponent(0);
    extern __shared__ double smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int rq = lane >> 2, cq = lane & 3;   // fragment row in an 8-row tile, fragment column
    const PrimPool Pool = tce_pool(smem, wib);
    // per row of the batch: pq, p + q, R^2, phi per periodic direction
    double *Rows = reinterpret_cast<double *>(reinterpret_cast<char *>(smem) + 8 * (size_t)TCE_POOL_BYTES) + (size_t)wib * BT * RW;

    while (true) {
        int it = 0;
        if (lane == 0) it = (int)atomicAdd(A.next, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= A.nitems) break;
        const int4 q = A.items[it];
        const TcRule R = tce_tc_rule<LG>(S, A, it);
        const int nq = R.nq, ng = nq / 8, nchunk = (ng + NT - 1) / NT;
        // lane c holds what pass c needs to know of its nodes: 1/C = a^2 / (2 t^2), last stored order
        float vmin[NDP], vmax[NDP];
        int glast[NDP];
        {
            float lo = __int_as_float(0x7f800000), hi = -lo;
#pragma unroll
            for (int d = 0; d < NDP; ++d) glast[d] = -1;
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const int g = lane * NT + t;
                if (g < ng) {
                    const float2 w = R.t2[g];
                    lo = fminf(lo, w.x);
                    hi = fmaxf(hi, w.y);
#pragma unroll
                    for (int d = 0; d < NDP; ++d) glast[d] = max(glast[d], R.gmax[d * TCE_MAXG + g]);
                }
            }
#pragma unroll
            for (int d = 0; d < NDP; ++d) {
                const float a2 = 0.5f * (float)(S.a[d] * S.a[d]);
                vmin[d] = a2 / hi;
                vmax[d] = a2 / lo;
                if (!(lo <= hi)) glast[d] = -1;   // padding nodes only
            }
        }
        const int cK = q.z / S.nshuc;
        const int SK0 = q.z - cK * S.nshuc;
        const int SLp = tce_shift_to(q.w, cK, S.nshuc, S.ncl);
        const UnitPair Ub = S.up[(long long)q.x * S.nsh + q.y];
        const UnitPair Uk = S.up[(long long)SK0 * S.nsh + SLp];
        double Tsh[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) Tsh[d] = S.sh_r[3 * q.z + d] - S.sh_r[3 * SK0 + d];
        const int nppb = Ub.npp, nppk = Uk.npp;
        const long long total = (long long)nppb * nppk;
        double blk = 0.0, blkG = 0.0;
        int np = 0;
        for (long long base = 0; base < total; base += 32) {
            np = tce_pool_add<true, NDP>(S, A, Ub, Uk, q, base, total, lane, Pool, np);
            if (!(np > TCE_POOL - 32 || (base + 32 >= total && np > 0))) continue;
            tce_pool_order(Pool, np, lane);
            for (int b0 = 0; b0 < np; b0 += BT) {
                // this lane's fragment rows (primitive quartets 8 m + rq of the batch; past
                // its end the first one, with factor zero)
                const double *Gp[NDP][MT], *Hp[NDP][MT];
                double c1[NDP][MT], s1[NDP][MT];
                float umin[NDP], umax[NDP], pmin[NDP], pmax[NDP];
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const int r = b0 + 8 * m + rq;
                    const int2 pq = Pool.pq[Pool.key[r < np ? r : b0]];
                    const PairPrim &Pb = S.pp[Ub.pp_off + pq.x];
                    const PairPrim &Pk = S.pp[Uk.pp_off + pq.y];
                    double *row = Rows + (8 * m + rq) * RW;
                    double R2 = 0.0;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const double x = Pb.cen[d] - (Pk.cen[d] + Tsh[d]);
                        if (d < NDP) {
                            const double phi = S.a[d] * x;
                            row[3 + (d < NDP ? d : 0)] = phi;
                            const float u = 1.0f / (float)Pb.A[d] + 1.0f / (float)Pk.A[d], ap = tce_fold_phase(phi);
                            umin[d < NDP ? d : 0] = m == 0 ? u : fminf(umin[d < NDP ? d : 0], u);
                            umax[d < NDP ? d : 0] = m == 0 ? u : fmaxf(umax[d < NDP ? d : 0], u);
                            pmin[d < NDP ? d : 0] = m == 0 ? ap : fminf(pmin[d < NDP ? d : 0], ap);
                            pmax[d < NDP ? d : 0] = m == 0 ? ap : fmaxf(pmax[d < NDP ? d : 0], ap);
                        } else {
                            R2 += x * x;
                        }
                    }
                    row[0] = Pb.esum * Pk.esum;
                    row[1] = Pb.esum + Pk.esum;
                    row[2] = R2;
#pragma unroll
                    for (int d = 0; d < NDP; ++d) {
                        Gp[d][m] = S.rvec + Ub.r_off + (long long)d * Ub.Nlen * nppb + pq.x;
                        Hp[d][m] = S.rvec + Uk.r_off + (long long)d * Uk.Nlen * nppk + pq.y;
                    }
                }
                OrderPlan plan[NDP];   // of pass `lane`; last: with the number of steps in pstep
                int pstep[NDP];
#pragma unroll
                for (int d = 0; d < NDP; ++d) {
#pragma unroll
                    for (int o = 4; o < 32; o <<= 1) {
                        umin[d] = fminf(umin[d], __shfl_xor_sync(0xffffffffu, umin[d], o));
                        umax[d] = fmaxf(umax[d], __shfl_xor_sync(0xffffffffu, umax[d], o));
                        pmin[d] = fminf(pmin[d], __shfl_xor_sync(0xffffffffu, pmin[d], o));
                        pmax[d] = fmaxf(pmax[d], __shfl_xor_sync(0xffffffffu, pmax[d], o));
                    }
                    const int nlast = min(glast[d], min(Ub.Nlen, Uk.Nlen) - 1);
                    plan[d] = tce_order_plan(E, 0, umin[d], umax[d], pmin[d], pmax[d], vmin[d], vmax[d], nlast);
                    pstep[d] = plan[d].h > 0 ? plan[d].last / (4 * plan[d].h) + 1 : 0;
                    if (glast[d] < 0) plan[d].h = 0;
                }
                __syncwarp();
                double vK[MT], vG[MT];
#pragma unroll
                for (int m = 0; m < MT; ++m) vK[m] = vG[m] = 0.0;
#pragma unroll 1
                for (int c = 0; c < nchunk; ++c) {
                    // cos, sin of h phi for four passes at a time: lane column cq computes pass c + cq's
                    if ((c & 3) == 0) {
#pragma unroll
                        for (int d = 0; d < NDP; ++d) {
                            const double hd = (double)__shfl_sync(0xffffffffu, plan[d].h, c + cq);
#pragma unroll
                            for (int m = 0; m < MT; ++m) sincos(hd * Rows[(8 * m + rq) * RW + 3 + d], &s1[d][m], &c1[d][m]);
                        }
                    }
                    double pr[2 * MT * NT];
                    bool none = false;
                    double hw = 1.0;
                    int h[NDP], last[NDP], steps[NDP];
#pragma unroll
                    for (int d = 0; d < NDP; ++d) {
                        h[d] = __shfl_sync(0xffffffffu, plan[d].h, c);
                        last[d] = __shfl_sync(0xffffffffu, plan[d].last, c);
                        steps[d] = __shfl_sync(0xffffffffu, pstep[d], c);
                        none = none || h[d] == 0;
                        hw *= (double)h[d];
                    }
                    if (none) continue;
                    int col[NT];
#pragma unroll
                    for (int t = 0; t < NT; ++t) col[t] = 8 * min(c * NT + t, ng - 1) + rq;
#pragma unroll
                    for (int d = 0; d < NDP; ++d) {
                        const double *Tg = R.T + d * R.strideD;
                        const int h4 = 4 * h[d];
                        int n = h[d] * cq;
                        double acc[2 * MT * NT];
#pragma unroll
                        for (int x = 0; x < 2 * MT * NT; ++x) acc[x] = 0.0;
                        double cc[MT], sc[MT], c4[MT], s4[MT];   // e^{i n phi}, e^{4 i h phi}
                        // US steps of loads at once: a step's mma take far less than the L2's latency
#pragma unroll 1
                        for (int s = 0; s < steps[d]; s += US) {
                            double gN[US][MT], hN[US][MT], tN[US][NT];
#pragma unroll
                            for (int u = 0; u < US; ++u) {
                                const int nn = min(n + u * h4, last[d]);
#pragma unroll
                                for (int m = 0; m < MT; ++m) {
                                    gN[u][m] = __ldg(Gp[d][m] + (long long)nn * nppb);
                                    hN[u][m] = __ldg(Hp[d][m] + (long long)nn * nppk);
                                }
#pragma unroll
                                for (int t = 0; t < NT; ++t) tN[u][t] = __ldg(Tg + ((long long)nn * nq + col[t]));
                            }
                            if (s == 0) {
#pragma unroll
                                for (int m = 0; m < MT; ++m) {
                                    const int src = (lane & ~3) | (c & 3);
                                    tce_phase_start(__shfl_sync(0xffffffffu, c1[d][m], src), __shfl_sync(0xffffffffu, s1[d][m], src),
                                                    cq, cc[m], sc[m], c4[m], s4[m]);
                                }
                            }
#pragma unroll
                            for (int u = 0; u < US; ++u) {
                                if (s + u >= steps[d]) break;
                                double F[MT];
#pragma unroll
                                for (int m = 0; m < MT; ++m) {
                                    F[m] = n <= last[d] ? gN[u][m] * hN[u][m] * cc[m] : 0.0;
                                    tce_phase_step(cc[m], sc[m], c4[m], s4[m]);
                                }
                                n += h4;
#pragma unroll
                                for (int t = 0; t < NT; ++t)
#pragma unroll
                                    for (int m = 0; m < MT; ++m) tce_dmma(acc[(m * NT + t) * 2], acc[(m * NT + t) * 2 + 1], F[m], tN[u][t]);
                            }
                        }
#pragma unroll
                        for (int x = 0; x < 2 * MT * NT; ++x) pr[x] = d == 0 ? acc[x] : pr[x] * acc[x];
                    }
                    // epilogue: pr[2 (m NT + t) + i] = prod_d I_d[8 m + rq][8 (c NT + t) + 2 cq + i] / h_d
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        if (NT > 1 && c * NT + t >= ng) continue;
                        const int k = 8 * (c * NT + t) + 2 * cq;
                        const double2 tn = *reinterpret_cast<const double2 *>(R.t + k);
                        double2 wk = *reinterpret_cast<const double2 *>(R.wk + k), wg = make_double2(0.0, 0.0);
                        if (LG) {
                            wg = *reinterpret_cast<const double2 *>(R.wg + k);
                            wg.x *= hw;
                            wg.y *= hw;
                        }
                        wk.x *= hw;
                        wk.y *= hw;
                        const double t2[2] = {tn.x * tn.x, tn.y * tn.y};
                        double D[MT][2];   // 1 / (pq + (p + q) t^2), for NDP = 2 its square root
                        if (NDP < 3) {
#pragma unroll
                            for (int m = 0; m < MT; ++m)
#pragma unroll
                                for (int i = 0; i < 2; ++i) D[m][i] = fma(Rows[(8 * m + rq) * RW + 1], t2[i], Rows[(8 * m + rq) * RW]);
                            if (NDP == 1) {   // one reciprocal for all of them
                                double q0 = D[0][0] * D[0][1], q1 = MT > 1 ? D[MT - 1][0] * D[MT - 1][1] : 1.0;
                                const double ri = 1.0 / (q0 * q1), x = q0;
                                q0 = ri * q1;
                                q1 = ri * x;
#pragma unroll
                                for (int m = 0; m < MT; ++m) {
                                    const double qm = m == 0 ? q0 : q1, y = D[m][0];
                                    D[m][0] = qm * D[m][1];
                                    D[m][1] = qm * y;
                                }
                            } else {
#pragma unroll
                                for (int m = 0; m < MT; ++m)
#pragma unroll
                                    for (int i = 0; i < 2; ++i) D[m][i] = rsqrt(D[m][i]);
                            }
                        }
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
                            double b[2] = {pr[(m * NT + t) * 2], pr[(m * NT + t) * 2 + 1]};
                            if (NDP < 3) {
                                b[0] *= D[m][0];
                                b[1] *= D[m][1];
                                const double R2 = Rows[(8 * m + rq) * RW + 2];
                                if (R2 != 0.0) {
                                    const double w = -Rows[(8 * m + rq) * RW] * R2;
#pragma unroll
                                    for (int i = 0; i < 2; ++i) b[i] *= exp(w * t2[i] * (NDP == 1 ? D[m][i] : D[m][i] * D[m][i]));
                                }
                            }
                            vK[m] = fma(b[0], wk.x, vK[m]);
                            vK[m] = fma(b[1], wk.y, vK[m]);
                            if (LG) {
                                vG[m] = fma(b[0], wg.x, vG[m]);
                                vG[m] = fma(b[1], wg.y, vG[m]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const int r = b0 + 8 * m + rq;
                    const double f = r < np ? Pool.fac[Pool.key[r]] : 0.0;
                    blk = fma(f, vK[m], blk);
                    if (LG) blkG = fma(f, vG[m], blkG);
                }
                __syncwarp();
            }
            __syncwarp();
            np = 0;
        }
        const double rc = NDP == 1 ? PI_D * PI_D : NDP == 2 ? PI_D : 1.0;   // the real directions' pi^(3 - ndp)
        blk = tce_warp_sum(blk) * rc;
        if (LG) {
            blkG = tce_warp_sum(blkG) * rc;
            if (!tce_judge_accepts(fabs(blk - blkG), fabs(blk), A.judge_tol)) {
                if (lane == 0) tce_queue_fallback(A, q);
                __syncwarp();
                continue;
            }
        }
        if (lane == 0) {
            const int fI = S.sh_first[q.x], fJ = S.sh_first[q.y], fK = S.sh_first[q.z], fL = S.sh_first[q.w];
            const int f[4] = {fI, fJ, fK, fL};
            if (S.Q[fI + (long long)S.nbas * fJ] * S.Q[fK + (long long)S.nbas * fL] >= S.thr) {
                if (!LG && A.eri)
                    tce_store_eri(S, A.eri, A.eri_size, A.physicist, f, blk);
                else
                    tce_scatter_jk(S, A.P, A.J, A.K, f, blk, fI, 1, fJ, 1, fK, 1, fL, 1);
            }
        }
        __syncwarp();
    }
}

int tce_tc_shapes_sp(int nq)
{
    return (nq == 32 || nq == 64) ? 2 : 0;
}

// one p shell.  shape 1: 8 rows x 16 nodes per pass, 2: 8 x 8
template <bool LG>
static int sp1_launch(const DevSys &S, int cls, const SArgs &A, int shape, int nsm, cudaStream_t st)
{
#define TCE_SP1(MTv, NTv)                                                              \
    switch (cls) {                                                                     \
    case 1: sp_tc_launch<1, 0, 0, 0, MTv, NTv, LG>(S, A, nsm, st); break;              \
    case 2: sp_tc_launch<0, 1, 0, 0, MTv, NTv, LG>(S, A, nsm, st); break;              \
    case 4: sp_tc_launch<0, 0, 1, 0, MTv, NTv, LG>(S, A, nsm, st); break;              \
    case 8: sp_tc_launch<0, 0, 0, 1, MTv, NTv, LG>(S, A, nsm, st); break;              \
    default: return TCE_ERR_UNSUPPORTED;                                               \
    }
    if (shape == 1) { TCE_SP1(1, 2) } else { TCE_SP1(1, 1) }
#undef TCE_SP1
    return TCE_OK;
}

int tce_launch_quartets_sp_tc(const DevSys &S, int cls, const SArgsHost &h, int nq, int shape, cudaStream_t st)
{
    const bool lg = h.item_rule != nullptr;
    if (lg && (!h.rules || !h.rule_T || !h.fb_items || !h.fb_count)) return TCE_ERR_ARG;
    if (S.ndp != 1) return TCE_ERR_UNSUPPORTED;
    if (lg && (nq != 32 && nq != 64)) return TCE_ERR_UNSUPPORTED;
    if (shape < 1 || shape > 2) return TCE_ERR_ARG;
    const int np = __builtin_popcount(cls & 15);
    if (cls < 1 || cls > 15 || np > 2) return TCE_ERR_UNSUPPORTED;
    SArgs A{};
    tc_args(A, h);
    if (cudaMemsetAsync(h.next, 0, sizeof(unsigned int), st) != cudaSuccess) return TCE_ERR_CUDA;
    const int nsm = h.num_sms > 0 ? h.num_sms : 148;
    const int s = np == 2 ? tce_sp2_launch(S, cls, A, shape, nsm, st)
                  : lg    ? sp1_launch<true>(S, cls, A, shape, nsm, st)
                          : sp1_launch<false>(S, cls, A, shape, nsm, st);
    if (s != TCE_OK) return s;
    return cudaGetLastError() == cudaSuccess ? TCE_OK : TCE_ERR_CUDA;
}

int tce_tc_shapes_s(int nq)
{
    return (nq == 32 || nq == 64) ? 4 : 0;
}

// shape 1: 16 rows x 8 nodes per pass, 2: 16 x 16, 3: 8 x 8, 4: 8 x 16
int tce_launch_quartets_s_tc(const DevSys &S, const SArgsHost &h, int nq, int shape, cudaStream_t st)
{
    const bool lg = h.item_rule != nullptr;
    if (lg && (!h.rules || !h.rule_T || !h.fb_items || !h.fb_count)) return TCE_ERR_ARG;
    if (lg && (nq != 32 && nq != 64)) return TCE_ERR_UNSUPPORTED;
    if (shape < 1 || shape > 4) return TCE_ERR_ARG;
    SArgs A{};
    tc_args(A, h);
    if (cudaMemsetAsync(h.next, 0, sizeof(unsigned int), st) != cudaSuccess) return TCE_ERR_CUDA;
    const int nsm = h.num_sms > 0 ? h.num_sms : 148;
#define TCE_S_TC(NDPv, MTv, NTv, LGv) \
    tc_launch(k_quartets_s_tc<NDPv, MTv, NTv, LGv>, S, A, nsm, st, 8 * 8 * sizeof(double) * MTv * (3 + NDPv))
    if (!lg) {
        if (S.ndp == 2) TCE_S_TC(2, 1, 2, false);
        else if (S.ndp == 3) TCE_S_TC(3, 1, 2, false);
        else if (shape == 1) TCE_S_TC(1, 2, 1, false);
        else TCE_S_TC(1, 2, 2, false);
    } else if (S.ndp == 2) {
        TCE_S_TC(2, 1, 2, true);
    } else if (S.ndp == 3) {
        TCE_S_TC(3, 1, 2, true);
    } else {
        switch (shape) {
        case 1: TCE_S_TC(1, 2, 1, true); break;
        case 2: TCE_S_TC(1, 2, 2, true); break;
        case 3: TCE_S_TC(1, 1, 1, true); break;
        default: TCE_S_TC(1, 1, 2, true); break;
        }
    }
#undef TCE_S_TC
    return cudaGetLastError() == cudaSuccess ? TCE_OK : TCE_ERR_CUDA;
}
