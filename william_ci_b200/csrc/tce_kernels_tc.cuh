// tce_kernels_tc.cuh -- pieces shared by the FP64 tensor-core quartet kernels:
// the primitive pool fill and its order, the rule view, the launch helpers, and the s/p kernel of one periodic direction
// k_quartets_sp_tc (one or two p shells), instantiated per class in
// tce_kernels_tc.cu (one p) and tce_kernels_sp2.cu (two p).
#pragma once
#include "tce_kernels_s.cuh"
#include "tce_orders.cuh"

// Screen the primitive quartets base + lane of a shell quartet (as
// k_quartets_s) and append the kept ones to the warp's pool: pair indices,
// factor (FOLD: with the four contraction coefficients of s shells folded in)
// and the sort key, the bits of u = sum over the periodic directions of
// 1/A_bra + 1/A_ket with the entry's index in the low seven bits (positive
// floats order like their bits).  Returns the pool's new fill.
template <bool FOLD, int NDP>
__device__ __forceinline__ int tce_pool_add(const DevSys &S, const SArgs &A, const UnitPair &Ub, const UnitPair &Uk,
                                            const int4 &q, long long base, long long total, int lane,
                                            const PrimPool &Pool, int np)
{
    const int nppk = Uk.npp;
    const long long idx = base + lane;
    bool keep = idx < total;
    int ipb = 0, ipk = 0;
    float u = 0.0f;
    double fac = 0.0;
    if (keep) {
        ipb = total <= 0x7fffffffLL ? (int)idx / nppk : (int)(idx / nppk);
        ipk = (int)(idx - (long long)ipb * nppk);
        const PairPrim &Pb = S.pp[Ub.pp_off + ipb];
        const PairPrim &Pk = S.pp[Uk.pp_off + ipk];
        fac = S.fac_const * Pb.pfac * Pk.pfac;
        const double bra = fabs(S.fac_const * Pb.pfac) * Pb.cmax12;
        if (bra * Uk.ket_max <= 2.22e-16) keep = false;
        else if (fabs(fac) * Pb.cmax12 * Pk.cmax12 <= 2.22e-16) keep = false;
        else if (A.prim_screen && Pb.ps * Pk.ps < S.prim_thr) keep = false;
        if (keep) {
            if (FOLD)
                fac *= S.sh_coef[S.sh_coff[q.x] + ipb / Ub.np2] * S.sh_coef[S.sh_coff[q.y] + ipb % Ub.np2] *
                       S.sh_coef[S.sh_coff[q.z] + ipk / Uk.np2] * S.sh_coef[S.sh_coff[q.w] + ipk % Uk.np2];
#pragma unroll
            for (int d = 0; d < NDP; ++d) u += 1.0f / (float)Pb.A[d] + 1.0f / (float)Pk.A[d];
        }
    }
    const unsigned msk = __ballot_sync(0xffffffffu, keep);
    const int at = np + __popc(msk & ((1u << lane) - 1u));
    if (keep) {
        Pool.pq[at] = make_int2(ipb, ipk);
        Pool.fac[at] = fac;
        Pool.key[at] = (int)((__float_as_uint(u) & ~127u) | (unsigned)at);
    }
    __syncwarp();
    return np + __popc(msk);
}

// Sort the keys of pool entries [0, n), n <= 32 R, ascending in registers
// (bitonic over lane + 32 r) and write the entries' indices in that order to
// Pool.key.  Rows of about the same concentration end up in one tile, so that
// they need about the same orders (tce_orders.cuh).
template <int R>
__device__ __forceinline__ void tce_pool_order_r(const PrimPool &P, int n, int lane)
{
    unsigned k[R];
#pragma unroll
    for (int r = 0; r < R; ++r) k[r] = lane + 32 * r < n ? (unsigned)P.key[lane + 32 * r] : 0xffffffffu;
#pragma unroll
    for (int s = 2; s <= 32 * R; s <<= 1)
#pragma unroll
        for (int j = s >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int x = r ^ (j >> 5);
                    if (x > r) {
                        const bool up = ((32 * r) & s) == 0;
                        const unsigned lo = min(k[r], k[x]), hi = max(k[r], k[x]);
                        k[r] = up ? lo : hi;
                        k[x] = up ? hi : lo;
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const unsigned o = __shfl_xor_sync(0xffffffffu, k[r], j);
                    const bool up = ((lane + 32 * r) & s) == 0, lower = (lane & j) == 0;
                    k[r] = up == lower ? min(k[r], o) : max(k[r], o);
                }
            }
        }
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (lane + 32 * r < n) P.key[lane + 32 * r] = (int)(k[r] & 127u);
    __syncwarp();
}
__device__ __forceinline__ void tce_pool_order(const PrimPool &P, int n, int lane)
{
    __syncwarp();
    if (n <= 32) tce_pool_order_r<1>(P, n, lane);
    else if (n <= 64) tce_pool_order_r<2>(P, n, lane);
    else tce_pool_order_r<4>(P, n, lane);
}

// The quadrature rule of a shell quartet for the tensor-core kernels: learned
// grid (LG) a dictionary rule with its judge weights, else the system's rule.
struct TcRule {
    const double *T;      // direction d at T + d * strideD, row n at + n * nq
    long long strideD;
    const double *t, *wk, *wg;
    const int *gmax;
    const float2 *t2;     // per 8-node group: smallest and largest t^2
    int nq;
};
template <bool LG>
__device__ __forceinline__ TcRule tce_tc_rule(const DevSys &S, const SArgs &A, int it)
{
    TcRule R;
    if (LG) {
        const RuleDev *D = A.rules + A.item_rule[it];
        R.nq = D->nq;
        R.T = A.rule_T + D->T_off;
        R.t = A.rule_t + D->node_off;
        R.wk = A.rule_wk + D->node_off;
        R.wg = A.rule_wg + D->node_off;
        R.gmax = D->gmax;
        R.t2 = D->t2;
    } else {
        R.nq = S.nq;
        R.T = S.Tt;
        R.t = S.tnode;
        R.wk = S.tweight;
        R.wg = nullptr;
        R.gmax = S.rule_gmax;
        R.t2 = S.rule_t2;
    }
    R.strideD = (long long)(S.ncap + 1) * R.nq;
    return R;
}

static inline void tc_args(SArgs &A, const SArgsHost &h)
{
    A.items = h.items;
    A.nitems = h.nitems;
    A.prim_screen = h.prim_screen;
    A.next = h.next;
    A.P = h.P;
    A.J = h.J;
    A.K = h.K;
    A.eri = h.eri;
    A.eri_size = h.eri_size;
    A.physicist = h.physicist;
    A.item_rule = h.item_rule;
    A.rules = h.rules;
    A.rule_T = h.rule_T;
    A.rule_t = h.rule_t;
    A.rule_wk = h.rule_wk;
    A.rule_wg = h.rule_wg;
    A.judge_tol = h.judge_tol;
    A.fb_items = h.fb_items;
    A.fb_count = h.fb_count;
}

// persistent launch: as many 256-thread blocks as fit on every SM; shared
// memory = the eight warps' pools and `extra` bytes
template <class Kern>
static void tc_launch(Kern kern, const DevSys &S, const SArgs &A, int nsm, cudaStream_t st, size_t extra)
{
    const size_t smem = 8 * (size_t)TCE_POOL_BYTES + extra;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, 256, smem);
    if (per < 1) per = 1;
    kern<<<nsm * per, 256, smem, st>>>(S, A);
}

// ============================================================================
// s/p classes with one or two p shells, one periodic direction
// (compile-time class LA, LB | LC, LD in {0, 1}), learned-grid or system rule: the quartet of
// ERI_shell_block_toroidal.f90:28-366 for these classes, scattered like
// direct_JK (eri_direct.f90:331-357), with the node sums on the tensor cores.
//
// Power combinations.  The periodic direction has one row per x-power
// combination (ia, ib | ic, id) of the p shells (2^NP of them):
//     I_cmb[pq][k] = sum_n Re[G^(ia,ib)_n H^(ic,id)_n e^{i n phi}] T[n][k],
// all of them in the same step loop over the orders of tce_order_plan: the
// zero-power vectors G^(0,0), H^(0,0) are real and loaded once for every
// combination, and e^{i n phi} advances by one rotation per step of four strides.  The A fragments are F = Re(G H) cos(n phi) - Im(G H) sin(n phi)
// with the products of real factors left out.
//
// Epilogue by moments.  The real directions add, per node k and component c
// (x powers = combination cmb), w_k I_cmb I_y I_z with the McMurchie-Davidson
// sums of ERI_shell_block_toroidal.f90:302-335:
//     I_d = sum_{u,v} (-1)^u E_u E'_v g_d[u + v],
//     g_d[m] = pi sqrt(D2) e^{-w R_d^2} h_m(w),  D2 = 1 / (pq + (p + q) t_k^2),
//     w = pq t_k^2 D2,  h_0 = 1,  h_{m+1} = 2 w R_d h_m - 2 m w h_{m-1}.
// So I_y I_z = pi^2 D2 e^{-w R^2} P_c(w) (R^2 = R_y^2 + R_z^2), P_c a
// polynomial in w of degree <= the component's y and z powers whose
// coefficients depend on the primitive quartet only.  Each lane sums, over its
// nodes, the moments
//     M_cmb,j = sum_k I_cmb[pq][k] D2 e^{-w R^2} w^j   (Kronrod and Gauss weights)
// and each component follows once per row: pi^2 a^-xs sum_j P_c[j] M_cmb,j.
//
// A batch is 8 MT primitive quartets (rows, sorted by concentration), a pass
// NT node tiles of 8 with the orders and stride of tce_order_plan; per pass and
// step of four orders a warp issues 2^NP MT NT mma.sync.m8n8k4.  The moments of
// a row are kept over the passes of a batch, the components follow once.
// ============================================================================
template <int LA, int LB, int LC, int LD, int MT, int NT, bool LG>
__global__ void __launch_bounds__(256, LA + LB + LC + LD == 1 ? 2 : 1) k_quartets_sp_tc(DevSys S, SArgs A)
{
    constexpr int NP = LA + LB + LC + LD;
    static_assert(NP >= 1 && NP <= 2, "one or two p shells");
    constexpr int BT = 8 * MT;
    constexpr float E = tce_order_exponent(NP);
    constexpr int SHIFT = LA + LB > LC + LD ? LA + LB : LC + LD;
    constexpr int NA = LA == 0 ? 1 : 3, NB = LB == 0 ? 1 : 3, NC = LC == 0 ? 1 : 3, ND = LD == 0 ? 1 : 3;
    constexpr int NCQ = NA * NB * NC * ND;
    constexpr int NCOMB = (LA + 1) * (LB + 1) * (LC + 1) * (LD + 1);
    constexpr int NGV = (LA + 1) * (LB + 1), NHV = (LC + 1) * (LD + 1);
    constexpr int NN = NP;                                // largest y + z power of a component
    constexpr int EB = tce_ecount(LA, LB), EK = tce_ecount(LC, LD);
    constexpr int AT = 2 * MT * NT;                       // accumulators per combination and lane
    constexpr int US = NP == 1 ? 3 : 2;                   // steps loaded together
    constexpr int NW = LG ? 2 : 1;                        // Kronrod sums, and Gauss sums with the judge
    extern __shared__ double smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int rq = lane >> 2, cq = lane & 3;   // fragment row in an 8-row tile, fragment column
    const PrimPool Pool = tce_pool(smem, wib);
    // per-lane Kronrod / Gauss block accumulators of the components (shared
    // memory, after the eight pools): [c][lane] and [NCQ + c][lane]
    double *bacc = reinterpret_cast<double *>(reinterpret_cast<char *>(smem) + 8 * (size_t)TCE_POOL_BYTES) +
                   (size_t)wib * 2 * NCQ * 32;
    const double PI2 = PI_D * PI_D, ainv = 1.0 / S.a[0];
    // x-power sum of a combination
    auto xsum = [](int cmb) {
        return cmb % (LA + 1) + (cmb / (LA + 1)) % (LB + 1) + (cmb / NGV) % (LC + 1) + cmb / (NGV * (LC + 1));
    };

    while (true) {
        int it = 0;
        if (lane == 0) it = (int)atomicAdd(A.next, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= A.nitems) break;
        const int4 q = A.items[it];
        const TcRule R = tce_tc_rule<LG>(S, A, it);
        const int nq = R.nq, ng = nq / 8, nchunk = (ng + NT - 1) / NT;
        // lane c holds what pass c needs to know of its nodes: 1/C = a^2 / (2 t^2), last stored order
        float vmin, vmax;
        int glast = -1;
        {
            float lo = __int_as_float(0x7f800000), hi = -lo;
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const int g = lane * NT + t;
                if (g < ng) {
                    const float2 w = R.t2[g];
                    lo = fminf(lo, w.x);
                    hi = fmaxf(hi, w.y);
                    glast = max(glast, R.gmax[g]);
                }
            }
            const float a2 = 0.5f * (float)(S.a[0] * S.a[0]);
            vmin = a2 / hi;
            vmax = a2 / lo;
            if (!(lo <= hi)) glast = -1;   // padding nodes only
        }
        const int cK = q.z / S.nshuc;
        const int SK0 = q.z - cK * S.nshuc;
        const int SLp = tce_shift_to(q.w, cK, S.nshuc, S.ncl);
        const UnitPair Ub = S.up[(long long)q.x * S.nsh + q.y];
        const UnitPair Uk = S.up[(long long)SK0 * S.nsh + SLp];
        const double Tx = S.sh_r[3 * q.z] - S.sh_r[3 * SK0];
        const int nppb = Ub.npp, nppk = Uk.npp;
        const int npA = S.sh_np[q.x], npB = S.sh_np[q.y], npC = S.sh_np[q.z], npD = S.sh_np[q.w];
        const long long total = (long long)nppb * nppk;
        // power vectors of the periodic direction: combination g = ia + (LA + 1) ib
        // of the bra is the slab ia (LB + 1) + ib, at Gv + 2 slab gl; the ket alike
        const long long gl = (long long)Ub.Nlen * nppb, hl = (long long)Uk.Nlen * nppk;
        const double2 *Gv = S.vec + Ub.vec_off, *Hv = S.vec + Uk.vec_off + hl;
        const double *G0 = S.rvec + Ub.r_off, *H0 = S.rvec + Uk.r_off;   // the zero powers, real
#pragma unroll
        for (int c = 0; c < NW * NCQ; ++c) bacc[c * 32 + lane] = 0.0;
        int np = 0;
        for (long long base = 0; base < total; base += 32) {
            np = tce_pool_add<false, 1>(S, A, Ub, Uk, q, base, total, lane, Pool, np);
            if (!(np > TCE_POOL - 32 || (base + 32 >= total && np > 0))) continue;
            tce_pool_order(Pool, np, lane);
            for (int b0 = 0; b0 < np; b0 += BT) {
                // this lane's fragment rows (past the batch's end its first one, not used)
                int go[MT], ho[MT];
                double phi[MT], pq_[MT], ps[MT], R2[MT], c1[MT], s1[MT];
                float umin = 0.0f, umax = 0.0f, pmin = 0.0f, pmax = 0.0f;
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const int r = b0 + 8 * m + rq;
                    const int2 pq = Pool.pq[Pool.key[r < np ? r : b0]];
                    const PairPrim &Pb = S.pp[Ub.pp_off + pq.x];
                    const PairPrim &Pk = S.pp[Uk.pp_off + pq.y];
                    go[m] = pq.x;
                    ho[m] = pq.y;
                    phi[m] = S.a[0] * (Pb.cen[0] - (Pk.cen[0] + Tx));
                    pq_[m] = Pb.esum * Pk.esum;
                    ps[m] = Pb.esum + Pk.esum;
                    const double Ry = Pb.cen[1] - Pk.cen[1], Rz = Pb.cen[2] - Pk.cen[2];
                    R2[m] = Ry * Ry + Rz * Rz;
                    const float u = 1.0f / (float)Pb.A[0] + 1.0f / (float)Pk.A[0], ap = tce_fold_phase(phi[m]);
                    umin = m == 0 ? u : fminf(umin, u);
                    umax = m == 0 ? u : fmaxf(umax, u);
                    pmin = m == 0 ? ap : fminf(pmin, ap);
                    pmax = m == 0 ? ap : fmaxf(pmax, ap);
                }
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    umin = fminf(umin, __shfl_xor_sync(0xffffffffu, umin, o));
                    umax = fmaxf(umax, __shfl_xor_sync(0xffffffffu, umax, o));
                    pmin = fminf(pmin, __shfl_xor_sync(0xffffffffu, pmin, o));
                    pmax = fmaxf(pmax, __shfl_xor_sync(0xffffffffu, pmax, o));
                }
                OrderPlan plan = tce_order_plan(E, SHIFT, umin, umax, pmin, pmax, vmin, vmax,
                                                min(glast, min(Ub.Nlen, Uk.Nlen) - 1));   // of pass `lane`
                const int pstep = plan.h > 0 ? plan.last / (4 * plan.h) + 1 : 0;
                if (glast < 0) plan.h = 0;
                // moments [m][cmb][j][Kronrod, Gauss], j <= NN - xsum(cmb)
                double Mo[MT][NCOMB][NN + 1][NW];
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int cmb = 0; cmb < NCOMB; ++cmb)
#pragma unroll
                        for (int j = 0; j <= NN; ++j)
#pragma unroll
                            for (int w = 0; w < NW; ++w) Mo[m][cmb][j][w] = 0.0;
#pragma unroll 1
                for (int c = 0; c < nchunk; ++c) {
                    // cos, sin of h phi for four passes at a time: lane column cq computes pass c + cq's
                    if ((c & 3) == 0) {
                        const double hd = (double)__shfl_sync(0xffffffffu, plan.h, c + cq);
#pragma unroll
                        for (int m = 0; m < MT; ++m) sincos(hd * phi[m], &s1[m], &c1[m]);
                    }
                    const int h = __shfl_sync(0xffffffffu, plan.h, c), last = __shfl_sync(0xffffffffu, plan.last, c);
                    if (h == 0) continue;
                    int col[NT];
#pragma unroll
                    for (int t = 0; t < NT; ++t) col[t] = 8 * min(c * NT + t, ng - 1) + rq;
                    double acc[NCOMB][AT];
#pragma unroll
                    for (int cmb = 0; cmb < NCOMB; ++cmb)
#pragma unroll
                        for (int x = 0; x < AT; ++x) acc[cmb][x] = 0.0;
                    double cc[MT], sc[MT], c4[MT], s4[MT];   // e^{i n phi}, e^{4 i h phi}
                    const int steps = __shfl_sync(0xffffffffu, pstep, c), h4 = 4 * h;
                    int n = h * cq;
                    // US steps of loads at once: a step's mma take far less than the L2's latency
#pragma unroll 1
                    for (int s = 0; s < steps; s += US) {
                        double g0N[US][MT], h0N[US][MT], tN[US][NT];
                        double2 gN[US][NGV - 1 > 0 ? NGV - 1 : 1][MT], hN[US][NHV - 1 > 0 ? NHV - 1 : 1][MT];
#pragma unroll
                        for (int u = 0; u < US; ++u) {
                            const int nn = min(n + u * h4, last);
#pragma unroll
                            for (int m = 0; m < MT; ++m) {
                                const double2 *gp = Gv + ((long long)nn * nppb + go[m]), *hp = Hv + ((long long)nn * nppk + ho[m]);
                                g0N[u][m] = __ldg(G0 + ((long long)nn * nppb + go[m]));
                                h0N[u][m] = __ldg(H0 + ((long long)nn * nppk + ho[m]));
#pragma unroll
                                for (int g = 1; g < NGV; ++g) gN[u][g - 1][m] = __ldg(gp + 2 * (g % (LA + 1) * (LB + 1) + g / (LA + 1)) * gl);
#pragma unroll
                                for (int x = 1; x < NHV; ++x) hN[u][x - 1][m] = __ldg(hp + 2 * (x % (LC + 1) * (LD + 1) + x / (LC + 1)) * hl);
                            }
#pragma unroll
                            for (int t = 0; t < NT; ++t) tN[u][t] = __ldg(R.T + ((long long)nn * nq + col[t]));
                        }
                        if (s == 0) {
#pragma unroll
                            for (int m = 0; m < MT; ++m) {
                                const int src = (lane & ~3) | (c & 3);
                                tce_phase_start(__shfl_sync(0xffffffffu, c1[m], src), __shfl_sync(0xffffffffu, s1[m], src), cq, cc[m],
                                                sc[m], c4[m], s4[m]);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < US; ++u) {
                            if (s + u >= steps) break;
                            double F[NCOMB][MT];
#pragma unroll
                            for (int m = 0; m < MT; ++m) {
                                const bool in = n <= last;
#pragma unroll
                                for (int cmb = 0; cmb < NCOMB; ++cmb) {
                                    const int gi = cmb % NGV, hi = cmb / NGV;
                                    double v;
                                    if (gi == 0 && hi == 0) {
                                        v = g0N[u][m] * h0N[u][m] * cc[m];
                                    } else if (gi == 0) {
                                        const double2 hv = hN[u][hi > 0 ? hi - 1 : 0][m];
                                        v = g0N[u][m] * (hv.x * cc[m] - hv.y * sc[m]);
                                    } else if (hi == 0) {
                                        const double2 gv = gN[u][gi > 0 ? gi - 1 : 0][m];
                                        v = h0N[u][m] * (gv.x * cc[m] - gv.y * sc[m]);
                                    } else {
                                        const double2 gv = gN[u][gi - 1][m], hv = hN[u][hi - 1][m];
                                        const double ar = gv.x * hv.x - gv.y * hv.y, ai = gv.x * hv.y + gv.y * hv.x;
                                        v = ar * cc[m] - ai * sc[m];
                                    }
                                    F[cmb][m] = in ? v : 0.0;
                                }
                                tce_phase_step(cc[m], sc[m], c4[m], s4[m]);
                            }
                            n += h4;
#pragma unroll
                            for (int t = 0; t < NT; ++t)
#pragma unroll
                                for (int m = 0; m < MT; ++m)
#pragma unroll
                                    for (int cmb = 0; cmb < NCOMB; ++cmb) {
                                        const int x = (m * NT + t) * 2;
                                        tce_dmma(acc[cmb][x], acc[cmb][x + 1], F[cmb][m], tN[u][t]);
                                    }
                        }
                    }
                    // epilogue: acc[cmb][2 (m NT + t) + i] = I_cmb[8 m + rq][8 (c NT + t) + 2 cq + i] / h
                    const double hw = (double)h;
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        if (NT > 1 && c * NT + t >= ng) continue;
                        const int k = 8 * (c * NT + t) + 2 * cq;
                        const double2 tn = *reinterpret_cast<const double2 *>(R.t + k);
                        const double2 wk = *reinterpret_cast<const double2 *>(R.wk + k);
                        double2 wg = make_double2(0.0, 0.0);
                        if (LG) wg = *reinterpret_cast<const double2 *>(R.wg + k);
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
                            const double t20 = tn.x * tn.x, t21 = tn.y * tn.y;
                            const double d0 = fma(ps[m], t20, pq_[m]), d1 = fma(ps[m], t21, pq_[m]);
                            const double ri = 1.0 / (d0 * d1);
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const double D2 = i == 0 ? ri * d1 : ri * d0;
                                const double w = pq_[m] * (i == 0 ? t20 : t21) * D2;
                                double bse = D2 * hw;
                                if (R2[m] != 0.0) bse *= exp(-w * R2[m]);
                                double wj[NN + 1][NW];   // weight x D2 e^{-w R^2} w^j
                                wj[0][0] = bse * (i == 0 ? wk.x : wk.y);
                                if (LG) wj[0][NW - 1] = bse * (i == 0 ? wg.x : wg.y);
#pragma unroll
                                for (int j = 1; j <= NN; ++j)
#pragma unroll
                                    for (int v = 0; v < NW; ++v) wj[j][v] = wj[j - 1][v] * w;
#pragma unroll
                                for (int cmb = 0; cmb < NCOMB; ++cmb) {
                                    const double b = acc[cmb][(m * NT + t) * 2 + i];
#pragma unroll
                                    for (int j = 0; j <= NN - xsum(cmb); ++j)
#pragma unroll
                                        for (int v = 0; v < NW; ++v) Mo[m][cmb][j][v] = fma(b, wj[j][v], Mo[m][cmb][j][v]);
                                }
                            }
                        }
                    }
                }
                // the components of this lane's rows from their moments
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const int r = b0 + 8 * m + rq;
                    if (r >= np) continue;
                    const int e = Pool.key[r];
                    const int2 pq = Pool.pq[e];
                    const PairPrim &Pb = S.pp[Ub.pp_off + pq.x];
                    const PairPrim &Pk = S.pp[Uk.pp_off + pq.y];
                    const double Ry = Pb.cen[1] - Pk.cen[1], Rz = Pb.cen[2] - Pk.cen[2];
                    // Hermite E coefficients of the real directions y (dr = 0), z (dr = 1)
                    double eb[2][EB], ek[2][EK];
                    const double *Ebp = S.ecoef + Ub.e_off + (long long)pq.x * 2 * (LA + 1) * (LB + 1) * TCE_ECO;
                    const double *Ekp = S.ecoef + Uk.e_off + (long long)pq.y * 2 * (LC + 1) * (LD + 1) * TCE_ECO;
#pragma unroll
                    for (int dr = 0; dr < 2; ++dr) {
#pragma unroll
                        for (int a = 0; a <= LA; ++a)
#pragma unroll
                            for (int b = 0; b <= LB; ++b)
#pragma unroll
                                for (int u = 0; u <= a + b; ++u)
                                    eb[dr][tce_eoff(LB, a, b) + u] = Ebp[((dr * (LA + 1) + a) * (LB + 1) + b) * TCE_ECO + u];
#pragma unroll
                        for (int a = 0; a <= LC; ++a)
#pragma unroll
                            for (int b = 0; b <= LD; ++b)
#pragma unroll
                                for (int u = 0; u <= a + b; ++u)
                                    ek[dr][tce_eoff(LD, a, b) + u] = Ekp[((dr * (LC + 1) + a) * (LD + 1) + b) * TCE_ECO + u];
                    }
                    // coefficients in w of h_m(w) per real direction: hc[dr][m][j]
                    double hc[2][NN + 1][NN + 1];
#pragma unroll
                    for (int dr = 0; dr < 2; ++dr) {
                        const double Rr = dr == 0 ? Ry : Rz;
#pragma unroll
                        for (int mm = 0; mm <= NN; ++mm)
#pragma unroll
                            for (int j = 0; j <= NN; ++j) hc[dr][mm][j] = (mm == 0 && j == 0) ? 1.0 : 0.0;
#pragma unroll
                        for (int mm = 0; mm < NN; ++mm)
#pragma unroll
                            for (int j = 1; j <= NN; ++j)
                                hc[dr][mm + 1][j] = 2.0 * Rr * hc[dr][mm][j - 1] - (mm > 0 ? 2.0 * mm * hc[dr][mm - 1][j - 1] : 0.0);
                    }
                    const double fac = Pool.fac[e] * PI2;
                    const int i0 = pq.x / Ub.np2, j0 = pq.x - i0 * Ub.np2;
                    const int k0 = pq.y / Uk.np2, l0 = pq.y - k0 * Uk.np2;
#pragma unroll
                    for (int c = 0; c < NCQ; ++c) {
                        const int ca = c % NA, cb = (c / NA) % NB, cc_ = (c / (NA * NB)) % NC, cd = c / (NA * NB * NC);
                        const int cmb = tce_pw(LA, ca, 0) + (LA + 1) * (tce_pw(LB, cb, 0) + (LB + 1) * (tce_pw(LC, cc_, 0) + (LC + 1) * tce_pw(LD, cd, 0)));
                        const int xs = xsum(cmb);
                        // P_d(w) = sum_{u,v} (-1)^u E_u E'_v h_{u+v}(w) per real direction
                        double Pd[2][NN + 1];
#pragma unroll
                        for (int dr = 0; dr < 2; ++dr) {
                            const int pa = tce_pw(LA, ca, dr + 1), pb = tce_pw(LB, cb, dr + 1);
                            const int pc = tce_pw(LC, cc_, dr + 1), pd = tce_pw(LD, cd, dr + 1);
#pragma unroll
                            for (int j = 0; j <= NN; ++j) Pd[dr][j] = 0.0;
#pragma unroll
                            for (int u = 0; u <= pa + pb; ++u)
#pragma unroll
                                for (int v = 0; v <= pc + pd; ++v) {
                                    const double e1 = eb[dr][tce_eoff(LB, pa, pb) + u];
                                    const double ee = ((u & 1) ? -e1 : e1) * ek[dr][tce_eoff(LD, pc, pd) + v];
#pragma unroll
                                    for (int j = 0; j <= u + v; ++j) Pd[dr][j] = fma(ee, hc[dr][u + v][j], Pd[dr][j]);
                                }
                        }
                        double vs[NW];
#pragma unroll
                        for (int v = 0; v < NW; ++v) vs[v] = 0.0;
#pragma unroll
                        for (int j = 0; j <= NN - xs; ++j) {
                            double cj = 0.0;
#pragma unroll
                            for (int j1 = 0; j1 <= j; ++j1) cj = fma(Pd[0][j1], Pd[1][j - j1], cj);
#pragma unroll
                            for (int v = 0; v < NW; ++v) vs[v] = fma(cj, Mo[m][cmb][j][v], vs[v]);
                        }
                        const double sg = xs == 0 ? 1.0 : xs == 1 ? ainv : ainv * ainv;
                        const double cf = S.sh_coef[S.sh_coff[q.x] + ca * npA + i0] * S.sh_coef[S.sh_coff[q.y] + cb * npB + j0] *
                                          S.sh_coef[S.sh_coff[q.z] + cc_ * npC + k0] * S.sh_coef[S.sh_coff[q.w] + cd * npD + l0];
                        const double f = fac * cf * sg;
#pragma unroll
                        for (int v = 0; v < NW; ++v)
                            bacc[(v * NCQ + c) * 32 + lane] = fma(f, vs[v], bacc[(v * NCQ + c) * 32 + lane]);
                    }
                }
            }
            __syncwarp();
            np = 0;
        }
        const int fI = S.sh_first[q.x], fJ = S.sh_first[q.y], fK = S.sh_first[q.z], fL = S.sh_first[q.w];
        double e = 0.0, M = 0.0;
        double blk[NCQ];
#pragma unroll
        for (int c = 0; c < NCQ; ++c) {
            blk[c] = tce_warp_sum(bacc[c * 32 + lane]);
            if (LG) {
                const double vg = tce_warp_sum(bacc[(NCQ + c) * 32 + lane]);
                e = fmax(e, fabs(blk[c] - vg));
                M = fmax(M, fabs(blk[c]));
            }
        }
        if (LG && !tce_judge_accepts(e, M, A.judge_tol)) {
            if (lane == 0) tce_queue_fallback(A, q);
            __syncwarp();
            continue;
        }
#pragma unroll
        for (int c = 0; c < NCQ; ++c) {
            const double v = blk[c];
            if (lane == (c & 31)) {
                const int ca = c % NA, cb = (c / NA) % NB, cc_ = (c / (NA * NB)) % NC, cd = c / (NA * NB * NC);
                const int f[4] = {fI + ca, fJ + cb, fK + cc_, fL + cd};
                if (S.Q[f[0] + (long long)S.nbas * f[1]] * S.Q[f[2] + (long long)S.nbas * f[3]] < S.thr) continue;
                if (!LG && A.eri)
                    tce_store_eri(S, A.eri, A.eri_size, A.physicist, f, v);
                else
                    tce_scatter_jk(S, A.P, A.J, A.K, f, v, fI, NA, fJ, NB, fK, NC, fL, ND);
            }
        }
        __syncwarp();
    }
}

// one class of the s/p kernel in tile shape (MT, NT): ncq components
template <int LA, int LB, int LC, int LD, int MT, int NT, bool LG>
static void sp_tc_launch(const DevSys &S, const SArgs &A, int nsm, cudaStream_t st)
{
    constexpr int ncq = (LA ? 3 : 1) * (LB ? 3 : 1) * (LC ? 3 : 1) * (LD ? 3 : 1);
    tc_launch(k_quartets_sp_tc<LA, LB, LC, LD, MT, NT, LG>, S, A, nsm, st, 8 * 2 * (size_t)ncq * 32 * sizeof(double));
}

// the classes with two p shells (tce_kernels_sp2.cu), as sp1_launch in tce_kernels_tc.cu
int tce_sp2_launch(const DevSys &S, int cls, const SArgs &A, int shape, int nsm, cudaStream_t st);
