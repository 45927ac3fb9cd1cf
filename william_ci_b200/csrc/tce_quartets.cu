// tce_quartets.cu -- the generic quartet kernel (sm_100a): every class up to
// d shells, one warp per shell quartet.  ERI_shell_block_toroidal
// (ERI_shell_block_toroidal.f90:28-366) evaluated with a t-quadrature rule
// given as a RuleView (nodes, weights, optional judge weights, the table
// c_n e^{-C_k} I_n(C_k) of the nodes), so the same code serves
//   * the reference rule (32/40-node mapped Gauss-Legendre or a 64/128 table),
//   * the learned grid: a per-quartet mapped Gauss-Kronrod rule picked by the
//     network; the embedded Gauss weights give a second estimate, and the
//     quartet is accepted when the error estimate of its block (block_judge)
//     is <= tol, otherwise it is queued for
//   * the plain method: adaptive bisection of u in [0,1] with a 15-point
//     Kronrod / 7-point Gauss pair per panel, the Bessel columns of each
//     panel's nodes computed on the fly (Miller recurrence as setup_t_tables,
//     clifford_tools.f90:620-709, or Debye-seeded downward recurrence).
// Consumers of a block: Schwarz / parity blocks, the primitive Schwarz table,
// the J/K scatter (direct_JK, eri_direct.f90:331-357) and the stored-ERI
// scatter (ERI_toroidal.f90:416-454).
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#include "tce_device.cuh"
#include "tce_kernels.h"
#include "tce_orders.cuh"

#define PI_D 3.14159265358979323846
#define PLAIN_PMAX 24

struct RuleView {
    const double *T;          // direction d at T + d * strideD, row n at + n * NQ
    long long strideD;
    const double *t, *wk, *wg;   // nodes, weights, judge weights (nullptr: no judge)
    const int *gmax;          // gmax[d * TCE_MAXG + g]: last n with a nonzero entry in node group g
    const float2 *t2;         // per node group: smallest and largest t^2
};

template <bool RO>
__device__ __forceinline__ double ldT(const double *p)
{
    if (RO) return __ldg(p);
    return *p;
}

// One row I_r(t_k) = sgn sum_n F_n T[n][k] of the nodes of one chunk: the
// 8-node groups g0 .. g0 + 3 (32 nodes, fewer at the end of the rule), out[x]
// for node 8 g0 + x.
template <int NQ, bool RO>
__device__ __forceinline__ void row_dot(const RuleView &R, int d, const double2 *__restrict__ G, int nppb, int ib_,
                                        const double2 *__restrict__ H, int nppk, int ik_, int nm, double phi,
                                        double sgn, int g0, double *out)
{
    constexpr int NG = NQ / 8;
    const double *T = R.T + (size_t)d * R.strideD;
    const int *gm = R.gmax + d * TCE_MAXG;
    double c1, s1;
    sincos(phi, &s1, &c1);
    double acc[32];
#pragma unroll
    for (int x = 0; x < 32; ++x) acc[x] = 0.0;
    double cn = 1.0, sn = 0.0;
    int n = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        if (g0 + s >= NG) break;
        int nend = gm[g0 + s];
        nend = nend < nm ? nend : nm;
        for (; n <= nend; ++n) {
            if (n > 0) {
                if ((n & 31) == 0) {
                    sincos((double)n * phi, &sn, &cn);
                } else {
                    double tmp = cn * c1 - sn * s1;
                    sn = sn * c1 + cn * s1;
                    cn = tmp;
                }
            }
            double2 g = __ldg(G + (size_t)n * nppb + ib_);
            double2 h = __ldg(H + (size_t)n * nppk + ik_);
            double ar = g.x * h.x - g.y * h.y, ai = g.x * h.y + g.y * h.x;
            double F = ar * cn - ai * sn;
            const double *Tn = T + (size_t)n * NQ + 8 * g0;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                if (g >= s && g0 + g < NG) {
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)
                        acc[8 * g + kk] = fma(F, ldT<RO>(Tn + 8 * g + kk), acc[8 * g + kk]);
                }
            }
        }
    }
#pragma unroll
    for (int x = 0; x < 32; ++x)
        if (8 * g0 + x < NQ) out[x] = acc[x] * sgn;
}

struct QCtx {
    int SI, SJ, SK, SL, nA, nB, nC, nD, lsA, lsB, lsC, lsD, ncomb, ncq, NN, R;
    int cqp;   // lanes of one primitive quartet in the component contraction: power of two >= ncq, at most 32
    UnitPair Ub, Uk;
    double Tsh[3];
    RuleView R_;             // the quadrature rule of the evaluation at hand
};

// Row numbering of a batch of nb primitive quartets: row d nb ncomb + p ncomb +
// cmb is direction d, primitive quartet p, power combination cmb; tiles of 16
// rows of one direction.
//
// Per-warp shared memory (WarpBuf), sized for the launch's largest class by
// tce_warp_doubles: rows of a chunk of 32 nodes at stride RS = 34 doubles (even,
// so that two nodes load as one double2, and 16 bytes past a multiple of 128,
// so that eight rows fall into different banks; 18 for the plain method's
// 16-node panels).  The every-order form (process_batch_every) has lanes on rows
// and no use for most of it: stride 33 (17), and a whole warp's 32 rows where the
// tensor cores take 16 per direction.
constexpr int TCE_NC = 32;        // nodes of a chunk
constexpr int TCE_GT_ROWS = 12;   // rows of g_m(t) of the real directions: (NN + 1) x primitive quartets at once
struct RowMeta {
    long long g, h;      // first elements of the bra and ket vectors, from the unit pairs' slabs
    double phi;
    float u, ap;         // 1/A_bra + 1/A_ket, |phi| in [0, pi]
};
struct WarpBuf {
    int2 *qlist;                 // primitive pairs
    short4 *qidx;                // primitive of each of the four shells
    double *qfac, *rows, *realb, *gt, *blkK, *blkG, *cf, *wts, *pqm, *extra;
    RowMeta *meta;
    int2 *plan;                  // [tile][half]: stride and last order of a tile's 16-node half
    double2 *cs;                 // [row][half]: cos and sin of h phi
    unsigned *cmap;              // per component: power combination of x, y, z (8 bits each)
    unsigned char *dig;          // per power combination: ia, ib, ic, id (2 bits each)
};

struct WarpLayout {              // offsets in doubles
    int qlist, qidx, qfac, rows, realb, gt, blkK, blkG, cf, wts, pqm, meta, plan, cs, cmap, dig, extra;
};
__host__ __device__ inline WarpLayout tce_warp_layout(bool tc, int rowcap, int RS, int nreal, int cstride, int blkcap, int nhalf)
{
    WarpLayout o;
    int at = ((int)(sizeof(QCtx) + 7) / 8 + 1) & ~1;   // the quartet at hand
    auto take = [&](int n) { const int r = at; at += (n + 1) & ~1; return r; };
    o.qlist = take(rowcap);
    o.qidx = take(tc ? rowcap : 0);
    o.qfac = take(rowcap);
    o.rows = take(rowcap * RS);
    o.realb = take(nreal * cstride * RS);
    o.gt = take(tc ? nreal * TCE_GT_ROWS * RS : 0);
    o.blkK = take(blkcap);
    o.blkG = take(blkcap);
    o.cf = take(tc ? 72 : 0);
    o.wts = take(tc ? 64 : 0);
    o.pqm = take(tc && nreal > 0 ? 4 * rowcap : 0);
    o.meta = take(tc ? rowcap * (int)(sizeof(RowMeta) / 8) : 0);
    o.plan = take(tc ? (rowcap / 16 + 3) * nhalf : 0);
    o.cs = take(tc ? 2 * rowcap * nhalf : 0);
    o.cmap = take(tc ? (blkcap + 1) / 2 : 0);
    o.dig = take(tc ? 12 : 0);
    o.extra = at;
    return o;
}

struct QuartetArgs {
    const int4 *items;
    const int *prim_sel;
    int nitems;
    const unsigned int *nitems_dev;   // when set, the item count is read on the device
    int mode, method;
    int prim_screen;
    unsigned int *next;
    double *blk_out, *blk_out2;
    const long long *blk_off;
    const double *P;
    double *J, *K;
    double *eri;
    int eri_size, physicist;
    PairPrim *pp_rw;
    int rowcap, cstride, blkcap, warp_smem_doubles;
    WarpLayout lay;
    const int *fixed_gmax;
    // learned grid
    const RuleDev *rules;
    const double *rule_T, *rule_t, *rule_wk, *rule_wg;
    const int *item_rule;
    int rule_override;
    double judge_tol;
    int4 *fb_items;
    int *fb_index;
    unsigned int *fb_count;
    // plain
    double *scratch;
    long long scratch_per_warp, T_doubles;
    double plain_tol, plain_scale;
    int plain_max_panels;
    const double *gk_u, *gk_wk, *gk_wg;
    unsigned long long *node_evals;
};

// Shared memory of a block: [DevSys][WarpLayout][warp buffers]; a warp buffer
// starts with the quartet at hand (QCtx).  The device functions below get a
// warp buffer's offset and read all of it from shared memory: what is uniform
// over the warp stays out of the registers, and every access is known to be a
// shared-memory one.
constexpr int TCE_SYS_DOUBLES = ((int)(sizeof(DevSys) + 7) / 8 + 1) & ~1;
constexpr int TCE_HDR_DOUBLES = TCE_SYS_DOUBLES + (((int)(sizeof(WarpLayout) + 7) / 8 + 1) & ~1);
extern __shared__ __align__(16) double smem[];

__device__ __forceinline__ const DevSys &blk_sys() { return *reinterpret_cast<const DevSys *>(smem); }
__device__ __forceinline__ QCtx &warp_ctx(int wofs) { return *reinterpret_cast<QCtx *>(smem + wofs); }
__device__ __forceinline__ WarpBuf warp_buf(int wofs)
{
    const WarpLayout &o = *reinterpret_cast<const WarpLayout *>(smem + TCE_SYS_DOUBLES);
    double *ws = smem + wofs;
    WarpBuf b;
    b.qlist = reinterpret_cast<int2 *>(ws + o.qlist);
    b.qidx = reinterpret_cast<short4 *>(ws + o.qidx);
    b.qfac = ws + o.qfac;
    b.rows = ws + o.rows;
    b.realb = ws + o.realb;
    b.gt = ws + o.gt;
    b.blkK = ws + o.blkK;
    b.blkG = ws + o.blkG;
    b.cf = ws + o.cf;
    b.wts = ws + o.wts;
    b.pqm = ws + o.pqm;
    b.meta = reinterpret_cast<RowMeta *>(ws + o.meta);
    b.plan = reinterpret_cast<int2 *>(ws + o.plan);
    b.cs = reinterpret_cast<double2 *>(ws + o.cs);
    b.cmap = reinterpret_cast<unsigned *>(ws + o.cmap);
    b.dig = reinterpret_cast<unsigned char *>(ws + o.dig);
    b.extra = ws + o.extra;
    return b;
}
// header of the block's shared memory, by all threads
__device__ __forceinline__ void blk_header(const DevSys &S, const WarpLayout &lay)
{
    if (threadIdx.x == 0) *reinterpret_cast<DevSys *>(smem) = S;
    if (threadIdx.x == blockDim.x - 1) *reinterpret_cast<WarpLayout *>(smem + TCE_SYS_DOUBLES) = lay;
    __syncthreads();
}

__device__ __forceinline__ double tce_ipow(double x, int k)
{
    double r = 1.0;
    for (int i = 0; i < k; ++i) r *= x;
    return r;
}

// What the rows of a batch need, once per batch: vector offsets and phase of
// every row (RowMeta), and for every tile of 16 rows and every 16-node half of
// the rule the stride and last order (tce_order_plan): lane = half + nhalf x
// tile.  Kept out of the node chunks: index divisions, the PairPrim loads and
// the plans cost more than a tile's mma instructions.
template <int NQ>
__device__ __noinline__ void row_setup(int wofs, int nb, int lane)
{
    const DevSys &S = blk_sys();
    const QCtx &Q = warp_ctx(wofs);
    const RuleView &Rv = Q.R_;
    const WarpBuf b = warp_buf(wofs);
    constexpr int NH = NQ / 16 + (NQ % 16 ? 1 : 0);
    const int ndp = S.ndp, nd = Q.ncomb, per = nb * nd;
    const int nppb = Q.Ub.npp, nppk = Q.Uk.npp;
    for (int r = lane; r < per * ndp; r += 32) {
        const int d = r / per, rr = r - d * per, p = rr / nd;
        const int dg = b.dig[rr - p * nd];
        const int ia = dg & 3, ib = (dg >> 2) & 3, ic = (dg >> 4) & 3, id = dg >> 6;
        const int2 pq = b.qlist[p];
        const PairPrim &Pb = S.pp[Q.Ub.pp_off + pq.x];
        const PairPrim &Pk = S.pp[Q.Uk.pp_off + pq.y];
        RowMeta m;
        m.g = ((((long long)d * (Q.lsA + 1) + ia) * (Q.lsB + 1) + ib) * 2 + 0) * Q.Ub.Nlen * nppb + pq.x;
        m.h = ((((long long)d * (Q.lsC + 1) + ic) * (Q.lsD + 1) + id) * 2 + 1) * Q.Uk.Nlen * nppk + pq.y;
        m.phi = S.a[d] * (Pb.cen[d] - (Pk.cen[d] + Q.Tsh[d]));
        m.u = 1.0f / (float)Pb.A[d] + 1.0f / (float)Pk.A[d];
        m.ap = tce_fold_phase(m.phi);
        b.meta[r] = m;
    }
    __syncwarp();
    const int tiles = (per + 15) / 16, shift = max(Q.lsA + Q.lsB, Q.lsC + Q.lsD);
    const float E = tce_order_exponent(Q.NN);
    for (int x = lane; x < tiles * ndp * NH; x += 32) {
        const int tile = x / NH, half = x - tile * NH, d = tile / tiles, r0 = d * per + (tile - d * tiles) * 16;
        const int r1 = min(r0 + 16, (d + 1) * per);
        float umin = b.meta[r0].u, umax = umin, pmin = b.meta[r0].ap, pmax = pmin;
        for (int r = r0 + 1; r < r1; ++r) {
            const float u = b.meta[r].u, ap = b.meta[r].ap;
            umin = fminf(umin, u);
            umax = fmaxf(umax, u);
            pmin = fminf(pmin, ap);
            pmax = fmaxf(pmax, ap);
        }
        float lo = __int_as_float(0x7f800000), hi = -lo;
        int glast = -1;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int g = 2 * half + t;
            if (g < NQ / 8) {
                const float2 w = Rv.t2[g];
                lo = fminf(lo, w.x);
                hi = fmaxf(hi, w.y);
                glast = max(glast, Rv.gmax[d * TCE_MAXG + g]);
            }
        }
        const float a2 = 0.5f * (float)(S.a[d] * S.a[d]);
        OrderPlan plan;
        plan.h = 0;
        plan.last = 0;
        if (lo <= hi && glast >= 0)   // the half has real nodes
            plan = tce_order_plan(E, shift, umin, umax, pmin, pmax, a2 / hi, a2 / lo, min(glast, min(Q.Ub.Nlen, Q.Uk.Nlen) - 1));
        b.plan[x] = make_int2(plan.h, plan.last);
    }
    __syncwarp();
    for (int x = lane; x < per * ndp * NH; x += 32) {
        const int r = x / NH, half = x - r * NH, d = r / per;
        const int h = b.plan[(d * tiles + (r - d * per) / 16) * NH + half].x;
        double2 v;
        sincos((double)h * b.meta[r].phi, &v.y, &v.x);
        b.cs[x] = v;
    }
    __syncwarp();
}

// The rows of one chunk of 32 nodes on the FP64 tensor cores: per tile of 16
// rows the A operand F = Re[G_n H_n e^{i n phi}], the rule's T table of the
// direction the B operand; mma.sync.m8n8k4 per 8 x 8 tile and step of four
// orders.  Lane l builds the A fragments of rows 8 m + l/4 (m = 0, 1) at order
// h (4 s + l%4), e^{i n phi} by rotation, and loads the next step's G, H and T
// before the current step's mma.  Halves of the same stride run in one loop, so that
// they share the A fragments.  rows[r * RS + x] = a^-powers I_r(t_{8 g0c + x}).
// Rows of one primitive quartet are next to each other, so a tile's rows share
// phase and concentration.
template <int NQ, bool RO, int RS>
__device__ __noinline__ void tc_rows(int wofs, int nb, int lane, int g0c)
{
    const DevSys &S = blk_sys();
    const QCtx &Q = warp_ctx(wofs);
    const RuleView &Rv = Q.R_;
    const WarpBuf b = warp_buf(wofs);
    constexpr int MT = 2, NTC = (NQ < TCE_NC ? NQ : TCE_NC) / 8;
    constexpr int NH = NQ / 16 + (NQ % 16 ? 1 : 0);
    const int ng = NQ / 8 - g0c < NTC ? NQ / 8 - g0c : NTC;   // groups of this chunk
    const int rq = lane >> 2, cq = lane & 3;
    const int nd = Q.ncomb, per = nb * nd, tiles = (per + 15) / 16;
    const int nppb = Q.Ub.npp, nppk = Q.Uk.npp;
    const double2 *Gv = S.vec + Q.Ub.vec_off, *Hv = S.vec + Q.Uk.vec_off;
#pragma unroll 1
    for (int tile = 0; tile < tiles * S.ndp; ++tile) {
        const int d = tile / tiles, r0 = d * per + (tile - d * tiles) * 16, rend = (d + 1) * per;
        const double *T = Rv.T + (size_t)d * Rv.strideD + 8 * g0c + rq;
        const int2 pl0 = b.plan[tile * NH + g0c / 2];
        const int2 pl1 = NTC > 2 && g0c / 2 + 1 < NH ? b.plan[tile * NH + g0c / 2 + 1] : make_int2(0, 0);
        const int h0 = pl0.x, l0 = pl0.y, h1 = pl1.x, l1 = pl1.y;
        const double2 *gp[MT], *hp[MT], *cs[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const int r = min(r0 + 8 * m + rq, rend - 1);   // past the end: the last row again
            gp[m] = Gv + b.meta[r].g;
            hp[m] = Hv + b.meta[r].h;
            cs[m] = b.cs + (r * NH + g0c / 2);
        }
        double acc[NTC][MT][2];
#pragma unroll
        for (int t = 0; t < NTC; ++t)
#pragma unroll
            for (int m = 0; m < MT; ++m) acc[t][m][0] = acc[t][m][1] = 0.0;
        // node tiles [T0, T1) of the chunk over the orders 0, h, .., last
        auto run = [&](auto t0c, auto t1c, int half, int h, int last) {
            constexpr int T0 = decltype(t0c)::value, T1 = decltype(t1c)::value;
            const int h4 = 4 * h;
            int n = h * cq;
            double2 gN[MT], hN[MT];
            double tN[T1 - T0];
            auto load = [&]() {   // the values of order n (past the last order: F = 0)
                const int nn = min(n, last);
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    gN[m] = __ldg(gp[m] + (long long)nn * nppb);
                    hN[m] = __ldg(hp[m] + (long long)nn * nppk);
                }
#pragma unroll
                for (int t = T0; t < T1; ++t) tN[t - T0] = ldT<RO>(T + ((long long)nn * NQ + 8 * (t < ng ? t : 0)));
            };
            load();
            // e^{i n phi} at n = h cq and the rotation by 4 h phi per step (errors add up
            // linearly, one rounding per step, and few steps are taken: no re-seeding)
            double cc[MT], sc[MT], c4[MT], s4[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const double2 z = cs[m][half];
                tce_phase_start(z.x, z.y, cq, cc[m], sc[m], c4[m], s4[m]);
            }
#pragma unroll 1
            for (int n0 = 0; n0 <= last; n0 += h4) {
                double F[MT], Tb[T1 - T0];
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const double ar = gN[m].x * hN[m].x - gN[m].y * hN[m].y, ai = gN[m].x * hN[m].y + gN[m].y * hN[m].x;
                    F[m] = n <= last ? ar * cc[m] - ai * sc[m] : 0.0;
                }
#pragma unroll
                for (int t = 0; t < T1 - T0; ++t) Tb[t] = tN[t];
                n += h4;
                load();
#pragma unroll
                for (int m = 0; m < MT; ++m) tce_phase_step(cc[m], sc[m], c4[m], s4[m]);
#pragma unroll
                for (int t = T0; t < T1; ++t)
#pragma unroll
                    for (int m = 0; m < MT; ++m) tce_dmma(acc[t][m][0], acc[t][m][1], F[m], Tb[t - T0]);
            }
        };
        using I0 = std::integral_constant<int, 0>;
        using I2 = std::integral_constant<int, 2>;
        using IN = std::integral_constant<int, NTC>;
        if constexpr (NTC > 2) {
            if (h0 != 0 && h0 == h1) {
                run(I0{}, IN{}, 0, h0, max(l0, l1));
            } else {
                if (h0 != 0) run(I0{}, I2{}, 0, h0, l0);
                if (h1 != 0) run(I2{}, IN{}, 1, h1, l1);
            }
        } else {
            if (h0 != 0) run(I0{}, IN{}, 0, h0, l0);
        }
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const int r = r0 + 8 * m + rq;
            if (r >= rend) continue;
#pragma unroll
            for (int t = 0; t < NTC; ++t) {
                if (t >= ng) continue;
                const double w = (double)(t < 2 ? h0 : h1);
                *reinterpret_cast<double2 *>(b.rows + (size_t)r * RS + 8 * t + 2 * cq) =
                    make_double2(acc[t][m][0] * w, acc[t][m][1] * w);
            }
        }
    }
}

// A batch of nb primitive quartets: the rows of a chunk of 32 nodes, then the
// chunk's share of every component's node sum (the row buffer holds 32 nodes
// instead of NQ: more warps per SM).  With at most 32 components lane l
// accumulates component l % cqp into accK (and accG) for the primitive quartets
// l / cqp + PW j; otherwise the lanes run over the components of one primitive
// quartet after the other and accumulate into blkK (and blkG).
template <int NQ, bool RO>
__device__ __noinline__ void process_batch(int wofs, int nb, int lane, int cstride, double &accK_, double &accG_)
{
    const DevSys &S = blk_sys();
    const QCtx &Q = warp_ctx(wofs);
    const RuleView &Rv = Q.R_;
    const WarpBuf b = warp_buf(wofs);
    constexpr int NC = NQ < TCE_NC ? NQ : TCE_NC;
    constexpr int RS = NC + 2;
    const int ndp = S.ndp, nreal = 3 - ndp;
    const int ncomb = Q.ncomb, per = nb * ncomb, NN = Q.NN;
    const bool judge = Rv.wg != nullptr;
    const bool few = Q.ncq <= 32;
    const int nAB = Q.nA * Q.nB, nCD = Q.nC * Q.nD;
    int PW = 1, pl = 0, cl = lane;                   // primitive quartets at once; this lane's, its component
    if (few) {
        PW = 32 / Q.cqp;
        pl = lane / Q.cqp;
        cl = lane - pl * Q.cqp;
    }
    // primitive quartets whose real-direction tables are built together
    const int RP = nreal > 0 ? max(1, min(cstride / ncomb, TCE_GT_ROWS / (NN + 1))) : nb;
    const double *coA = S.sh_coef + S.sh_coff[Q.SI], *coB = S.sh_coef + S.sh_coff[Q.SJ];
    const double *coC = S.sh_coef + S.sh_coff[Q.SK], *coD = S.sh_coef + S.sh_coff[Q.SL];
    const int npA = S.sh_np[Q.SI], npB = S.sh_np[Q.SJ], npC = S.sh_np[Q.SK], npD = S.sh_np[Q.SL];
    // 1/a per power of the periodic directions (the rows leave it out), by function
    auto apow = [&](int shell, int comp) {
        const int *pw = S.fn_pw + 3 * (S.sh_first[shell] + comp);
        double f = 1.0;
        for (int d = 0; d < ndp; ++d) f *= tce_ipow(1.0 / S.a[d], pw[d]);
        return f;
    };
    unsigned cm0 = 0;
    double f0 = 1.0;
    if (few && cl < Q.ncq) {                         // this lane's component
        const int ca = cl % Q.nA, r1 = cl / Q.nA, cb = r1 % Q.nB, r2 = r1 / Q.nB, cc = r2 % Q.nC, cd = r2 / Q.nC;
        coA += ca * npA;
        coB += cb * npB;
        coC += cc * npC;
        coD += cd * npD;
        cm0 = b.cmap[cl];
        f0 = apow(Q.SI, ca) * apow(Q.SJ, cb) * apow(Q.SK, cc) * apow(Q.SL, cd);
    }
    double accK = 0.0, accG = 0.0;
    if (nreal > 0)   // exponents and real distances of every primitive quartet of the batch
        for (int p = lane; p < nb; p += 32) {
            const int2 pq = b.qlist[p];
            const PairPrim &Pb = S.pp[Q.Ub.pp_off + pq.x];
            const PairPrim &Pk = S.pp[Q.Uk.pp_off + pq.y];
            b.pqm[4 * p] = Pb.esum * Pk.esum;
            b.pqm[4 * p + 1] = Pb.esum + Pk.esum;
            for (int dr = 0; dr < nreal; ++dr) b.pqm[4 * p + 2 + dr] = Pb.cen[ndp + dr] - (Pk.cen[ndp + dr] + Q.Tsh[ndp + dr]);
        }
    row_setup<NQ>(wofs, nb, lane);
#pragma unroll 1
    for (int k0 = 0; k0 < NQ; k0 += NC) {
        const int g0c = k0 / 8, kn = NQ - k0 < NC ? NQ - k0 : NC;
        tc_rows<NQ, RO, RS>(wofs, nb, lane, g0c);
        for (int k = lane; k < 2 * kn; k += 32) {   // the chunk's weights: Kronrod, then Gauss
            const int kk = k < kn ? k : k - kn;
            b.wts[(k < kn ? 0 : 32) + kk] = k < kn ? Rv.wk[k0 + kk] : (judge ? Rv.wg[k0 + kk] : 0.0);
        }
        __syncwarp();
#pragma unroll 1
        for (int q0 = 0; q0 < nb; q0 += RP) {
            const int qn = nb - q0 < RP ? nb - q0 : RP;
            if (nreal > 0) {
                // g_m(t) of the real directions, then every combination's
                // sum_{u,v} (-1)^u E_u E'_v g_{u+v}: the products of E by order first
                for (int x = lane; x < qn * kn; x += 32) {
                    const int pi = x / kn, k = x - pi * kn;
                    const double *pm = b.pqm + 4 * (q0 + pi);
                    const double t = Rv.t[k0 + k], t2 = t * t;
                    const double rr = rsqrt(fma(pm[1], t2, pm[0])), D2 = rr * rr;
                    const double w2 = 2.0 * (pm[0] * t2 * D2), rs = PI_D * rr;
                    for (int dr = 0; dr < nreal; ++dr) {
                        const double Rr = pm[2 + dr], wR = w2 * Rr;
                        double *g = b.gt + (size_t)(dr * TCE_GT_ROWS + pi * (NN + 1)) * RS + k;
                        double gm1 = 0.0, g0 = (Rr == 0.0) ? rs : rs * exp(-0.5 * wR * Rr);
                        g[0] = g0;
                        for (int n = 0; n < NN; ++n) {
                            const double gp1 = wR * g0 - (double)n * w2 * gm1;
                            g += RS;
                            g[0] = gp1;
                            gm1 = g0;
                            g0 = gp1;
                        }
                    }
                }
                __syncwarp();
                const int nrow = qn * ncomb * nreal;
                const int sp = nrow <= 8 ? 4 : nrow <= 16 ? 2 : 1, kp = ((kn >> 1) + sp - 1) / sp;   // lanes per row, node pairs each
                for (int xs = lane; xs < nrow * sp; xs += 32) {
                    const int part = xs / nrow, x = xs - part * nrow;
                    const int dr = x / (qn * ncomb), y = x - dr * qn * ncomb, pi = y / ncomb, cmb = y - pi * ncomb;
                    const int dg = b.dig[cmb];
                    const int ia = dg & 3, ib = (dg >> 2) & 3, ic = (dg >> 4) & 3, id = dg >> 6;
                    const int2 pq = b.qlist[q0 + pi];
                    const double *eb = S.ecoef + Q.Ub.e_off + ((((long long)pq.x * nreal + dr) * (Q.lsA + 1) + ia) * (Q.lsB + 1) + ib) * TCE_ECO;
                    const double *ek = S.ecoef + Q.Uk.e_off + ((((long long)pq.y * nreal + dr) * (Q.lsC + 1) + ic) * (Q.lsD + 1) + id) * TCE_ECO;
                    double sm[2 * TCE_ECO - 1];
#pragma unroll
                    for (int m = 0; m < 2 * TCE_ECO - 1; ++m) sm[m] = 0.0;
#pragma unroll
                    for (int u = 0; u < TCE_ECO; ++u) {
                        if (u > ia + ib) continue;
                        const double e = (u & 1) ? -eb[u] : eb[u];
#pragma unroll
                        for (int v = 0; v < TCE_ECO; ++v)
                            if (v <= ic + id) sm[u + v] = fma(e, ek[v], sm[u + v]);
                    }
                    const int mm = ia + ib + ic + id;
                    const double2 *g = reinterpret_cast<const double2 *>(b.gt + (size_t)(dr * TCE_GT_ROWS + pi * (NN + 1)) * RS);
                    double2 *o = reinterpret_cast<double2 *>(b.realb + (size_t)(dr * cstride + y) * RS);
                    for (int k = part * kp; k < min((part + 1) * kp, kn >> 1); ++k) {
                        double2 v = g[k];
                        v.x *= sm[0];
                        v.y *= sm[0];
#pragma unroll
                        for (int m = 1; m < 2 * TCE_ECO - 1; ++m)
                            if (m <= mm) {
                                const double2 z = g[m * (RS / 2) + k];
                                v.x = fma(sm[m], z.x, v.x);
                                v.y = fma(sm[m], z.y, v.y);
                            }
                        o[k] = v;
                    }
                }
                __syncwarp();
            }
#pragma unroll 1
            for (int p0 = q0; p0 < q0 + qn; p0 += PW) {
                const int pn = q0 + qn - p0 < PW ? q0 + qn - p0 : PW;
                if (!few) {   // the primitive quartet's coefficient products of bra and ket components
                    const short4 ix = b.qidx[p0];
                    const double fac = b.qfac[p0];
                    for (int x = lane; x < nAB + nCD; x += 32) {
                        const int z = x - nAB;
                        if (x < nAB) {
                            const int ca = x % Q.nA, cb = x / Q.nA;
                            b.cf[x] = fac * (coA[ca * npA + ix.x] * apow(Q.SI, ca)) * (coB[cb * npB + ix.y] * apow(Q.SJ, cb));
                        } else {
                            const int cc = z % Q.nC, cd = z / Q.nC;
                            b.cf[36 + z] = (coC[cc * npC + ix.z] * apow(Q.SK, cc)) * (coD[cd * npD + ix.w] * apow(Q.SL, cd));
                        }
                    }
                    __syncwarp();
                }
                // sum_k w_k I_x I_y I_z per component: one lane per component (and primitive
                // quartet), two nodes per load
                const int p = p0 + pl;
                for (int c = cl; c < Q.ncq && pl < pn; c += 32) {
                    const unsigned cm = few ? cm0 : b.cmap[c];
                    const double2 *rw[3];
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const int x = (cm >> (8 * d)) & 255;
                        rw[d] = reinterpret_cast<const double2 *>(d < ndp ? b.rows + (size_t)(d * per + p * ncomb + x) * RS
                                                                          : b.realb + (size_t)((d - ndp) * cstride + (p - q0) * ncomb + x) * RS);
                    }
                    const double2 *wk2 = reinterpret_cast<const double2 *>(b.wts), *wg2 = wk2 + 16;
                    double vK = 0.0, vG = 0.0, vK1 = 0.0, vG1 = 0.0;
#pragma unroll 4
                    for (int k = 0; k < (kn >> 1); ++k) {
                        const double2 x = rw[0][k], y = rw[1][k], z = rw[2][k], w = wk2[k];
                        const double a0 = x.x * y.x * z.x, a1 = x.y * y.y * z.y;
                        vK = fma(w.x, a0, vK);
                        vK1 = fma(w.y, a1, vK1);
                        if (judge) {
                            const double2 g = wg2[k];
                            vG = fma(g.x, a0, vG);
                            vG1 = fma(g.y, a1, vG1);
                        }
                    }
                    if (few) {
                        const short4 ix = b.qidx[p];
                        const double f = b.qfac[p] * f0 * (coA[ix.x] * coB[ix.y] * coC[ix.z] * coD[ix.w]);
                        accK = fma(f, vK + vK1, accK);
                        if (judge) accG = fma(f, vG + vG1, accG);
                    } else {
                        const int cd = c / nAB;
                        const double f = b.cf[c - cd * nAB] * b.cf[36 + cd];
                        b.blkK[c] = fma(f, vK + vK1, b.blkK[c]);
                        if (judge) b.blkG[c] = fma(f, vG + vG1, b.blkG[c]);
                    }
                }
                __syncwarp();
            }
        }
    }
    accK_ += accK;
    accG_ += accG;
}

// The same batch on the CUDA cores over every order of the reference's truncation
// (tensor cores off, density-fitting blocks), accumulating into blkK (and blkG).
// The fit's pivoted Cholesky follows the last bits of its integrals where
// symmetric functions tie, so this form keeps its order of operations.
template <int NQ, bool RO>
__device__ __forceinline__ void process_batch_every(const DevSys &S, int wofs, int nb, int lane, int cstride)
{
    const QCtx &Q = warp_ctx(wofs);
    const RuleView &Rv = Q.R_;
    const WarpBuf b = warp_buf(wofs);
    constexpr int NC = NQ < TCE_NC ? NQ : TCE_NC;
    constexpr int RS = NC + 1;
    const int ndp = S.ndp, nreal = 3 - ndp;
    const int lsA = Q.lsA, lsB = Q.lsB, lsC = Q.lsC, lsD = Q.lsD, ncomb = Q.ncomb, R = Q.R;
    const int nppb = Q.Ub.npp, nppk = Q.Uk.npp;
    const int nrows = nb * R;
    int cqg = 1;   // lanes per component: 32 / next power of two of the component count
    while (cqg < Q.ncq && cqg < 32) cqg <<= 1;
    cqg = 32 / cqg;
    const int npA = S.sh_np[Q.SI], npB = S.sh_np[Q.SJ], npC = S.sh_np[Q.SK], npD = S.sh_np[Q.SL];
    const bool judge = Rv.wg != nullptr;
#pragma unroll 1
    for (int k0 = 0; k0 < NQ; k0 += NC) {
        const int g0c = k0 / 8, kn = NQ - k0 < NC ? NQ - k0 : NC;
        for (int r = lane; r < nrows; r += 32) {
            int p = r / R, rem = r - p * R;
            int d = rem / ncomb, cmb = rem - d * ncomb;
            int ia = cmb % (lsA + 1), t1 = cmb / (lsA + 1);
            int ib = t1 % (lsB + 1), t2 = t1 / (lsB + 1);
            int ic = t2 % (lsC + 1), id = t2 / (lsC + 1);
            int2 pq = b.qlist[p];
            const PairPrim &Pb = S.pp[Q.Ub.pp_off + pq.x];
            const PairPrim &Pk = S.pp[Q.Uk.pp_off + pq.y];
            const double2 *G = S.vec + Q.Ub.vec_off +
                               ((((long long)d * (lsA + 1) + ia) * (lsB + 1) + ib) * 2 + 0) * (long long)Q.Ub.Nlen * nppb;
            const double2 *H = S.vec + Q.Uk.vec_off +
                               ((((long long)d * (lsC + 1) + ic) * (lsD + 1) + id) * 2 + 1) * (long long)Q.Uk.Nlen * nppk;
            int nm = Pb.N[d] < Pk.N[d] ? Pb.N[d] : Pk.N[d];
            double phi = S.a[d] * (Pb.cen[d] - (Pk.cen[d] + Q.Tsh[d]));
            double sgn = pow(S.a[d], -(double)(ia + ib + ic + id));
            row_dot<NQ, RO>(Rv, d, G, nppb, pq.x, H, nppk, pq.y, nm, phi, sgn, g0c, b.rows + (size_t)r * RS);
        }
        __syncwarp();
        for (int p = 0; p < nb; ++p) {
            int2 pq = b.qlist[p];
            const PairPrim &Pb = S.pp[Q.Ub.pp_off + pq.x];
            const PairPrim &Pk = S.pp[Q.Uk.pp_off + pq.y];
            const double pp_ = Pb.esum, qq = Pk.esum;
            if (nreal > 0) {
                const double *Eb = S.ecoef + Q.Ub.e_off + (long long)pq.x * nreal * (lsA + 1) * (lsB + 1) * TCE_ECO;
                const double *Ek = S.ecoef + Q.Uk.e_off + (long long)pq.y * nreal * (lsC + 1) * (lsD + 1) * TCE_ECO;
                for (int k = lane; k < kn; k += 32) {
                    double t = Rv.t[k0 + k], t2 = t * t;
                    const double rr = rsqrt(pp_ * qq + (pp_ + qq) * t2), D2 = rr * rr;
                    double w = pp_ * qq * t2 * D2, rs = PI_D * rr;
                    for (int dr = 0; dr < nreal; ++dr) {
                        int d = ndp + dr;
                        double Rr = Pb.cen[d] - (Pk.cen[d] + Q.Tsh[d]);
                        double gt[4 * TCE_LMAX + 2];
                        gt[0] = (Rr == 0.0) ? rs : rs * exp(-w * Rr * Rr);
                        double gm1 = 0.0, g0 = gt[0];
                        for (int n = 0; n < Q.NN; ++n) {
                            double gp1 = 2.0 * w * Rr * g0 - 2.0 * (double)n * w * gm1;
                            gt[n + 1] = gp1;
                            gm1 = g0;
                            g0 = gp1;
                        }
                        for (int cmb = 0; cmb < ncomb; ++cmb) {
                            int ia = cmb % (lsA + 1), u1 = cmb / (lsA + 1);
                            int ib = u1 % (lsB + 1), u2 = u1 / (lsB + 1);
                            int ic = u2 % (lsC + 1), id = u2 / (lsC + 1);
                            const double *eb = Eb + ((dr * (lsA + 1) + ia) * (lsB + 1) + ib) * TCE_ECO;
                            const double *ek = Ek + ((dr * (lsC + 1) + ic) * (lsD + 1) + id) * TCE_ECO;
                            double val = 0.0;
                            for (int n = 0; n <= ia + ib; ++n) {
                                double sb = (n & 1) ? -eb[n] : eb[n];
                                for (int kk = 0; kk <= ic + id; ++kk) val += sb * ek[kk] * gt[n + kk];
                            }
                            b.realb[((size_t)dr * cstride + cmb) * RS + k] = val;
                        }
                    }
                }
                __syncwarp();
            }
            const double fac = b.qfac[p];
            const double *rowp = b.rows + (size_t)p * R * RS;
            const int i = pq.x / Q.Ub.np2, j = pq.x % Q.Ub.np2;
            const int kp = pq.y / Q.Uk.np2, lp = pq.y % Q.Uk.np2;
            // The component quartets: sum_k w_k I_x I_y I_z per component.  G lanes
            // share one component and split its nodes (G = 32 / next power of two of
            // the component count, at most NQ), so that the warp holds 32 / G
            // components at once and each needs log2(G) shuffles instead of a full
            // warp reduction; each component's block entry has one owning lane.
            const int G = cqg < NC ? cqg : NC;
            const int slots = 32 / G, slot = lane / G, sub = lane - slot * G;
            for (int c0 = 0; c0 < Q.ncq; c0 += slots) {
                const int cq = c0 + slot;
                double vK = 0.0, vG = 0.0;
                int ca = 0, cb = 0, cc = 0, cd = 0;
                if (cq < Q.ncq) {
                    ca = cq % Q.nA;
                    const int r1 = cq / Q.nA;
                    cb = r1 % Q.nB;
                    const int r2 = r1 / Q.nB;
                    cc = r2 % Q.nC;
                    cd = r2 / Q.nC;
                    const int *pa = S.fn_pw + 3 * (S.sh_first[Q.SI] + ca);
                    const int *pb = S.fn_pw + 3 * (S.sh_first[Q.SJ] + cb);
                    const int *pc = S.fn_pw + 3 * (S.sh_first[Q.SK] + cc);
                    const int *pd = S.fn_pw + 3 * (S.sh_first[Q.SL] + cd);
                    const double *rw[3];
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const int cm = pa[d] + (lsA + 1) * (pb[d] + (lsB + 1) * (pc[d] + (lsC + 1) * pd[d]));
                        rw[d] = (d < ndp) ? rowp + ((size_t)d * ncomb + cm) * RS
                                          : b.realb + ((size_t)(d - ndp) * cstride + cm) * RS;
                    }
                    // two partial sums per estimate: shorter dependent FMA chains
                    double vK1 = 0.0, vG1 = 0.0;
                    int k = sub;
                    for (; k + G < kn; k += 2 * G) {
                        const double p0 = rw[0][k] * rw[1][k] * rw[2][k];
                        const double p1 = rw[0][k + G] * rw[1][k + G] * rw[2][k + G];
                        vK = fma(Rv.wk[k0 + k], p0, vK);
                        vK1 = fma(Rv.wk[k0 + k + G], p1, vK1);
                        if (judge) {
                            vG = fma(Rv.wg[k0 + k], p0, vG);
                            vG1 = fma(Rv.wg[k0 + k + G], p1, vG1);
                        }
                    }
                    if (k < kn) {
                        const double p0 = rw[0][k] * rw[1][k] * rw[2][k];
                        vK = fma(Rv.wk[k0 + k], p0, vK);
                        if (judge) vG = fma(Rv.wg[k0 + k], p0, vG);
                    }
                    vK += vK1;
                    vG += vG1;
                }
                for (int o = G >> 1; o > 0; o >>= 1) {
                    vK += __shfl_xor_sync(0xffffffffu, vK, o);
                    if (judge) vG += __shfl_xor_sync(0xffffffffu, vG, o);
                }
                if (cq < Q.ncq && sub == 0) {
                    const double cf = S.sh_coef[S.sh_coff[Q.SI] + ca * npA + i] * S.sh_coef[S.sh_coff[Q.SJ] + cb * npB + j] *
                                      S.sh_coef[S.sh_coff[Q.SK] + cc * npC + kp] * S.sh_coef[S.sh_coff[Q.SL] + cd * npD + lp];
                    b.blkK[cq] += fac * cf * vK;
                    if (judge) b.blkG[cq] += fac * cf * vG;
                }
            }
            __syncwarp();
        }
    }
}

__device__ __forceinline__ void make_ctx(const DevSys &S, int4 q, QCtx &Q)
{
    Q.SI = q.x; Q.SJ = q.y; Q.SK = q.z; Q.SL = q.w;
    Q.nA = S.sh_n[Q.SI]; Q.nB = S.sh_n[Q.SJ]; Q.nC = S.sh_n[Q.SK]; Q.nD = S.sh_n[Q.SL];
    Q.lsA = S.sh_l[Q.SI]; Q.lsB = S.sh_l[Q.SJ]; Q.lsC = S.sh_l[Q.SK]; Q.lsD = S.sh_l[Q.SL];
    Q.ncomb = (Q.lsA + 1) * (Q.lsB + 1) * (Q.lsC + 1) * (Q.lsD + 1);
    Q.ncq = Q.nA * Q.nB * Q.nC * Q.nD;
    Q.cqp = 1;
    while (Q.cqp < Q.ncq && Q.cqp < 32) Q.cqp <<= 1;
    Q.NN = Q.lsA + Q.lsB + Q.lsC + Q.lsD;
    Q.R = Q.ncomb * S.ndp;
    const int cK = Q.SK / S.nshuc;
    const int SK0 = Q.SK - cK * S.nshuc;
    const int SLp = tce_shift_to(Q.SL, cK, S.nshuc, S.ncl);
    Q.Ub = S.up[(long long)Q.SI * S.nsh + Q.SJ];
    Q.Uk = S.up[(long long)SK0 * S.nsh + SLp];
#pragma unroll
    for (int d = 0; d < 3; ++d) Q.Tsh[d] = S.sh_r[3 * Q.SK + d] - S.sh_r[3 * SK0 + d];
}

// The block of one shell quartet with its rule (Q.R_): screen and batch the primitive
// quartets, accumulate into b.blkK (and b.blkG); both are zeroed first.
template <int NQ, bool RO, bool TC>
__device__ __forceinline__ void eval_block(const DevSys &S, const QuartetArgs &A, int wofs, int lane, int want)
{
    const QCtx &Q = warp_ctx(wofs);
    const WarpBuf b = warp_buf(wofs);
    double accK = 0.0, accG = 0.0;
    for (int c = lane; c < Q.ncq; c += 32) {
        b.blkK[c] = 0.0;
        b.blkG[c] = 0.0;
        if (!TC) continue;
        // the power combination of each direction
        const int ca = c % Q.nA, r1 = c / Q.nA, cb = r1 % Q.nB, r2 = r1 / Q.nB, cc = r2 % Q.nC, cd = r2 / Q.nC;
        const int *pa = S.fn_pw + 3 * (S.sh_first[Q.SI] + ca), *pb = S.fn_pw + 3 * (S.sh_first[Q.SJ] + cb);
        const int *pc = S.fn_pw + 3 * (S.sh_first[Q.SK] + cc), *pd = S.fn_pw + 3 * (S.sh_first[Q.SL] + cd);
        unsigned cm = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d)
            cm |= (unsigned)(pa[d] + (Q.lsA + 1) * (pb[d] + (Q.lsB + 1) * (pc[d] + (Q.lsC + 1) * pd[d]))) << (8 * d);
        b.cmap[c] = cm;
    }
    for (int x = lane; TC && x < Q.ncomb; x += 32) {
        const int ia = x % (Q.lsA + 1), t1 = x / (Q.lsA + 1), ib = t1 % (Q.lsB + 1), t2 = t1 / (Q.lsB + 1);
        b.dig[x] = (unsigned char)(ia | ib << 2 | (t2 % (Q.lsC + 1)) << 4 | (t2 / (Q.lsC + 1)) << 6);
    }
    __syncwarp();
    auto batch = [&](int n) {
        if constexpr (TC) process_batch<NQ, RO>(wofs, n, lane, A.cstride, accK, accG);
        else process_batch_every<NQ, RO>(S, wofs, n, lane, A.cstride);
    };
    int B = A.rowcap / Q.R;
    if (B < 1) B = 1;
    const int nppb = Q.Ub.npp, nppk = Q.Uk.npp;
    const long long total = (long long)nppb * nppk;
    int nb = 0;
    for (long long base = 0; base < total; base += 32) {
        long long idx = base + lane;
        bool keep = idx < total;
        int ipb = 0, ipk = 0;
        double fac = 0.0;
        if (keep) {
            ipb = (int)(idx / nppk);
            ipk = (int)(idx - (long long)ipb * nppk);
            const PairPrim &Pb = S.pp[Q.Ub.pp_off + ipb];
            const PairPrim &Pk = S.pp[Q.Uk.pp_off + ipk];
            fac = S.fac_const * Pb.pfac * Pk.pfac;
            if (A.mode == TCE_MODE_PRIMTAB) {
                keep = (ipb == want) && (ipk == want);
            } else if (A.mode != TCE_MODE_NOSCREEN) {
                // prefactor screens (ERI_shell_block_toroidal.f90:191,216) and the
                // primitive Schwarz screen (:217-219)
                double bra = fabs(S.fac_const * Pb.pfac) * Pb.cmax12;
                if (bra * Q.Uk.ket_max <= 2.22e-16) keep = false;
                else if (fabs(fac) * Pb.cmax12 * Pk.cmax12 <= 2.22e-16) keep = false;
                else if (A.prim_screen && Pb.ps * Pk.ps < S.prim_thr) keep = false;
            }
        }
        const unsigned msk = __ballot_sync(0xffffffffu, keep);
        const int pos = __popc(msk & ((1u << lane) - 1u));
        const int cnt = __popc(msk);
        int done = 0;
        while (done < cnt) {
            int take = B - nb;
            if (take > cnt - done) take = cnt - done;
            if (keep && pos >= done && pos < done + take) {
                b.qlist[nb + pos - done] = make_int2(ipb, ipk);
                if (TC) {
                    const int i = ipb / Q.Ub.np2, k = ipk / Q.Uk.np2;
                    b.qidx[nb + pos - done] = make_short4((short)i, (short)(ipb - i * Q.Ub.np2), (short)k, (short)(ipk - k * Q.Uk.np2));
                }
                b.qfac[nb + pos - done] = fac;
            }
            nb += take;
            done += take;
            __syncwarp();
            if (nb == B) {
                batch(nb);
                nb = 0;
                __syncwarp();
            }
        }
    }
    if (nb > 0) batch(nb);
    if (TC && Q.ncq <= 32) {
        for (int o = Q.cqp; o < 32; o <<= 1) {
            accK += __shfl_xor_sync(0xffffffffu, accK, o);
            accG += __shfl_xor_sync(0xffffffffu, accG, o);
        }
        if (lane < Q.ncq) {
            b.blkK[lane] = accK;
            b.blkG[lane] = accG;
        }
    }
    __syncwarp();
}

__device__ __forceinline__ RuleView dict_rule(const DevSys &S, const QuartetArgs &A, int r, bool judge)
{
    const RuleDev &D = A.rules[r];
    RuleView R;
    R.T = A.rule_T + D.T_off;
    R.strideD = (long long)(S.ncap + 1) * D.nq;
    R.t = A.rule_t + D.node_off;
    R.wk = A.rule_wk + D.node_off;
    R.wg = judge ? A.rule_wg + D.node_off : nullptr;
    R.gmax = D.gmax;
    R.t2 = D.t2;
    return R;
}

// The consumer of a finished block (J/K, stored ERIs, blocks, primitive table)
__device__ void consume(const DevSys &S, const QuartetArgs &A, const QCtx &Q, const WarpBuf &b, int it, int lane,
                        int want)
{
    const double *blk = b.blkK;
    const int nA = Q.nA, nB = Q.nB, nC = Q.nC, nD = Q.nD;
    if (A.mode == TCE_MODE_BLOCK || A.mode == TCE_MODE_NOSCREEN) {
        double *o = A.blk_out + A.blk_off[it];
        for (int c = lane; c < Q.ncq; c += 32) o[c] = blk[c];
        if (A.blk_out2) {
            double *o2 = A.blk_out2 + A.blk_off[it];
            for (int c = lane; c < Q.ncq; c += 32) o2[c] = b.blkG[c];
        }
    } else if (A.mode == TCE_MODE_PRIMTAB) {
        if (lane == 0) {
            double m = 0.0;
            for (int a = 0; a < nA; ++a)
                for (int c = 0; c < nB; ++c) {
                    double v = sqrt(fabs(blk[a + nA * (c + nB * (a + nA * c))]));
                    if (v > m) m = v;
                }
            A.pp_rw[Q.Ub.pp_off + want].ps = m;
        }
    } else {
        const int fI = S.sh_first[Q.SI], fJ = S.sh_first[Q.SJ], fK = S.sh_first[Q.SK], fL = S.sh_first[Q.SL];
        for (int cq = lane; cq < Q.ncq; cq += 32) {
            int ca = cq % nA, r1 = cq / nA;
            int cb = r1 % nB, r2 = r1 / nB;
            int cc = r2 % nC, cd = r2 / nC;
            int f[4] = {fI + ca, fJ + cb, fK + cc, fL + cd};
            if (S.Q[f[0] + (long long)S.nbas * f[1]] * S.Q[f[2] + (long long)S.nbas * f[3]] < S.thr) continue;
            const double val = blk[cq];
            if (A.mode == TCE_MODE_STORE) {
                tce_store_eri(S, A.eri, A.eri_size, A.physicist, f, val);
                continue;
            }
            tce_scatter_jk(S, A.P, A.J, A.K, f, val, fI, nA, fJ, nB, fK, nC, fL, nD);
        }
    }
}

// Error estimate of a block from its Kronrod (blkK) and Gauss (blkG) values,
// in the form of QUADPACK's QK rules (Piessens et al. 1983): with
// e = max |K - G| and the block scale M = max |K|,
// est = M min(1, (200 e / M)^1.5)  (est = e when M = 0).
__device__ __forceinline__ double block_judge(const double *K, const double *G, int ncq, int lane)
{
    double e = 0.0, M = 0.0;
    for (int c = lane; c < ncq; c += 32) {
        e = fmax(e, fabs(K[c] - G[c]));
        M = fmax(M, fabs(K[c]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        e = fmax(e, __shfl_xor_sync(0xffffffffu, e, o));
        M = fmax(M, __shfl_xor_sync(0xffffffffu, M, o));
    }
    if (M <= 0.0 || e <= 0.0) return e;
    const double r = 200.0 * e / M;
    return r >= 1.0 ? M : M * r * sqrt(r);
}

__device__ __forceinline__ int item_count(const QuartetArgs &A)
{
    return A.nitems_dev ? (int)*A.nitems_dev : A.nitems;
}

// method 0: one fixed rule for every item (the system's rule, or dictionary rule
// rule_override, judged when blk_out2 is set); method 1: the learned grid.
// TC: rows on the tensor cores over few orders, 128 registers; else every order
// on the CUDA cores, whose 32 node sums per lane want 255.  With both in one kernel
// of 128 registers and the tensor-core form's buffers the every-order form took
// (16-cell chain, 40 nodes / 12 cells, 128 nodes / 3x2 sheet / 2x2x2 cube, ms)
// 39.8 / 121 / 44.5 / 30.9; by itself 21.7 / 54.5 / 30.8 / 23.5.
template <int NQ, bool TC>
__global__ void __launch_bounds__(256, TC ? 2 : 1) k_quartets(DevSys S, QuartetArgs A)
{
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    blk_header(S, A.lay);
    const int wofs = TCE_HDR_DOUBLES + wib * A.warp_smem_doubles;
    const WarpBuf b = warp_buf(wofs);
    QCtx &Q = warp_ctx(wofs);
    const bool lg = (A.method == TCE_METHOD_LEARNED);
    if (lane == 0 && !lg) {
        if (A.rule_override >= 0) {
            Q.R_ = dict_rule(S, A, A.rule_override, A.blk_out2 != nullptr);
        } else {
            RuleView R;
            R.T = S.Tt;
            R.strideD = (long long)(S.ncap + 1) * S.nq;
            R.t = S.tnode;
            R.wk = S.tweight;
            R.wg = nullptr;
            R.gmax = A.fixed_gmax;
            R.t2 = S.rule_t2;
            Q.R_ = R;
        }
    }
    const int nitems = item_count(A);
    while (true) {
        int it = 0;
        if (lane == 0) it = (int)atomicAdd(A.next, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= nitems) break;
        if (lane == 0) {
            make_ctx(S, A.items[it], Q);
            if (lg) Q.R_ = dict_rule(S, A, A.item_rule[it], true);
        }
        __syncwarp();
        int want = -1;
        if (A.mode == TCE_MODE_PRIMTAB) want = A.prim_sel[2 * it] * Q.Ub.np2 + A.prim_sel[2 * it + 1];
        eval_block<NQ, true, TC>(S, A, wofs, lane, want);
        if (lg) {
            const double e = block_judge(b.blkK, b.blkG, Q.ncq, lane);
            if (!(e <= A.judge_tol)) {      // the judge rejects the predicted rule
                if (lane == 0) {
                    unsigned int slot = atomicAdd(A.fb_count, 1u);
                    A.fb_items[slot] = A.items[it];
                    if (A.fb_index) A.fb_index[slot] = it;
                }
                __syncwarp();
                continue;
            }
        }
        consume(S, A, Q, b, it, lane, want);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// The plain method.  Per panel [a,b] of u the warp computes the Bessel columns
// c_n e^{-C} I_n(C), C = 2 t^2 / a^2, of the panel's 15 nodes (lane k: node k)
// into its HBM scratch:
//   C <= 125: Miller recurrence from nneed + 30 + sqrt(80 C), normalised by
//             e^{-C} I_0(C), as the system's t-tables (setup_t_tables,
//             clifford_tools.f90:620-709);
//   C >  125: the two top orders Ns+1, Ns (Ns >= 50, where I_n/I_0 has fallen
//             to about 1e-30 or at nneed + 1) from Debye's uniform asymptotic
//             expansion (Abramowitz & Stegun 9.7.7, terms u_0..u_13), then the
//             stable downward recurrence I_{n-1} = I_{n+1} + (2n/C) I_n.
// Either way the column is truncated 5 orders past the first entry below
// 1e-16 of I~_0, like the t-tables.  Then the warp evaluates the block and
// keeps splitting the panel with the largest error estimate (block_judge) at
// its middle until the summed estimates are below plain_tol or
// plain_max_panels panels are in use.
// ---------------------------------------------------------------------------
#define TCE_DEBYE_K 14
__constant__ double c_debye[TCE_DEBYE_K][TCE_DEBYE_K];   // u_k(p) = p^k sum_j c[k][j] p^{2j}

__device__ __forceinline__ double tce_ive_debye(double nu, double x)
{
    const double z = x / nu, w = sqrt(1.0 + z * z), p = 1.0 / w, p2 = p * p;
    double s = 0.0, pk = 1.0, ik = 1.0;
    const double inv = 1.0 / nu;
#pragma unroll
    for (int k = 0; k < TCE_DEBYE_K; ++k) {
        double P = c_debye[k][k];
        for (int j = k - 1; j >= 0; --j) P = fma(P, p2, c_debye[k][j]);
        s = fma(pk * ik, P, s);
        pk *= p;
        ik *= inv;
    }
    return exp(nu * (1.0 / (w + z) + log(z / (1.0 + w)))) / sqrt(2.0 * PI_D * nu * w) * s;
}

__device__ void plain_columns(const DevSys &S, const QuartetArgs &A, double *T, int nneed, double a, double bnd,
                              double *tn, double *wk, double *wg, int *gmax, float2 *t2, int lane)
{
    double t = 0.0, w1 = 0.0, w2 = 0.0;
    if (lane < 15) {
        const double u = a + (bnd - a) * A.gk_u[lane];
        const double jac = (bnd - a) * A.plain_scale / ((1.0 - u) * (1.0 - u));
        t = A.plain_scale * u / (1.0 - u);
        w1 = A.gk_wk[lane] * jac;
        w2 = A.gk_wg[lane] * jac;
    }
    if (lane < 16) {
        tn[lane] = t;
        wk[lane] = w1;
        wg[lane] = w2;
    }
    {   // t^2 range of the two node groups (the 16th node is padding)
        float lo = lane < 15 ? (float)(t * t) : __int_as_float(0x7f800000), hi = lane < 15 ? lo : -lo;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane < 16 && (lane & 7) == 0) t2[lane >> 3] = make_float2(lo * 0.999999f, hi * 1.000001f);
    }
    for (int d = 0; d < S.ndp; ++d) {
        double *Td = T + (size_t)d * (nneed + 1) * 16;
        int tnm = -1;
        if (lane < 15) {
            const double C = 2.0 * t * t / (S.a[d] * S.a[d]);
            if (C < 1e-12) {
                for (int n = 0; n <= nneed; ++n) Td[(size_t)n * 16 + lane] = (n == 0) ? 1.0 : 0.0;
                tnm = 0;
            } else {
                double norm = 1.0;
                if (C <= 125.0) {
                    const long long n0 = (long long)nneed + 30 + (long long)sqrt(80.0 * C);
                    double ip1 = 0.0, ik = 1e-300, im1;
                    for (long long kk = n0; kk >= 1; --kk) {
                        im1 = ip1 + (2.0 * (double)kk / C) * ik;
                        ip1 = ik;
                        ik = im1;
                        if (kk - 1 <= nneed) Td[(size_t)(kk - 1) * 16 + lane] = ik;
                        if (fabs(ik) > 1e250) {
                            for (long long m = kk - 1; m <= nneed; ++m) Td[(size_t)m * 16 + lane] *= 1e-250;
                            ip1 *= 1e-250;
                            ik *= 1e-250;
                        }
                    }
                    norm = tce_iv0_scaled(C) / Td[lane];
                } else {
                    int Ns = (int)ceil(sqrt(140.0 * C)) + 10;
                    if (Ns > nneed + 1) Ns = nneed + 1;
                    if (Ns < 50) Ns = 50;
                    double ip1 = tce_ive_debye((double)(Ns + 1), C), ik = tce_ive_debye((double)Ns, C), im1;
                    for (int n = Ns + 1; n <= nneed; ++n) Td[(size_t)n * 16 + lane] = 0.0;
                    if (Ns <= nneed) Td[(size_t)Ns * 16 + lane] = ik;
                    for (int n = Ns; n >= 1; --n) {
                        im1 = ip1 + (2.0 * (double)n / C) * ik;
                        ip1 = ik;
                        ik = im1;
                        if (n - 1 <= nneed) Td[(size_t)(n - 1) * 16 + lane] = ik;
                    }
                }
                const double w0 = Td[lane];
                tnm = nneed;
                for (int n = 0; n <= nneed; ++n)
                    if (Td[(size_t)n * 16 + lane] < 1e-16 * w0) {
                        tnm = (n + 5 < nneed) ? n + 5 : nneed;
                        break;
                    }
                for (int n = 0; n <= nneed; ++n) {
                    const double v = Td[(size_t)n * 16 + lane] * norm;
                    Td[(size_t)n * 16 + lane] = (n == 0) ? v : (n <= tnm ? 2.0 * v : 0.0);
                }
            }
        } else if (lane == 15) {
            for (int n = 0; n <= nneed; ++n) Td[(size_t)n * 16 + lane] = 0.0;
        }
        int g0 = lane < 8 ? tnm : -1;
        int g1 = (lane >= 8 && lane < 16) ? tnm : -1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            g0 = max(g0, __shfl_xor_sync(0xffffffffu, g0, o));
            g1 = max(g1, __shfl_xor_sync(0xffffffffu, g1, o));
        }
        if (lane == 0) {
            gmax[d * TCE_MAXG + 0] = g0;
            gmax[d * TCE_MAXG + 1] = g1;
        }
    }
    __syncwarp();
}

// 168 registers: the columns' recurrences and the panels' bookkeeping spill at 128
// (plain method, 24-cell chain 185 / 177 ms at 128 / 168; learned grid of the 2x1x1
// cube, which waits for its plain list, 6.6 / 6.0).
template <bool TC>
__global__ void __launch_bounds__(128, 3) k_plain(DevSys S, QuartetArgs A)
{
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    blk_header(S, A.lay);
    const int wofs = TCE_HDR_DOUBLES + wib * A.warp_smem_doubles;
    const WarpBuf b = warp_buf(wofs);
    QCtx &Q = warp_ctx(wofs);
    // extra: panel bounds and errors, the panel's nodes and weights, gmax
    double *pa = b.extra, *pb = pa + PLAIN_PMAX, *perr = pb + PLAIN_PMAX;
    double *tn = perr + PLAIN_PMAX, *wk = tn + 16, *wg = wk + 16;
    int *gmax = reinterpret_cast<int *>(wg + 16);
    float2 *t2 = reinterpret_cast<float2 *>(gmax + 3 * TCE_MAXG);
    const long long gw = (long long)blockIdx.x * (blockDim.x >> 5) + wib;
    double *T = A.scratch + gw * A.scratch_per_warp;
    double *pblk = T + A.T_doubles;      // [PLAIN_PMAX][blkcap]
    const int plimit = A.plain_max_panels < PLAIN_PMAX ? A.plain_max_panels : PLAIN_PMAX;
    for (int g = lane; g < 3 * TCE_MAXG; g += 32) gmax[g] = -1;
    __syncwarp();
    const int nitems = item_count(A);
    while (true) {
        int it = 0;
        if (lane == 0) it = (int)atomicAdd(A.next, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= nitems) break;
        if (lane == 0) make_ctx(S, A.items[it], Q);
        __syncwarp();
        int nneed = 0;
        {   // largest truncation order among the bra's pair primitives (bounds min(N_bra, N_ket))
            int m = 0;
            for (int x = lane; x < Q.Ub.npp; x += 32)
                for (int d = 0; d < S.ndp; ++d) m = max(m, S.pp[Q.Ub.pp_off + x].N[d]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            nneed = m;
        }
        unsigned long long evals = 0;
        if (lane == 0) {
            RuleView R;
            R.T = T;
            R.strideD = (long long)(nneed + 1) * 16;
            R.t = tn;
            R.wk = wk;
            R.wg = wg;
            R.gmax = gmax;
            R.t2 = t2;
            Q.R_ = R;
        }
        __syncwarp();
        auto eval_panel = [&](int slot, double a, double bnd) {
            plain_columns(S, A, T, nneed, a, bnd, tn, wk, wg, gmax, t2, lane);
            eval_block<16, false, TC>(S, A, wofs, lane, -1);
            const double e = block_judge(b.blkK, b.blkG, Q.ncq, lane);
            for (int c = lane; c < Q.ncq; c += 32) pblk[(size_t)slot * A.blkcap + c] = b.blkK[c];
            if (lane == 0) {
                pa[slot] = a;
                pb[slot] = bnd;
                perr[slot] = e;
            }
            evals += 15;
            __syncwarp();
        };
        eval_panel(0, 0.0, 1.0);
        int np = 1;
        while (np < plimit) {
            double tot = 0.0, worst = -1.0;
            int wi = 0;
            for (int p = 0; p < np; ++p) {
                tot += perr[p];
                if (perr[p] > worst) {
                    worst = perr[p];
                    wi = p;
                }
            }
            if (tot <= A.plain_tol) break;
            const double a = pa[wi], bnd = pb[wi], m = 0.5 * (a + bnd);
            __syncwarp();
            eval_panel(wi, a, m);
            eval_panel(np, m, bnd);
            ++np;
        }
        for (int c = lane; c < Q.ncq; c += 32) {
            double v = 0.0;
            for (int p = 0; p < np; ++p) v += pblk[(size_t)p * A.blkcap + c];
            b.blkK[c] = v;
        }
        __syncwarp();
        if (lane == 0 && A.node_evals) atomicAdd(A.node_evals, evals);
        consume(S, A, Q, b, it, lane, -1);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// launch
// ---------------------------------------------------------------------------
// Warps per block and blocks per SM of k_quartets<NQ, TC> for a per-warp buffer of
// wbytes: the shape with the most warps resident on an SM (shared memory and
// registers decide), found once per (NQ, TC, wbytes) with the occupancy calculator.
template <int NQ, bool TC>
static int2 quartet_shape(size_t wbytes)
{
    static std::mutex mu;
    static std::map<size_t, int2> known;
    std::lock_guard<std::mutex> lock(mu);
    auto it = known.find(wbytes);
    if (it != known.end()) return it->second;
    int2 best = make_int2(0, 0);   // (warps, blocks per SM)
    for (int w = 8; w >= 1; --w) {
        const size_t smem = TCE_HDR_DOUBLES * 8 + wbytes * (size_t)w;
        if (smem > 226 * 1024) continue;
        cudaFuncSetAttribute(k_quartets<NQ, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        int per = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_quartets<NQ, TC>, 32 * w, smem) != cudaSuccess) per = 0;
        if (per * w > best.x * best.y) best = make_int2(w, per);
    }
    known[wbytes] = best;
    return best;
}

template <int NQ, bool TC>
static cudaError_t launch_form(const DevSys &S, const QuartetArgs &A, size_t wbytes, int nsm, cudaStream_t st)
{
    const int2 sh = quartet_shape<NQ, TC>(wbytes);
    if (sh.x < 1 || sh.y < 1) return cudaErrorInvalidConfiguration;
    const size_t smem = TCE_HDR_DOUBLES * 8 + wbytes * (size_t)sh.x;
    cudaFuncSetAttribute(k_quartets<NQ, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_quartets<NQ, TC><<<nsm * sh.y, 32 * sh.x, smem, st>>>(S, A);
    return cudaGetLastError();
}

template <int NQ>
static cudaError_t launch_nq(bool tc, const DevSys &S, const QuartetArgs &A, size_t wbytes, int nsm, cudaStream_t st)
{
    return tc ? launch_form<NQ, true>(S, A, wbytes, nsm, st) : launch_form<NQ, false>(S, A, wbytes, nsm, st);
}

// Debye polynomials u_k(t) (Abramowitz & Stegun 9.3.9-9.3.10):
//   u_0 = 1, u_{k+1}(t) = t^2 (1 - t^2) u_k'(t) / 2 + (1/8) int_0^t (1 - 5 s^2) u_k(s) ds,
// generated in long double; u_k(t) = t^k sum_j c[k][j] t^{2j}.  Uploaded once per device.
static int upload_debye()
{
    static std::mutex mu;
    static bool done[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TCE_ERR_CUDA;
    std::lock_guard<std::mutex> lock(mu);
    if (done[dev]) return TCE_OK;
    std::vector<std::vector<long double>> U(1, std::vector<long double>(1, 1.0L));
    for (int k = 0; k + 1 < TCE_DEBYE_K; ++k) {
        const std::vector<long double> &u = U.back();
        std::vector<long double> nx(u.size() + 3, 0.0L);
        for (size_t i = 1; i < u.size(); ++i) {         // t^2 (1 - t^2) u' / 2
            const long double du = (long double)i * u[i];
            nx[i + 1] += 0.5L * du;
            nx[i + 3] -= 0.5L * du;
        }
        for (size_t i = 0; i < u.size(); ++i) {         // (1/8) int_0^t (1 - 5 s^2) u
            nx[i + 1] += u[i] / (8.0L * (long double)(i + 1));
            nx[i + 3] -= 5.0L * u[i] / (8.0L * (long double)(i + 3));
        }
        U.push_back(nx);
    }
    double c[TCE_DEBYE_K][TCE_DEBYE_K] = {};
    for (int k = 0; k < TCE_DEBYE_K; ++k)
        for (int j = 0; j <= k; ++j) {
            const size_t e = (size_t)(k + 2 * j);
            c[k][j] = e < U[k].size() ? (double)U[k][e] : 0.0;
        }
    if (cudaMemcpyToSymbol(c_debye, c, sizeof c) != cudaSuccess) return TCE_ERR_CUDA;
    done[dev] = true;
    return TCE_OK;
}

long long tce_plain_scratch_per_warp(const DevSys &S, int max_ncq)
{
    const int blkcap = (max_ncq + 3) / 4 * 4;
    return (long long)S.ndp * (S.ncap + 1) * 16 + (long long)PLAIN_PMAX * blkcap;
}

// The per-warp buffers of a launch: layout and capacities into A, their bytes
static size_t quartet_buffers(const DevSys &S, int nq, bool tc, bool plain, int max_ncomb, int max_ncq, QuartetArgs &A)
{
    const int R = max_ncomb * S.ndp;
    const int rowcap = std::max(R, tc ? 16 * S.ndp : 32);   // at least a tile of rows per periodic direction, or a row per lane
    const int RS = (nq < TCE_NC ? nq : TCE_NC) + (tc ? 2 : 1);   // rows of one chunk of at most 32 nodes
    const int nreal = 3 - S.ndp;
    const int blkcap = (max_ncq + 3) / 4 * 4;
    // real-direction rows: of one primitive quartet, or (tensor-core form) 32 / cqp small ones
    const int cstride = tc && max_ncomb < 16 ? 16 : max_ncomb;
    A.lay = tce_warp_layout(tc, rowcap, RS, nreal, cstride, blkcap, (nq + 15) / 16);
    long long wdoubles = A.lay.extra;
    if (plain) wdoubles += 3 * PLAIN_PMAX + 48 + 3 * TCE_MAXG / 2 + 4;
    wdoubles = (wdoubles + 31) / 32 * 32;
    A.rowcap = rowcap;
    A.cstride = cstride;
    A.blkcap = blkcap;
    A.warp_smem_doubles = (int)wdoubles;
    return (size_t)wdoubles * sizeof(double);
}

long long tce_quartet_resident(const DevSys &S, int max_ncomb, int max_ncq, int nsm)
{
    QuartetArgs A;
    const size_t wbytes = quartet_buffers(S, S.nq, true, false, max_ncomb, max_ncq, A);
    const int2 sh = S.nq == 32   ? quartet_shape<32, true>(wbytes)
                    : S.nq == 40 ? quartet_shape<40, true>(wbytes)
                    : S.nq == 64 ? quartet_shape<64, true>(wbytes)
                                 : quartet_shape<128, true>(wbytes);
    return (long long)sh.x * sh.y * (nsm > 0 ? nsm : 148);
}

int tce_launch_quartets(const DevSys &S, const QuartetHostArgs &h, cudaStream_t st)
{
    QuartetArgs A;
    A.items = h.items;
    A.prim_sel = h.prim_sel;
    A.nitems = h.nitems;
    A.nitems_dev = h.nitems_dev;
    A.mode = h.mode;
    A.method = h.method;
    A.prim_screen = h.prim_screen;
    A.next = h.next;
    A.blk_out = h.blk_out;
    A.blk_out2 = h.blk_out2;
    A.blk_off = h.blk_off;
    A.P = h.P;
    A.J = h.J;
    A.K = h.K;
    A.eri = h.eri;
    A.eri_size = h.eri_size;
    A.physicist = h.physicist;
    A.pp_rw = h.pp_rw;
    A.fixed_gmax = h.fixed_gmax;
    A.rules = h.rules;
    A.rule_T = h.rule_T;
    A.rule_t = h.rule_t;
    A.rule_wk = h.rule_wk;
    A.rule_wg = h.rule_wg;
    A.item_rule = h.item_rule;
    A.rule_override = h.rule_override;
    A.judge_tol = h.judge_tol;
    A.fb_items = h.fb_items;
    A.fb_index = h.fb_index;
    A.fb_count = h.fb_count;
    A.scratch = h.scratch;
    A.plain_tol = h.plain_tol;
    A.plain_scale = h.plain_scale;
    A.plain_max_panels = h.plain_max_panels;
    A.gk_u = h.gk_u;
    A.gk_wk = h.gk_wk;
    A.gk_wg = h.gk_wg;
    A.node_evals = h.node_evals;
    if (h.use_tc < 0) return TCE_ERR_ARG;
    const bool plain = (h.method == TCE_METHOD_PLAIN);
    const bool dict = (h.method == TCE_METHOD_LEARNED) || h.rule_override >= 0;
    if (plain && (h.mode == TCE_MODE_PRIMTAB || !h.scratch || !h.gk_u)) return TCE_ERR_ARG;
    if (dict && (!h.rules || !h.rule_T)) return TCE_ERR_ARG;
    if (h.method == TCE_METHOD_LEARNED && (!h.item_rule || !h.fb_items || !h.fb_count)) return TCE_ERR_ARG;
    if (!plain && !dict && !h.fixed_gmax) return TCE_ERR_ARG;
    const int nq = plain ? 16 : (dict ? h.dict_nq : S.nq);
    const bool tc = h.use_tc != 0;
    const size_t wbytes = quartet_buffers(S, nq, tc, plain, h.max_ncomb, h.max_ncq, A);
    int warps = 4;
    while (warps > 1 && wbytes * warps > 220 * 1024) --warps;
    if (wbytes > 220 * 1024) return TCE_ERR_UNSUPPORTED;
    const size_t smem = TCE_HDR_DOUBLES * 8 + wbytes * warps;
    if (cudaMemsetAsync(h.next, 0, sizeof(unsigned int), st) != cudaSuccess) return TCE_ERR_CUDA;
    const int nsm = h.num_sms > 0 ? h.num_sms : 148;
    cudaError_t e;
    if (plain) {
        if (upload_debye() != TCE_OK) return TCE_ERR_CUDA;
        A.T_doubles = (long long)S.ndp * (S.ncap + 1) * 16;
        A.scratch_per_warp = tce_plain_scratch_per_warp(S, h.max_ncq);
        auto kern = tc ? k_plain<true> : k_plain<false>;
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        int per = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, 32 * warps, smem);
        if (per < 1) per = 1;
        long long grid = (long long)nsm * per;
        if (grid * warps > h.scratch_warps) grid = h.scratch_warps / warps;
        // a list of known length takes no more warps than it has quartets: the
        // plain list runs next to the learned-grid kernels, and its idle blocks
        // would hold the registers and shared memory they need
        if (!h.nitems_dev && h.nitems > 0) grid = std::min<long long>(grid, (h.nitems + warps - 1) / warps);
        if (grid < 1) return TCE_ERR_NOMEM;
        kern<<<(unsigned)grid, 32 * warps, smem, st>>>(S, A);
        e = cudaGetLastError();
    } else if (nq == 32) e = launch_nq<32>(tc, S, A, wbytes, nsm, st);
    else if (nq == 40) e = launch_nq<40>(tc, S, A, wbytes, nsm, st);
    else if (nq == 64) e = launch_nq<64>(tc, S, A, wbytes, nsm, st);
    else if (nq == 128) e = launch_nq<128>(tc, S, A, wbytes, nsm, st);
    else return TCE_ERR_UNSUPPORTED;
    return e == cudaSuccess ? TCE_OK : TCE_ERR_CUDA;
}

template <int NQ>
static cudaError_t preload_nq()
{
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, k_quartets<NQ, true>);
    return e == cudaSuccess ? cudaFuncGetAttributes(&fa, k_quartets<NQ, false>) : e;
}

int tce_preload_quartets(int nq)
{
    cudaError_t e;
    if (nq == 32) e = preload_nq<32>();
    else if (nq == 40) e = preload_nq<40>();
    else if (nq == 64) e = preload_nq<64>();
    else if (nq == 128) e = preload_nq<128>();
    else return TCE_ERR_UNSUPPORTED;
    return e == cudaSuccess ? TCE_OK : TCE_ERR_CUDA;
}
