// tce_kmo.cu -- k-space MO integrals from the stored SAO integrals on the
// device (transform_ERI_AO_to_kMO, AO_to_MO_SAO.f90:34-393):
//   ERI_out(p, q, r, s, k1, k2, k3) = (p k1, q k2 | r k3, s k4),
//   k4 = k1 - k2 + k3, p, r in p_lo..p_hi, q, s in q_lo..q_hi.
// The handle's stored integrals ERI(a, j2, j3, j4) (tce_eri_stored with
// eri_size = nfuc, chemist order) stay on the device; per group of up to KMO_G k4:
//   k_kmo_x1: X1(a, j2, j3, d)    = sum_R4 ERI(a, j2, j3, d R4) e^{+i k4 R4}
//   k_kmo_x2: X2(a, j2, c, d, k3) = sum_R3 X1(a, j2, c R3, d) e^{-i k3 R3}
//   k_kmo_x3: S(a, b, c, d, k2, k3) = 1/N sum_R2 X2(a, b R2, c, d, k3) e^{+i k2 R2}
//   k_kmo_q : one block per (k1, k2), k3 = k4 - k1 + k2: the four quarter
//             transforms with the k-block coefficients
//             C_k(a, p) = coeff_SAO(k nfuc + a, k nfuc + p), in shared memory.
// The three sums over cells read every input once per KMO_T (x1: KMO_G) values of
// k, phases as shared-memory broadcasts; reading it once per k they moved N
// times the stored integrals, X1 and X2.  The groups follow each other on one
// stream without waiting for the host; the workspaces come from the pool of call
// memory (tce_pool.h).
#include <vector>

#include "tce_handle.h"

namespace {

__device__ __forceinline__ double2 kmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double2 kconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ void kadd(double2 &s, double2 v)
{
    s.x += v.x;
    s.y += v.y;
}

constexpr int KMO_G = 4;    // k4 values per group
constexpr int KMO_T = 8;    // k values per thread of the other two sums

constexpr int KMO_R = 128;  // cells per shared-memory tile of phases

// ph[k0 + j][r0 + R], j < T, R < KMO_R, into shared memory (zero past N)
template <int T>
__device__ __forceinline__ void kmo_phases(const double2 *__restrict__ ph, int k0, int r0, int N, double2 *sp)
{
    __syncthreads();
    for (int x = threadIdx.x; x < T * KMO_R; x += blockDim.x) {
        const int j = x % T, R = r0 + x / T;
        sp[x] = k0 + j < N && R < N ? ph[(size_t)(k0 + j) * N + R] : make_double2(0.0, 0.0);
    }
    __syncthreads();
}

__global__ void k_kmo_x1(int nf, int nbas, int N, int k4, int ng, const double *__restrict__ eri, const double2 *__restrict__ ph,
                         double2 *X1)
{
    __shared__ double2 sq[KMO_G * KMO_R];
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;   // a + nf (j2 + nbas (j3 + nbas d))
    const long long slab = (long long)nf * nbas * nbas, n = slab * nf;
    const long long abc = id % slab;
    const int d = (int)(id / slab);
    double2 s[KMO_G];
#pragma unroll
    for (int j = 0; j < KMO_G; ++j) s[j] = make_double2(0.0, 0.0);
    for (int r0 = 0; r0 < N; r0 += KMO_R) {
        kmo_phases<KMO_G>(ph, k4, r0, N, sq);
        for (int r = r0; id < n && r < min(N, r0 + KMO_R); ++r) {
            const double v = eri[(size_t)abc + (size_t)slab * (d + (size_t)r * nf)];
#pragma unroll
            for (int j = 0; j < KMO_G; ++j) {
                const double2 e = sq[(r - r0) * KMO_G + j];
                s[j].x = fma(v, e.x, s[j].x);
                s[j].y = fma(v, e.y, s[j].y);
            }
        }
    }
    if (id >= n) return;
#pragma unroll
    for (int j = 0; j < KMO_G; ++j)
        if (j < ng) X1[(size_t)n * j + id] = s[j];
}

// blockIdx.y: k3 tile, blockIdx.z: k4 of the group
__global__ void k_kmo_x2(int nf, int nbas, int N, const double2 *__restrict__ ph, const double2 *__restrict__ X1, double2 *X2)
{
    __shared__ double2 sq[KMO_T * KMO_R];
    const int k0 = blockIdx.y * KMO_T;
    // X2 index: a + nf (j2 + nbas (c + nf (d + nf k3)))
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long aj = (long long)nf * nbas, n = aj * nf * nf;
    X1 += (size_t)aj * nbas * nf * blockIdx.z;
    X2 += (size_t)n * N * blockIdx.z;
    const long long a2 = id % aj, cd = id / aj;
    const int c = (int)(cd % nf), d = (int)(cd / nf);
    double2 s[KMO_T];
#pragma unroll
    for (int j = 0; j < KMO_T; ++j) s[j] = make_double2(0.0, 0.0);
    for (int r0 = 0; r0 < N; r0 += KMO_R) {
        kmo_phases<KMO_T>(ph, k0, r0, N, sq);
        for (int r = r0; id < n && r < min(N, r0 + KMO_R); ++r) {
            const double2 x = X1[(size_t)a2 + (size_t)aj * ((c + (size_t)r * nf) + (size_t)nbas * d)];
#pragma unroll
            for (int j = 0; j < KMO_T; ++j) kadd(s[j], kmul(x, kconj(sq[(r - r0) * KMO_T + j])));
        }
    }
    if (id >= n) return;
#pragma unroll
    for (int j = 0; j < KMO_T; ++j)
        if (k0 + j < N) X2[(size_t)id + (size_t)n * (k0 + j)] = s[j];
}

// S(a, b, c, d; k2, k3), (a, b, c, d) fastest; blockIdx.y: k2 tile, blockIdx.z: k4 of the group
__global__ void k_kmo_x3(int nf, int nbas, int N, const double2 *__restrict__ ph, const double2 *__restrict__ X2, double2 *Sk)
{
    __shared__ double2 sq[KMO_T * KMO_R];
    const int k0 = blockIdx.y * KMO_T;
    const long long aj = (long long)nf * nbas, n = (long long)nf * nf * nf * nf;   // per (k2, k3)
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;         // (a, b, c, d) + n k3
    X2 += (size_t)aj * nf * nf * N * blockIdx.z;
    Sk += (size_t)n * N * N * blockIdx.z;
    const int ab = (int)(id % (nf * nf));
    const long long cdk = id / (nf * nf);                                          // c + nf (d + nf k3)
    const double2 *x2 = X2 + ab + (size_t)aj * cdk;
    double2 s[KMO_T];
#pragma unroll
    for (int j = 0; j < KMO_T; ++j) s[j] = make_double2(0.0, 0.0);
    for (int r0 = 0; r0 < N; r0 += KMO_R) {
        kmo_phases<KMO_T>(ph, k0, r0, N, sq);
        for (int r = r0; id < n * N && r < min(N, r0 + KMO_R); ++r) {
            const double2 x = x2[(size_t)nf * nf * r];
#pragma unroll
            for (int j = 0; j < KMO_T; ++j) kadd(s[j], kmul(x, sq[(r - r0) * KMO_T + j]));
        }
    }
    if (id >= n * N) return;
    const double invN = 1.0 / (double)N;
    const long long abcd = id % n, k3 = id / n;
#pragma unroll
    for (int j = 0; j < KMO_T; ++j)
        if (k0 + j < N) Sk[(size_t)abcd + (size_t)n * ((k0 + j) + (size_t)N * k3)] = make_double2(s[j].x * invN, s[j].y * invN);
}

struct KmoArgs {
    int nf, nbas, N, no, nv, p0, q0, k4, n0, n1, n2;
    const double2 *Sk, *C;   // C: coeff_SAO (nbas x nbas), column-major
    double2 *out;           // (no, nv, no, nv, N, N, N)
};

// blockIdx.y: k4 of the group
__global__ void k_kmo_q(KmoArgs A)
{
    extern __shared__ double2 sq[];
    const int nf = A.nf, N = A.N, no = A.no, nv = A.nv, nbas = A.nbas;
    const int k1 = blockIdx.x / N, k2 = blockIdx.x % N, k4 = A.k4 + blockIdx.y;
    auto wrap = [](int c, int n) { return (c % n + n) % n; };
    const int k3 = wrap(k4 % A.n0 - k1 % A.n0 + k2 % A.n0, A.n0) +
                   A.n0 * (wrap((k4 / A.n0) % A.n1 - (k1 / A.n0) % A.n1 + (k2 / A.n0) % A.n1, A.n1) +
                           A.n1 * wrap(k4 / (A.n0 * A.n1) - k1 / (A.n0 * A.n1) + k2 / (A.n0 * A.n1), A.n2));
    const int f2 = nf * nf, f3 = f2 * nf, f4 = f3 * nf;
    double2 *S = sq;                    // (a, b, c, d)
    double2 *T4 = S + f4;               // (a, b, c, s)
    double2 *T3 = T4 + f3 * nv;         // (a, b, r, s)
    double2 *T2 = T3 + f2 * no * nv;    // (a, q, r, s)
    const int t = threadIdx.x, nt = blockDim.x;
    auto C = [&](int k, int a, int p) { return A.C[(size_t)(k * nf + a) + (size_t)nbas * (k * nf + p)]; };
    const double2 *Sg = A.Sk + (size_t)f4 * (k2 + (size_t)N * (k3 + (size_t)N * blockIdx.y));
    for (int x = t; x < f4; x += nt) S[x] = Sg[x];
    __syncthreads();
    for (int x = t; x < f3 * nv; x += nt) {   // 4th index d -> s
        const int abc = x % f3, s = x / f3;
        double2 v = make_double2(0.0, 0.0);
        for (int d = 0; d < nf; ++d) kadd(v, kmul(S[abc + f3 * d], C(k4, d, A.q0 + s)));
        T4[x] = v;
    }
    __syncthreads();
    for (int x = t; x < f2 * no * nv; x += nt) {   // 3rd index c -> r (conjugated)
        const int ab = x % f2, r = (x / f2) % no, s = x / (f2 * no);
        double2 v = make_double2(0.0, 0.0);
        for (int c = 0; c < nf; ++c) kadd(v, kmul(T4[ab + f2 * c + f3 * s], kconj(C(k3, c, A.p0 + r))));
        T3[x] = v;
    }
    __syncthreads();
    for (int x = t; x < nf * nv * no * nv; x += nt) {   // 2nd index b -> q
        const int a = x % nf, q = (x / nf) % nv, rs = x / (nf * nv);
        double2 v = make_double2(0.0, 0.0);
        for (int b = 0; b < nf; ++b) kadd(v, kmul(T3[a + nf * b + f2 * rs], C(k2, b, A.q0 + q)));
        T2[x] = v;
    }
    __syncthreads();
    const long long blk = (long long)no * nv * no * nv;
    double2 *o = A.out + (size_t)blk * (k1 + (size_t)N * (k2 + (size_t)N * k3));
    for (int x = t; x < blk; x += nt) {   // 1st index a -> p (conjugated)
        const int p = x % no, qrs = x / no;
        double2 v = make_double2(0.0, 0.0);
        for (int a = 0; a < nf; ++a) kadd(v, kmul(kconj(C(k1, a, A.p0 + p)), T2[a + nf * qrs]));
        o[x] = v;
    }
}

}  // namespace

using namespace tcehost;

extern "C" int tce_ao_to_kmo(void *handle, const double *coeff, int32_t p_lo, int32_t p_hi, int32_t q_lo, int32_t q_hi,
                             double *out)
{
    Handle *h = static_cast<Handle *>(handle);
    if (!h || !coeff || !out) return fail(h, TCE_ERR_ARG, "NULL argument");
    const int nf = h->nfuc, nbas = h->nbas, N = h->ncell;
    if (p_lo < 1 || p_hi < p_lo || p_hi > nf || q_lo < 1 || q_hi < q_lo || q_hi > nf)
        return fail(h, TCE_ERR_ARG, "band ranges must lie in 1..nfuc");
    if (!h->d_eri || h->eri_size != nf || h->physicist)
        return fail(h, TCE_ERR_STATE, "needs the stored SAO integrals in chemist order (tce_eri_stored, eri_size = nfuc)");
    const int no = p_hi - p_lo + 1, nv = q_hi - q_lo + 1;
    const size_t smem = sizeof(double2) * ((size_t)nf * nf * nf * nf + (size_t)nf * nf * nf * nv +
                                           (size_t)nf * nf * no * nv + (size_t)nf * nv * no * nv);
    if (smem > 200 * 1024) return fail(h, TCE_ERR_UNSUPPORTED, "nfuc too large for the quarter-transform kernel");
    // phases (cells x fastest)
    std::vector<int> cx(N), cy(N), cz(N);
    for (int k = 0; k < N; ++k) {
        cx[k] = k % h->ncl[0];
        cy[k] = (k / h->ncl[0]) % h->ncl[1];
        cz[k] = k / (h->ncl[0] * h->ncl[1]);
    }
    std::vector<double2> ph((size_t)N * N);
    for (int k = 0; k < N; ++k)
        for (int r = 0; r < N; ++r) {
            const double th = 2.0 * kPi * ((double)cx[k] * cx[r] / h->ncl[0] + (double)cy[k] * cy[r] / h->ncl[1] +
                                          (double)cz[k] * cz[r] / h->ncl[2]);
            ph[(size_t)k * N + r] = make_double2(std::cos(th), std::sin(th));
        }
    const size_t f4 = (size_t)nf * nf * nf * nf;
    const size_t n1 = (size_t)nf * nbas * nbas * nf, n2 = (size_t)nf * nbas * nf * nf * N, n3 = f4 * N * N;
    const size_t nout = (size_t)no * nv * no * nv * N * N * N, nC = (size_t)nbas * nbas, nph = (size_t)N * N;
    // k4 per group (S shares X1's buffer): as many as the pool keeps the buffers
    // of, at least one; one also where the device has no room for more
    int G = std::min(KMO_G, N);
    auto bytes = [&](int g) { return sizeof(double2) * ((size_t)g * (std::max(n1, n3) + n2) + nout + nC + nph); };
    while (G > 1 && bytes(G) > TCE_POOL_KEEP) --G;
    double2 *d_ph = nullptr, *d_C = nullptr, *d_X1 = nullptr, *d_X2 = nullptr, *d_out = nullptr;
    CallMemory mem(h->st);
    auto take = [&](int g) {
        return mem.get(&d_ph, nph) && mem.get(&d_C, nC) && mem.get(&d_X1, g * std::max(n1, n3)) && mem.get(&d_X2, g * n2) &&
               mem.get(&d_out, nout);
    };
    if (!take(G)) {
        mem.drop_all();
        const int first = G;
        G = 1;
        if (first == 1 || !take(1))
            return fail(h, TCE_ERR_NOMEM, "device allocation of " + std::to_string(bytes(1)) + " bytes failed");
    }
    CK(h, cudaMemcpyAsync(d_ph, ph.data(), sizeof(double2) * nph, cudaMemcpyHostToDevice, h->st));
    CK(h, cudaMemcpyAsync(d_C, coeff, sizeof(double2) * nC, cudaMemcpyHostToDevice, h->st));
    CK(h, cudaFuncSetAttribute(k_kmo_q, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const unsigned tiles = (unsigned)((N + KMO_T - 1) / KMO_T);
    for (int k4 = 0; k4 < N; k4 += G) {
        const int ng = std::min(G, N - k4);
        k_kmo_x1<<<(unsigned)((n1 + 255) / 256), 256, 0, h->st>>>(nf, nbas, N, k4, ng, h->d_eri, d_ph, d_X1);
        k_kmo_x2<<<dim3((unsigned)((n2 / N + 127) / 128), tiles, ng), 128, 0, h->st>>>(nf, nbas, N, d_ph, d_X1, d_X2);
        k_kmo_x3<<<dim3((unsigned)((f4 * N + 127) / 128), tiles, ng), 128, 0, h->st>>>(nf, nbas, N, d_ph, d_X2, d_X1);
        KmoArgs A{nf, nbas, N, no, nv, p_lo - 1, q_lo - 1, k4, h->ncl[0], h->ncl[1], h->ncl[2], d_X1, d_C, d_out};
        k_kmo_q<<<dim3((unsigned)(N * N), ng), 256, smem, h->st>>>(A);
        CK(h, cudaGetLastError());
    }
    CK(h, cudaMemcpyAsync(out, d_out, sizeof(double2) * nout, cudaMemcpyDeviceToHost, h->st));
    CK(h, cudaStreamSynchronize(h->st));
    return TCE_OK;
}
