// Pieces shared by the two Hankel-transform tensor builders on the GPU: the IE Green's tensor
// (green.cu, calc_ie_tensor_module.F90) and the receiver tensor (continuation.cu,
// calc_rc_tensor_module.F90).
//   * the volume Bessel transform tables (VolumeBesselTransforms.F90:111-139) and the FFT deconvolution
//     that turns 1024 samples of an output function into the 501 Hankel weights (CalcWeights22,
//     :264-288);
//   * the layered-medium recursions of apq_module.F90 (Calc_Apq, Calc_p, Calc_q, Calc_pexpz_All,
//     Calc_qexpz_All) for one lambda, on one thread, 1-based layer and cell arrays;
//   * the FP64 GEMM that sums weights x lambda basis into the tensor.
// Everything sits in an anonymous namespace: each translation unit gets its own copy.
#pragma once
#include <cmath>
#include <vector>
#include <cuda/std/complex>
#include "common.cuh"

namespace {

using cplx = cuda::std::complex<double>;

constexpr int VN = 1024, VLOG = 10, NFIRST = 212, NLAST = 712, NLAM = NLAST - NFIRST + 1;
constexpr double Y_STEP = 1e-1 * 2e0;
constexpr double XI = -4.82205425726955430357775925664462079e-2 * 2e0;
constexpr double VQ = Y_STEP / 2.0;
constexpr double VP = VQ + XI;
constexpr int VN2 = -VN / 2;
constexpr double PI_D = 3.14159265358979323846264338327950288;
constexpr double SPI = 1.77245385090551602729816748334114518;
constexpr double WT_THRESHOLD = 1e-12;
constexpr int MAXL = 16;   // layers supported by the device recursion
constexpr int MAXZ = 64;   // cells in z supported by the device recursion

struct Bkg {
    int Nl, Nz;
    double2 csigma[MAXL + 1];  // 0..Nl
    double2 k2[MAXL + 1];
    double thick[MAXL + 1];    // 1..Nl-1
    double depth[MAXL + 1];    // 1..Nl-1
    double2 iwm;
    int L[MAXZ + 1];           // Lnumber 0..Nz
    double z[MAXZ + 1];        // 0..Nz
    double dz[MAXZ + 1];       // 1..Nz
};

G2_D cplx C(double2 v) { return cplx(v.x, v.y); }
G2_D double2 D2(cplx v) { return make_double2(v.real(), v.imag()); }

// Calc_Apq without the A matrix (apq_module.F90:230-248) with Calc_p (:267-290) and Calc_q (:291-312)
G2_D void dev_apq(const Bkg &b, double lms, cplx *eta, cplx *el, cplx (*p)[2], cplx (*q)[2], cplx (*Arr)[2])
{
    const int Nl = b.Nl;
    const cplx cs0 = C(b.csigma[0]);
    for (int i = 1; i <= Nl; i++) eta[i] = cuda::std::sqrt(lms * lms - C(b.k2[i]));
    for (int i = 1; i <= Nl - 1; i++) el[i] = cuda::std::exp(-2.0 * eta[i] * b.thick[i]);
    el[Nl] = 0.0;
    {  // Calc_p (:267-290)
        const cplx eta0 = cuda::std::sqrt(lms * lms - C(b.k2[0]));
        const cplx ceta = eta0 / eta[1];
        p[1][0] = (1.0 - ceta) / (1.0 + ceta);
        const cplx cgamma = cs0 / C(b.csigma[1]);
        p[1][1] = (cgamma - ceta) / (cgamma + ceta);
        for (int i = 2; i <= Nl; i++) {
            cplx w[2] = {el[i - 1] * p[i - 1][0], el[i - 1] * p[i - 1][1]};
            for (int k = 0; k < 2; k++) w[k] = (w[k] - 1.0) / (w[k] + 1.0);
            cplx a[2];
            a[0] = eta[i - 1] / eta[i];
            a[1] = a[0] * C(b.csigma[i]) / C(b.csigma[i - 1]);
            for (int k = 0; k < 2; k++) {
                w[k] = w[k] * a[k];
                p[i][k] = (1.0 + w[k]) / (1.0 - w[k]);
            }
        }
    }
    {  // Calc_q (:291-312)
        q[Nl][0] = q[Nl][1] = 0.0;
        if (Nl > 1) {
            cplx a[2];
            a[0] = eta[Nl] / eta[Nl - 1];
            a[1] = a[0] * C(b.csigma[Nl - 1]) / C(b.csigma[Nl]);
            for (int k = 0; k < 2; k++) q[Nl - 1][k] = (1.0 - a[k]) / (1.0 + a[k]);
            for (int i = Nl - 2; i >= 1; i--) {
                cplx w[2] = {el[i + 1] * q[i + 1][0], el[i + 1] * q[i + 1][1]};
                for (int k = 0; k < 2; k++) w[k] = (w[k] - 1.0) / (w[k] + 1.0);
                a[0] = eta[i + 1] / eta[i];
                a[1] = a[0] * C(b.csigma[i]) / C(b.csigma[i + 1]);
                for (int k = 0; k < 2; k++) {
                    w[k] = w[k] * a[k];
                    q[i][k] = (1.0 + w[k]) / (1.0 - w[k]);
                }
            }
        }
    }
    for (int i = 1; i <= Nl; i++)
        for (int k = 0; k < 2; k++) Arr[i][k] = 1.0 / eta[i] / (1.0 - p[i][k] * q[i][k] * el[i]);
}

// Calc_pexpz_All (apq_module.F90:112-137): pez[i] for cells 1..Nz
G2_D void dev_pexpz(const Bkg &b, const cplx *eta, const cplx (*p)[2], const cplx *expz, cplx (*pez)[2])
{
    const int Nz = b.Nz;
    int l = b.L[0];
    cplx e;
    if (l > 1) e = cuda::std::exp(-2.0 * eta[l] * (b.z[0] - b.depth[l - 1]));
    else if (l == 1) e = cuda::std::exp(-2.0 * eta[1] * b.z[0]);
    else e = 1.0;
    for (int i = 1; i <= Nz; i++) {
        if (l != b.L[i]) e = 1.0;
        l = b.L[i];
        pez[i][0] = e * p[l][0];
        pez[i][1] = e * p[l][1];
        e = e * expz[i] * expz[i];
    }
}

// Calc_qexpz_All (apq_module.F90:155-177): qez[i] for cells 1..Nz
G2_D void dev_qexpz(const Bkg &b, const cplx *eta, const cplx (*q)[2], const cplx *expz, cplx (*qez)[2])
{
    const int Nz = b.Nz, Nl = b.Nl;
    int l = b.L[Nz];
    cplx e;
    if (l != Nl) e = cuda::std::exp(-2.0 * eta[l] * (b.depth[l] - b.z[Nz]));
    else e = 0.0;
    for (int i = Nz; i >= 1; i--) {
        if (l != b.L[i]) e = 1.0;
        l = b.L[i];
        qez[i][0] = e * q[l][0];
        qez[i][1] = e * q[l][1];
        e = e * expz[i] * expz[i];
    }
}

struct VbtTab {
    int inds[VN];
    double2 twf[VN / 2];  // exp(-i pi j / (VN/2)) style table for smem_fft: exp(-2 pi i j / VN), j < VN/2
    double2 f1[VN];
    double lms[NLAM];
    double lambda_shift;
};

// G radix-2 stages (half lengths 2^S0 .. 2^(S0+G-1)) of the 6 interleaved VN-point transforms in g, in registers: the
// butterflies of smem_fft, so the results are the same bits, with one trip through shared memory for G stages (ten trips
// each way made the weights of a 64x64x16 grid 1.44 ms and of its receivers 5.0 ms; now 1.00 and 3.2 ms, about half of
// it the samples' exponentials and error functions).
template <int S0, int G, bool INV> G2_D void vbt_stages(double2 *g, const double2 *__restrict__ tw)
{
    constexpr int M = 1 << G, ITEMS = (VN >> G) * 6;
    for (int it = threadIdx.x; it < ITEMS; it += 256) {
        const int c = it % 6, grp = it / 6, lo = grp & ((1 << S0) - 1), base = ((grp >> S0) << (S0 + G)) | lo;
        double2 *p = g + base * 6 + c;
        double2 v[M];
#pragma unroll
        for (int m = 0; m < M; m++) v[m] = p[(m << S0) * 6];
#pragma unroll
        for (int t = 0; t < G; t++)
#pragma unroll
            for (int q = 0; q < (1 << t); q++) {
                double2 w = tw[(lo + (q << S0)) << (VLOG - 1 - S0 - t)];
                if (INV) w.y = -w.y;
#pragma unroll
                for (int m = q; m < M; m += 2 << t) {
                    const double2 a = v[m], b = cmul(v[m + (1 << t)], w);
                    v[m] = a + b;
                    v[m + (1 << t)] = a - b;
                }
            }
#pragma unroll
        for (int m = 0; m < M; m++) p[(m << S0) * 6] = v[m];
    }
    __syncthreads();
}
template <bool INV> G2_D void vbt_fft(double2 *g, const double2 *__restrict__ tw)
{
    static_assert(VLOG == 10, "the stages below are those of 1024 points");
    vbt_stages<0, 4, INV>(g, tw);
    vbt_stages<4, 3, INV>(g, tw);
    vbt_stages<7, 3, INV>(g, tw);
}

// CalcWeights22 (VolumeBesselTransforms.F90:264-288) after the output function's samples are in g
// ([VN][6] in shared memory, bit-reversed positions): forward FFT, deconvolution by the input function's
// spectrum, inverse FFT.  The caller normalises (h/N with the alternating sign) and takes the real part.
// Needs blockDim.x == 256 and a __syncthreads() between filling g and the call.
G2_D void vbt_weights22(double2 *g, const VbtTab *__restrict__ T)
{
    vbt_fft<false>(g, T->twf);
    // deconvolution by the input function's spectrum, written back bit-reversed (CalcWeights22 :277-280);
    // every thread reads its pairs before any thread writes (the permutation is in place)
    static_assert(VN / 2 == 2 * 256, "k_weights is written for 256 threads, two sample pairs each");
    double2 pa[2][6], pb[2][6];
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int j = 2 * (threadIdx.x + r * 256);
#pragma unroll
        for (int c = 0; c < 6; c++) { pa[r][c] = g[j * 6 + c]; pb[r][c] = g[(j + 1) * 6 + c]; }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int j = 2 * (threadIdx.x + r * 256);
        const cplx f0 = C(T->f1[j]), f1v = C(T->f1[j + 1]);
        const int p0 = T->inds[j], p1 = T->inds[j + 1];
#pragma unroll
        for (int c = 0; c < 6; c++) {
            g[p0 * 6 + c] = D2(C(pa[r][c]) / f0);
            g[p1 * 6 + c] = D2(-C(pb[r][c]) / f1v);
        }
    }
    __syncthreads();
    vbt_fft<true>(g, T->twf);
}

// ---- (3) GEMM: out[lag][off + col] = scale * sum_k (A1[lag][k] B1[k][col] + A2[lag][k] B2[k][col]) --------
// on the FP64 tensor cores (mma.m8n8k4.f64): B's complex columns are pairs of real columns.  All components of the
// tensor in one launch (blockIdx.y = a column tile of a job).  A CTA of 8 warps sums GM lags x NT real columns; the
// operands come in k-tiles of 16 through a ring of cp.async stages whose row strides (4 mod 8 doubles) keep the
// fragment reads free of bank conflicts.  Most of a lag's 501 weights lie below the threshold and are zero: krange
// holds every lag's first and last kept wave number, and a CTA sums the union of its lags' ranges.
// Bound by the FP64 pipe.  At 64x64x16 the six sums take 0.36 ms; six launches of 2 x 2 outputs per thread on FMAs took 2.02 ms
// (5.4 TF); the fifteen of a receiver at 64x64x16 take 0.17 ms against 3.5 ms.
constexpr int GM = 128, GK = 16, GSA = GK + 4, GSTAGES = 3;
struct GemmJob {
    const double *A1, *A2;   // [lags][NLAM]; A2 null: one product
    const double2 *B1, *B2;  // [NLAM][ncols]
    int ncols, off;
};
struct GemmJobs {
    static constexpr int MAX = 16;
    GemmJob job[MAX];
    int tile0[MAX + 1];  // first column tile of each job
    int n = 0;
};
template <int NT> constexpr size_t gemm_smem() { return GSTAGES * (GM * GSA + GK * (NT + 4)) * sizeof(double); }

G2_D void cp_async(void *dst, const void *src, int bytes, bool valid)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = valid ? bytes : 0;  // the rest is zero-filled
    if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int NT>
__global__ void __launch_bounds__(256, 2) k_gemm(const __grid_constant__ GemmJobs jobs, const int2 *__restrict__ krange,
                                                 int nlags, double2 *out, int T, double scale)
{
    constexpr int SB = NT + 4;                          // row stride of the B stage
    constexpr int WN = NT / 32, WM = 8 / WN;            // warps along columns and lags
    constexpr int MT = GM / WM / 8;                     // 8-row tiles per warp; 4 column tiles
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *As = reinterpret_cast<double *>(smem_raw), *Bs = As + GSTAGES * GM * GSA;
    __shared__ int klo, khi;
    int j = 0;
    while ((int)blockIdx.y >= jobs.tile0[j + 1]) j++;
    const GemmJob &jb = jobs.job[j];
    const int m0 = blockIdx.x * GM, c0 = (blockIdx.y - jobs.tile0[j]) * (NT / 2);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        klo = NLAM;
        khi = 0;
    }
    __syncthreads();
    if (tid < GM && m0 + tid < nlags) {
        const int2 r = krange[m0 + tid];
        if (r.y > r.x) {
            atomicMin(&klo, r.x);
            atomicMax(&khi, r.y);
        }
    }
    __syncthreads();
    const int k_first = klo, ntiles = khi > klo ? (khi - klo + GK - 1) / GK : 0;
    const int total = ntiles * (jb.A2 ? 2 : 1);
    auto load = [&](int t, int stage) {
        const bool second = t >= ntiles;
        const double *A = second ? jb.A2 : jb.A1;
        const double2 *B = second ? jb.B2 : jb.B1;
        const int k0 = k_first + (second ? t - ntiles : t) * GK;
        double *as = As + stage * GM * GSA, *bs = Bs + stage * GK * SB;
#pragma unroll
        for (int i = 0; i < GM * GK / 256; i++) {
            const int e = tid + i * 256, m = e / GK, k = e % GK;
            const bool ok = m0 + m < nlags && k0 + k < NLAM;
            cp_async(as + m * GSA + k, A + (ok ? (size_t)(m0 + m) * NLAM + k0 + k : 0), 8, ok);
        }
#pragma unroll
        for (int i = 0; i < GK * NT / 2 / 256; i++) {
            const int e = tid + i * 256, k = e / (NT / 2), c = e % (NT / 2);
            const bool ok = k0 + k < NLAM && c0 + c < jb.ncols;
            cp_async(bs + k * SB + 2 * c, B + (ok ? (size_t)(k0 + k) * jb.ncols + c0 + c : 0), 16, ok);
        }
    };
    double acc[MT][4][2] = {};
    const int mw = (warp / WN) * (MT * 8), nw = (warp % WN) * 32, kl = lane & 3, nl = lane >> 2;
#pragma unroll
    for (int s = 0; s < GSTAGES - 1; s++) {
        if (s < total) load(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int t = 0; t < total; t++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GSTAGES - 2) : "memory");
        __syncthreads();  // tile t has landed for every thread, and every thread is done with tile t - 1
        if (t + GSTAGES - 1 < total) load(t + GSTAGES - 1, (t + GSTAGES - 1) % GSTAGES);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double *as = As + (t % GSTAGES) * GM * GSA + (mw + nl) * GSA + kl;
        const double *bs = Bs + (t % GSTAGES) * GK * SB + kl * SB + nw + nl;
#pragma unroll
        for (int k = 0; k < GK; k += 4) {
            double a[MT], b[4];
#pragma unroll
            for (int i = 0; i < MT; i++) a[i] = as[i * 8 * GSA + k];
#pragma unroll
            for (int i = 0; i < 4; i++) b[i] = bs[k * SB + i * 8];
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int n = 0; n < 4; n++)
                    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                        : "+d"(acc[i][n][0]), "+d"(acc[i][n][1])
                        : "d"(a[i]), "d"(b[n]));
        }
    }
    // lane (nl, kl): row nl, real columns 2 kl and 2 kl + 1 = one complex column
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int n = 0; n < 4; n++) {
            const int gm = m0 + mw + i * 8 + nl, gc = c0 + (nw + n * 8) / 2 + kl;
            if (gm < nlags && gc < jb.ncols)
                out[(size_t)gm * T + jb.off + gc] = make_double2(acc[i][n][0] * scale, acc[i][n][1] * scale);
        }
}

inline void add_job(GemmJobs &g, int NT, const double *A1, const double2 *B1, const double *A2, const double2 *B2, int ncols,
                    int off)
{
    g.job[g.n] = GemmJob{A1, A2, B1, B2, ncols, off};
    if (g.n == 0) g.tile0[0] = 0;
    g.tile0[g.n + 1] = g.tile0[g.n] + (2 * ncols + NT - 1) / NT;
    g.n++;
}
// column tiles of 32 where 64 would be half empty
inline cudaError_t launch_gemm(const GemmJobs &g, int NT, const int2 *krange, int nlags, double2 *out, int T, double scale,
                               cudaStream_t st)
{
    const dim3 grid((nlags + GM - 1) / GM, g.tile0[g.n]);
    cudaError_t e;
    if (NT == 64) {
        e = cudaFuncSetAttribute(k_gemm<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem<64>());
        if (e == cudaSuccess) k_gemm<64><<<grid, 256, gemm_smem<64>(), st>>>(g, krange, nlags, out, T, scale);
    } else {
        e = cudaFuncSetAttribute(k_gemm<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem<32>());
        if (e == cudaSuccess) k_gemm<32><<<grid, 256, gemm_smem<32>(), st>>>(g, krange, nlags, out, T, scale);
    }
    return e == cudaSuccess ? cudaGetLastError() : e;
}
inline int gemm_tile(int ncols) { return (2 * ncols + 63) / 64 * 64 - 2 * ncols >= 32 ? 32 : 64; }

// ---- host tables (VolumeBesselTransforms.F90:111-139) -------------------------------------------
int bitrev_vbt(int i)
{
    int t = i;
    for (int J = VLOG; J >= 2; J--) {
        const int mask = (1 << J) - 1;
        int low = t & mask;
        low = (low >> 1) | ((low & 1) << (J - 1));
        t = (t & ~mask) | low;
    }
    return t;
}
double input_function(double t)
{
    const double y = std::exp(-t), y2 = y * y, y4 = y2 * y2;
    return 8.0 * std::exp(-y2) * (y4 - 4.0 * y2 + 2.0) * y;
}
void make_vbt(double s, VbtTab &T)
{
    for (int i = 0; i < VN; i++) T.inds[i] = bitrev_vbt(i);
    for (int j = 0; j < VN / 2; j++) {
        const double th = -2.0 * PI_D * j / VN;
        T.twf[j] = make_double2(std::cos(th), std::sin(th));
    }
    for (int J = NFIRST; J <= NLAST; J++) T.lms[J - NFIRST] = std::exp(XI + (J + VN2) * Y_STEP) / s;
    T.lambda_shift = std::log(s);
    std::vector<double2> f(VN);
    for (int i = 0; i < VN; i += 2) {
        double y1 = (i + VN2) * Y_STEP + VQ;
        f[T.inds[i]] = make_double2(input_function(y1), 0.0);
        y1 = y1 + Y_STEP;
        f[T.inds[i + 1]] = make_double2(-input_function(y1), 0.0);
    }
    // radix-2 DIT on bit-reversed input (FFT_16, :630-649)
    for (int h = 1; h < VN; h <<= 1)
        for (int J = 0; J < h; J++) {
            const double th = -PI_D / h * J;
            const double wr = std::cos(th), wi = std::sin(th);
            for (int ip = J; ip < VN; ip += 2 * h) {
                const int iq = ip + h;
                const double tr = wr * f[iq].x - wi * f[iq].y, ti = wr * f[iq].y + wi * f[iq].x;
                f[iq] = make_double2(f[ip].x - tr, f[ip].y - ti);
                f[ip] = make_double2(f[ip].x + tr, f[ip].y + ti);
            }
        }
    for (int i = 0; i < VN; i++) T.f1[i] = f[i];
}

}  // namespace
