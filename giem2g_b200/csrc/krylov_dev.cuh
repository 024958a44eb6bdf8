// Device pieces of the Krylov solver shared by its kernels (arnoldi.cu: a whole Arnoldi step in one launch;
// krylov.cu: everything else): the state of one GMRES level, the reductions and the scalar steps.
#pragma once
#include "common.cuh"
#include "krylov.h"

struct Level {
    int m = 0;
    double2 *H = nullptr;   // (m+1) x (m+1) column-major, column m holds g
    double *cs = nullptr;
    double2 *sn = nullptr;
    double2 *y = nullptr;
    double *scal = nullptr;
    int *flags = nullptr;
    unsigned *counter = nullptr;  // blocks done, for the last-block reductions (back to 0 after each use)
    unsigned *bar = nullptr;      // the grid barrier of arnoldi.cu
};

// Several instances of one batch in one launch (blockIdx.y = instance): vectors of one length, and per instance its
// partials, barrier and gate.
constexpr int KMI = 4;
template <typename C>
struct Multi {
    C *V[KMI];
    C *w[KMI];
    double2 *part[KMI];
    Level L[KMI];
    const int *gate[KMI];
};

// arnoldi.cu: Arnoldi step j (dots, correction passes, scaling, Givens) of n instances in one cooperative launch
int arnoldi_step(const Multi<float2> &mm, int n, size_t N, int nparts, int j, double tol, int *err, cudaStream_t st);
int arnoldi_step(const Multi<double2> &mm, int n, size_t N, int nparts, int j, double tol, int *err, cudaStream_t st);

// The inner cycles of several instances that start together: v right side, x0 start (x: the copy the cycle's solution is
// added to), r = A x0 on entry of krylov_residual, V the basis.  go: 0 makes the instance's cycle do nothing.
template <typename C>
struct Starts {
    const C *v[KMI], *x0[KMI];
    C *x[KMI], *r[KMI], *V[KMI];
    double2 *part[KMI];
    Level L[KMI];
    const int *go[KMI];
};
// arnoldi.cu: bn = ||v||, x = x0 (0 where bn vanishes), the level's flags and H reset (gmres.F90:129-145)
template <typename C> int krylov_begin(const Starts<C> &s, int n, size_t N, int nparts, int *err, cudaStream_t st);
// r = v - r, beta = ||r||, exit or V_0 = r / beta and a started cycle (gmres.F90:147-185)
template <typename C>
int krylov_residual(const Starts<C> &s, int n, size_t N, int nparts, double tol, int *err, cudaStream_t st);

namespace {

constexpr int kVT = 256;   // threads of the vector kernels
constexpr int kILP = 4;    // elements per thread and iteration of the element-wise vector kernels
constexpr int KMAX = 32;   // largest basis handled in one sweep
constexpr double ZERO_THRESHOLD = 1e-14;  // gmres.F90:21
constexpr int N_IGS = 3;                  // gmres.F90:22
constexpr double kHookGain = 0.5;         // an outer step through the hook must halve the misfit

enum { F_KRYLOV = 0, F_L = 2, F_ITER = 3, F_SOLVER = 4, F_NFLAGS = 8 };
enum { S_BN = 0, S_BETA = 1, S_BEA = 4, S_NRM2 = 5, S_NSCAL = 8 };

G2_HD int hix(int i, int j, int m) { return i + j * (m + 1); }

template <typename C> G2_D double2 ld2(const C *p, size_t i);
template <> G2_D double2 ld2<double2>(const double2 *p, size_t i) { return p[i]; }
template <> G2_D double2 ld2<float2>(const float2 *p, size_t i)
{
    const float2 v = p[i];
    return make_double2(v.x, v.y);
}
template <typename C> G2_D void st2(C *p, size_t i, double2 v);
template <> G2_D void st2<double2>(double2 *p, size_t i, double2 v) { p[i] = v; }
template <> G2_D void st2<float2>(float2 *p, size_t i, double2 v) { p[i] = make_float2((float)v.x, (float)v.y); }

// The basis sweeps move 16-byte words: two complex64 values per load (complex128 values are 16 bytes
// already).  On a B200 a two-instance sweep of 11 complex64 vectors of 1.57 M elements took 84 us with
// 8-byte loads and 52 us with 16-byte loads.  Vectors whose length (and column stride) is odd keep
// element-wise loads, since their odd columns are not 16-byte aligned.
template <typename C> struct Wide;
template <> struct Wide<float2> {
    using T = float4;
    static constexpr int E = 2;
};
template <> struct Wide<double2> {
    using T = double2;
    static constexpr int E = 1;
};
G2_D float2 part_of(const float4 &p, int e) { return e ? make_float2(p.z, p.w) : make_float2(p.x, p.y); }
G2_D double2 part_of(const double2 &p, int) { return p; }
G2_D void set_part(float4 &p, int e, float2 v)
{
    if (e) {
        p.z = v.x;
        p.w = v.y;
    } else {
        p.x = v.x;
        p.y = v.y;
    }
}
G2_D void set_part(double2 &p, int, double2 v) { p = v; }
// words of E elements over the whole vector, or 0 when the lengths do not allow them
template <typename C> G2_D size_t wide_words(size_t N, size_t ld)
{
    constexpr int E = Wide<C>::E;
    return (N % E == 0 && ld % E == 0) ? N / E : 0;
}

template <typename C> struct RealOf;
template <> struct RealOf<double2> { using T = double; };
template <> struct RealOf<float2> { using T = float; };

// Sums over a block and into its row of the grid's partial sums, in FP64; total(k) is the thread's k-th sum.
template <int KM, class F> G2_D void block_reduce_store(F total, double2 *part)
{
    __shared__ double2 red[kVT / 32][KM + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k <= KM; k++) {
        double2 v = total(k);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        if (lane == 0) red[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x <= KM) {
        double2 s = make_double2(0.0, 0.0);
        for (int w = 0; w < kVT / 32; w++) {
            s.x += red[w][threadIdx.x].x;
            s.y += red[w][threadIdx.x].y;
        }
        part[(size_t)blockIdx.x * (KMAX + 1) + (threadIdx.x == KM ? KMAX : threadIdx.x)] = s;
    }
}
// per-thread sums in the vector's precision
template <int KM, typename R> G2_D void block_reduce_store_r(R (&ax)[KM + 1], R (&ay)[KM + 1], double2 *part)
{
    block_reduce_store<KM>([&](int k) { return make_double2(ax[k], ay[k]); }, part);
}

// ---- scalar steps -------------------------------------------------------------------------------
G2_D double cabs_(double2 a) { return hypot(a.x, a.y); }
G2_D double2 cmul_(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
G2_D double2 cdivr(double2 a, double r) { return make_double2(a.x / r, a.y / r); }
// netlib ZROT on one pair
G2_D void zrot1(double2 &cx, double2 &cy, double c, double2 s)
{
    const double2 t = make_double2(c * cx.x + (s.x * cy.x - s.y * cy.y), c * cx.y + (s.x * cy.y + s.y * cy.x));
    const double2 sc = make_double2(s.x, -s.y);
    cy = make_double2(c * cy.x - (sc.x * cx.x - sc.y * cx.y), c * cy.y - (sc.x * cx.y + sc.y * cx.x));
    cx = t;
}
// ---- fused reductions: the last block to finish sums every block's partials ----------------------
// Each block stores its partials, then counts itself done; the block that counts last reduces all
// partials in a fixed order (lane-strided sums, shuffle tree: the result does not depend on which block
// is last) and runs the scalar step that used to be a separate one-thread launch.  It resets the counter
// for the next use.  Blocks test their gates before any of them can reach the last block, so a flag the
// last block changes cannot be seen half-way through the grid.
G2_D bool last_block(unsigned *counter)
{
    __shared__ bool am_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) am_last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (am_last && threadIdx.x == 0) *counter = 0u;
    __threadfence();
    return am_last;
}
// (after a barrier or last_block, which order the loads) sums of part[b][col] over blocks for columns 0..K-1 into h[], and of column KMAX into *nrm (one block)
G2_D void reduce_partials(const double2 *part, int nb, int K, double2 *h, double *nrm)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int k = warp; k <= K; k += nw) {
        const int col = (k == K) ? KMAX : k;
        double sx = 0.0, sy = 0.0;
        // eight independent loads per lane and round (rows past nb predicated off): the partials come from
        // L2, and each round is one L2 round trip, so 256 rows cost one
        for (int b0 = 0; b0 < nb; b0 += 256) {
            double2 v[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int b = b0 + lane + 32 * q;
                v[q] = b < nb ? __ldcg(part + (size_t)b * (KMAX + 1) + col) : make_double2(0.0, 0.0);
            }
            sx += ((v[0].x + v[1].x) + (v[2].x + v[3].x)) + ((v[4].x + v[5].x) + (v[6].x + v[7].x));
            sy += ((v[0].y + v[1].y) + (v[2].y + v[3].y)) + ((v[4].y + v[5].y) + (v[6].y + v[7].y));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sx += __shfl_xor_sync(0xffffffffu, sx, o);
            sy += __shfl_xor_sync(0xffffffffu, sy, o);
        }
        if (lane == 0) {
            if (k < K) h[k] = make_double2(sx, sy);
            else if (nrm) *nrm = sx;
        }
    }
    __syncthreads();
}

// elements per thread and round of the basis sweeps: all (K + 1) * U loads of a round are issued before the
// first product, so a round costs one memory round trip; the values held stay within 256 bytes per thread
// (32 complex64 or 16 complex128).  0: the basis is too wide to hold, the sweep loads one element at a time.
template <int K, typename C> struct SweepU {
    static constexpr int B = (K + 1) * (int)sizeof(C);
    static constexpr int v = B * 4 <= 256 ? 4 : (B * 2 <= 256 ? 2 : (B <= 256 ? 1 : 0));
};

G2_D float2 scaled(float2 a, double s) { return make_float2((float)(a.x * s), (float)(a.y * s)); }
G2_D double2 scaled(double2 a, double s) { return make_double2(a.x * s, a.y * s); }

}  // namespace
