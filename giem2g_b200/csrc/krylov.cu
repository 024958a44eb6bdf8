// Nested flexible GMRES on the GPU: GFGMRES (GFGMRES/gmres.F90, seq_fgmres.F90) as used by
// GIEM2G_FGMRES (ie_solver_module.F90:141-258), depth 2.
//
//   outer: flexible GMRES, FP64 (complex128) basis, Hessenberg, Givens and true residual;
//          right preconditioner = one cycle of the inner GMRES (FGMRES_BASED_PRECONDITIONER).
//   inner: GMRES, MaxIt = 1, x0 = b = v_in, complex128 (plain mode) or complex64 (mixed mode).
//
// Arnoldi uses the reference's iterated classical Gram-Schmidt (gmres.F90:263-281): up to four
// passes, stop when 2||w|| > ||h_pass||; each pass after the first is ONE sweep over the basis that
// subtracts V h, and accumulates the next pass's dots and ||w||^2.  Complex Givens rotations follow
// the netlib ZROTG/ZROT definitions; restarts use the Arnoldi residual (RESTART_RESIDUAL = .FALSE.).
// Dot products and norms: complex128 in FP64; complex64 up to 16 elements of a thread in FP32 (arnoldi.cu; the norms of
// k_norm2_fused: a thread's part of the vector), their sums in FP64.
//
// The inner solve is a fixed launch sequence whose kernels are gated by device flags, so it needs no
// host round trip; the outer loop reads two scalars back once per outer iteration (Inform callback).
// The inner solver's closing true-residual apply (gmres.F90:403) produces a number nobody reads; it
// is skipped unless the environment variable GIEM2G_INNER_TRUE_RESIDUAL=1 asks for it (the solution
// and iteration history are the same either way; only the apply count differs).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>
#include "common.cuh"
#include "krylov_dev.cuh"

namespace {

// ||w||^2 into *nrm2
template <typename C>
__global__ void __launch_bounds__(kVT) k_norm2_fused(const C *__restrict__ w, size_t N, double2 *part, double *nrm2,
                                                     unsigned *counter, const int *gate)
{
    pdl_wait();
    if (gate && *gate == 0) return;
    using R = typename RealOf<C>::T;
    using W = typename Wide<C>::T;
    constexpr int E = Wide<C>::E, U = 4;  // 16-byte words, U of them loaded before the first product
    R ax[1] = {R(0)}, ay[1] = {R(0)};
    const size_t S = (size_t)gridDim.x * kVT, t0 = blockIdx.x * (size_t)kVT + threadIdx.x;
    const size_t Nw = wide_words<C>(N, N);
    const W *__restrict__ ww = reinterpret_cast<const W *>(w);
    size_t i = t0;
    for (; i + (U - 1) * S < Nw; i += U * S) {
        W v[U];
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = ww[i + u * S];
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int e = 0; e < E; e++) {
                const C a = part_of(v[u], e);
                ax[0] += a.x * a.x + a.y * a.y;
            }
    }
    for (; i < Nw; i += S) {
        const W v = ww[i];
#pragma unroll
        for (int e = 0; e < E; e++) {
            const C a = part_of(v, e);
            ax[0] += a.x * a.x + a.y * a.y;
        }
    }
    for (i = Nw * E + t0; i < N; i += S) {
        const C wv = w[i];
        ax[0] += wv.x * wv.x + wv.y * wv.y;
    }
    block_reduce_store_r<0, R>(ax, ay, part);
    if (!last_block(counter)) return;
    __shared__ double nrm;
    reduce_partials(part, gridDim.x, 0, nullptr, &nrm);
    if (threadIdx.x == 0) *nrm2 = nrm;
}

G2_D double2 widen(float2 a) { return make_double2(a.x, a.y); }
G2_D double2 widen(double2 a) { return a; }

// ConstructCurrentSolution's triangular solve (gmres.F90:441-445): y = H(0:L,0:L)^-1 g by one warp, lane i holding row
// i's right side: each y_i found is taken off all rows above it at once.  (One thread going over the L^2/2 products took
// 9.7 k clocks at L = 10.)
__global__ void __launch_bounds__(32) k_trisolve(Level L, const int *gate)
{
    pdl_wait();
    if (gate && *gate == 0) return;
    __shared__ double2 Hs[KMAX * KMAX];  // column j < n of the triangle at j * KMAX
    const int m = L.m, n = L.flags[F_L], lane = threadIdx.x;
    for (int j = 0; j < n; j++)
        if (lane <= j) Hs[lane + j * KMAX] = L.H[hix(lane, j, m)];
    double2 t = make_double2(0.0, 0.0), d = make_double2(1.0, 0.0);
    if (lane < n) t = L.H[hix(lane, m, m)];
    __syncwarp();
    if (lane < n) d = Hs[lane + lane * KMAX];
    const double den = d.x * d.x + d.y * d.y;
    for (int i = n - 1; i >= 0; i--) {
        double2 y = make_double2((t.x * d.x + t.y * d.y) / den, (t.y * d.x - t.x * d.y) / den);  // lane i's is row i's
        y.x = __shfl_sync(0xffffffffu, y.x, i);
        y.y = __shfl_sync(0xffffffffu, y.y, i);
        if (lane < i) {
            const double2 p = cmul_(Hs[lane + i * KMAX], y);
            t.x -= p.x;
            t.y -= p.y;
        } else if (lane == i) {
            L.y[i] = y;
        }
    }
}

// start of a cycle: H(0,m) = beta, H(1..m, m) = 0, krylov active (gmres.F90:172-185)
__global__ void k_cycle_start(Level L, const int *gate)
{
    pdl_wait();
    if (gate && *gate == 0) return;
    const int m = L.m;
    L.H[hix(0, m, m)] = make_double2(L.scal[S_BETA], 0.0);
    for (int i = 1; i <= m; i++) L.H[hix(i, m, m)] = make_double2(0.0, 0.0);
    L.flags[F_KRYLOV] = 1;
    L.flags[F_L] = 0;
}

// inner solve start: bn from nrm2; beta from the residual; exit when beta/bn < tol (gmres.F90:139-168)
__global__ void k_set_bn(Level L)
{
    pdl_wait();
    L.scal[S_BN] = sqrt(L.scal[S_NRM2]);
    L.flags[F_SOLVER] = L.scal[S_BN] < ZERO_THRESHOLD ? 0 : 1;
    L.flags[F_ITER] = 0;
    L.flags[F_KRYLOV] = L.flags[F_SOLVER];
    L.flags[F_L] = 0;
}
__global__ void k_set_beta(Level L, double tol)
{
    pdl_wait();
    if (L.flags[F_SOLVER] == 0) return;
    const double beta = sqrt(L.scal[S_NRM2]);
    L.scal[S_BETA] = beta;
    if (beta / L.scal[S_BN] < tol) {
        L.flags[F_SOLVER] = 0;
        L.flags[F_KRYLOV] = 0;
    }
}
__global__ void k_zero_level(Level L, unsigned *bar_inner)
{
    pdl_wait();
    const int n = (L.m + 1) * (L.m + 1);
    for (int i = threadIdx.x; i < n; i += blockDim.x) L.H[i] = make_double2(0.0, 0.0);
    if (threadIdx.x == 0) *L.bar = *bar_inner = 0u;  // a step that gave up at its barrier may have left arrivals
}

// restart (gmres.F90:369-376): beta = |g_m|, g <- inverse rotations of (0..0, g_m)
__global__ void k_restart_g(Level L)
{
    pdl_wait();
    const int m = L.m;
    L.scal[S_BETA] = cabs_(L.H[hix(m, m, m)]);
    for (int J = m - 1; J >= 0; J--) {
        L.H[hix(J, m, m)] = make_double2(0.0, 0.0);
        zrot1(L.H[hix(J, m, m)], L.H[hix(J + 1, m, m)], L.cs[J], make_double2(-L.sn[J].x, -L.sn[J].y));
    }
    L.flags[F_L] = m + 1;  // the restart residual combines m+1 basis vectors with column m
}

// ---- vector kernels ----------------------------------------------------------------------------
// out = a*x + b*y (real scalars), x, y, out may differ in type
template <typename CO, typename CX, typename CY>
__global__ void __launch_bounds__(kVT) k_axpby(CO *out, double a, const CX *x, double b, const CY *y, size_t N,
                                               const int *gate)
{
    pdl_wait();
    if (gate && *gate == 0) return;
    auto elem = [&](double2 xv, double2 yv) {
        double2 r = make_double2(a * xv.x, a * xv.y);
        if (y) {
            r.x += b * yv.x;
            r.y += b * yv.y;
        }
        return r;
    };
    // kILP independent elements per thread and iteration, loads first (out may alias x or y: every
    // element is still read before it is written, by the same thread)
    const size_t S = (size_t)gridDim.x * kVT;
    size_t i = blockIdx.x * (size_t)kVT + threadIdx.x;
    for (; i + (kILP - 1) * S < N; i += kILP * S) {
        double2 xv[kILP], yv[kILP];
#pragma unroll
        for (int u = 0; u < kILP; u++) {
            xv[u] = ld2(x, i + u * S);
            yv[u] = y ? ld2(y, i + u * S) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int u = 0; u < kILP; u++) st2(out, i + u * S, elem(xv[u], yv[u]));
    }
    for (; i < N; i += S) st2(out, i, elem(ld2(x, i), y ? ld2(y, i) : make_double2(0.0, 0.0)));
}
// v = w / scal[idx]
template <typename C>
__global__ void __launch_bounds__(kVT) k_scale_by(C *v, const C *w, const double *scal, int idx, size_t N,
                                                  const int *gate)
{
    pdl_wait();
    if (gate && *gate == 0) return;
    const double inv = 1.0 / scal[idx];
    for (size_t i = blockIdx.x * (size_t)kVT + threadIdx.x; i < N; i += (size_t)gridDim.x * kVT) {
        const double2 x = ld2(w, i);
        st2(v, i, make_double2(x.x * inv, x.y * inv));
    }
}
// out = a0*in0 + sum_{k < n} B_k coef_k, n = flags[F_L] (or Kfix >= 0)
template <typename CO, typename CB>
__global__ void __launch_bounds__(kVT) k_lincomb(CO *out, double a0, const CO *in0, const CB *__restrict__ Bm,
                                                 size_t ld, const double2 *__restrict__ coef, const int *nflag,
                                                 size_t N, const int *gate)
{
    pdl_wait();
    if (gate && *gate == 0) return;
    __shared__ double2 cs[KMAX + 1];
    const int n = *nflag;
    if (threadIdx.x < n) cs[threadIdx.x] = coef[threadIdx.x];
    __syncthreads();
    using W = typename Wide<CB>::T;
    constexpr int E = Wide<CB>::E;
    constexpr int KU = 4;  // basis words loaded together
    const size_t S = (size_t)gridDim.x * kVT, t0 = blockIdx.x * (size_t)kVT + threadIdx.x;
    const size_t Nw = wide_words<CB>(N, ld), ldw = ld / E;
    const W *__restrict__ Bw = reinterpret_cast<const W *>(Bm);
    size_t i = t0;
    for (; i < Nw; i += S) {
        double2 r[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
            r[e] = make_double2(0.0, 0.0);
            if (in0) {
                const double2 x = ld2(in0, i * E + e);
                r[e] = make_double2(a0 * x.x, a0 * x.y);
            }
        }
        int k = 0;
        for (; k + KU <= n; k += KU) {
            W v[KU];
#pragma unroll
            for (int q = 0; q < KU; q++) v[q] = Bw[(size_t)(k + q) * ldw + i];
#pragma unroll
            for (int q = 0; q < KU; q++)
#pragma unroll
                for (int e = 0; e < E; e++) {
                    const double2 b = widen(part_of(v[q], e)), c = cs[k + q];
                    r[e].x += b.x * c.x - b.y * c.y;
                    r[e].y += b.x * c.y + b.y * c.x;
                }
        }
        for (; k < n; k++) {
            const W v = Bw[(size_t)k * ldw + i];
#pragma unroll
            for (int e = 0; e < E; e++) {
                const double2 b = widen(part_of(v, e)), c = cs[k];
                r[e].x += b.x * c.x - b.y * c.y;
                r[e].y += b.x * c.y + b.y * c.x;
            }
        }
#pragma unroll
        for (int e = 0; e < E; e++) st2(out, i * E + e, r[e]);
    }
    for (i = Nw * E + t0; i < N; i += S) {
        double2 r = make_double2(0.0, 0.0);
        if (in0) {
            const double2 x = ld2(in0, i);
            r = make_double2(a0 * x.x, a0 * x.y);
        }
        for (int k = 0; k < n; k++) {
            const double2 v = ld2(Bm, (size_t)k * ld + i);
            r.x += v.x * cs[k].x - v.y * cs[k].y;
            r.y += v.x * cs[k].y + v.y * cs[k].x;
        }
        st2(out, i, r);
    }
}
// copy the g column into a coefficient vector (restart residual w = V g)
__global__ void k_copy_g(Level L)
{
    pdl_wait();
    const int m = L.m;
    for (int i = threadIdx.x; i <= m; i += blockDim.x) L.y[i] = L.H[hix(i, m, m)];
}

// a level's scalars and the operator's error word into pinned host memory: one launch before the host's wait, where three
// copies to pageable memory had cost about 20 us in each outer step of a small solve
struct Report {
    double scal[S_NSCAL];
    int err;
};
__global__ void k_report(Level L, const int *err, Report *out)
{
    pdl_wait();
    if (threadIdx.x < S_NSCAL) out->scal[threadIdx.x] = L.scal[threadIdx.x];
    if (threadIdx.x == 0) out->err = *err;
}

// SolveEquation helpers (ie_solver_module.F90:64-97); vectors are [c][cell], cell = z*NxNy + y*Nx + x
__global__ void k_rhs(double2 *rhs, const double2 *Ebkg, const double *post, size_t plane, int Nz)
{
    pdl_wait();
    const size_t n = 3 * plane * Nz;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int z = (int)((i / plane) % Nz);
        rhs[i] = make_double2(post[z] * Ebkg[i].x, post[z] * Ebkg[i].y);
    }
}
__global__ void k_scale_asig(double2 *out, const double2 *in, const double2 *asig, size_t cells, bool divide)
{
    pdl_wait();
    const size_t n = 3 * cells;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double2 a = asig[i % cells];
        const double2 v = in[i];
        if (divide) {
            const double den = a.x * a.x + a.y * a.y;
            out[i] = make_double2((v.x * a.x + v.y * a.y) / den, (v.y * a.x - v.x * a.y) / den);
        } else {
            out[i] = make_double2(v.x * a.x - v.y * a.y, v.x * a.y + v.y * a.x);
        }
    }
}

int vec_grid(size_t N)
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    const size_t need = (N + kVT - 1) / kVT;
    const size_t g = (size_t)sms * 4;
    return (int)(need < g ? need : g);
}
// blocks of the sweeps that end in a last-block reduction: two per SM and instance streamed as fast as
// four in the basis sweeps, and leave the last block half as many partial sums to add
int sweep_grid(size_t N)
{
    const int g = vec_grid(N);
    return g > 8 ? (g + 1) / 2 : g;
}

}  // namespace

// --------------------------------------------------------------------------------------------------
struct KrylovWork {
    size_t N = 0;
    int mo = 0, mi = 0, precision = -1;
    // outer (FP64)
    double2 *Vo = nullptr, *x = nullptr, *b = nullptr, *r0 = nullptr, *w = nullptr, *tmp = nullptr;
    void *Zo = nullptr;  // complex128 (plain) or complex64 (mixed)
    // inner
    void *Vi = nullptr, *ri = nullptr, *wi = nullptr, *vin = nullptr, *xin = nullptr;
    Level Lo, Li;
    // the inner GMRES cycle as CUDA graphs (fixed buffers vin -> xin; slot 0 starts at x0 = vin as the
    // reference does, slot 1 at x0 = x0in, the outer preconditioner hook's guess), captured on second use
    cudaGraphExec_t inner_exec[2] = {nullptr, nullptr};
    double inner_tol[2] = {-1.0, -1.0};
    int inner_uses[2] = {0, 0}, inner_graph_applies[2] = {0, 0}, inner_graph_launches[2] = {0, 0};
    bool inner_true_res[2] = {false, false};
    long long inner_gen[2] = {-1, -1};          // operator launch configuration baked into the graphs
    void *x0in = nullptr;                       // warm start of the inner cycle (inner precision)
    double2 *part = nullptr;  // partial sums of a sweep, two sets
    int nparts = 0;
    int *err = nullptr;       // the operator's device error word
    void *mem = nullptr;      // all device buffers
    Report *report = nullptr;  // pinned; allocated by the first solve of its own (a batch has one for all instances)
    std::vector<double> history;
    int applies64 = 0, applies32 = 0;
    int hook_steps = 0;  // outer steps preconditioned through the hook in the last solve
};

// Pieces of one allocation, 256 bytes apart: without a base only their total is counted.  (The 28 buffers of a solve, each
// allocated on its own, took 3-4 ms of a new operator's first solve.)
struct Slab {
    char *base = nullptr;
    size_t used = 0;
    template <typename T> void take(T *&p, size_t bytes)
    {
        p = base ? reinterpret_cast<T *>(base + used) : nullptr;
        used += (bytes + 255) / 256 * 256;
    }
};
static void place_level(Level &L, int m, Slab &s)
{
    L.m = m;
    s.take(L.H, sizeof(double2) * (m + 1) * (m + 1));
    s.take(L.cs, sizeof(double) * (m + 1));
    s.take(L.sn, sizeof(double2) * (m + 1));
    s.take(L.y, sizeof(double2) * (KMAX + 1));
    s.take(L.scal, sizeof(double) * S_NSCAL);
    s.take(L.flags, sizeof(int) * F_NFLAGS);
    s.take(L.counter, sizeof(unsigned));
    s.take(L.bar, sizeof(unsigned));
}

static void kw_free(KrylovWork *k)
{
    if (!k) return;
    for (int q = 0; q < 2; q++)
        if (k->inner_exec[q]) cudaGraphExecDestroy(k->inner_exec[q]);
    if (k->mem) cudaFree(k->mem);
    if (k->report) cudaFreeHost(k->report);
    delete k;
}

void krylov_free(IeOp *op)
{
    kw_free(reinterpret_cast<KrylovWork *>(op->krylov));
    op->krylov = nullptr;
}

// solver workspace for vectors of N complex: outer basis mo, inner basis mi
static int kw_alloc(KrylovWork *k, size_t N, int mo, int mi, int precision)
{
    k->N = N;
    k->mo = mo;
    k->mi = mi;
    k->precision = precision;
    const size_t e64 = sizeof(double2), ei = precision ? sizeof(float2) : sizeof(double2);
    k->nparts = sweep_grid(N);
    Slab s;
    for (int pass = 0; pass < 2; pass++) {
        // the levels first: they are zeroed
        s.used = 0;
        place_level(k->Lo, mo, s);
        place_level(k->Li, mi, s);
        const size_t state = s.used;
        s.take(k->Vo, e64 * N * (mo + 1));
        s.take(k->x, e64 * N);
        s.take(k->b, e64 * N);
        s.take(k->r0, e64 * N);
        s.take(k->w, e64 * N);
        s.take(k->tmp, e64 * N);
        s.take(k->Zo, ei * N * mo);
        s.take(k->Vi, ei * N * (mi + 1));
        s.take(k->ri, ei * N);
        s.take(k->wi, ei * N);
        s.take(k->vin, ei * N);
        s.take(k->xin, ei * N);
        s.take(k->x0in, ei * N);
        s.take(k->part, 2 * sizeof(double2) * (size_t)k->nparts * (KMAX + 1));
        if (pass) {
            G2_CUDA_CHECK(cudaMemset(s.base, 0, state));
        } else {
            G2_CUDA_CHECK(cudaMalloc(&k->mem, s.used));
            s.base = static_cast<char *>(k->mem);
        }
    }
    // the solver's kernels run on non-blocking streams, which are not ordered after the legacy stream
    G2_CUDA_CHECK(cudaStreamSynchronize(cudaStreamLegacy));
    return G2_OK;
}

static int krylov_alloc(IeOp *op, int mo, int mi, int precision)
{
    KrylovWork *k = reinterpret_cast<KrylovWork *>(op->krylov);
    if (k && k->mo == mo && k->mi == mi && k->precision == precision) return G2_OK;
    krylov_free(op);
    k = new KrylovWork();
    k->err = op->d_err;
    op->krylov = k;
    const int rc = kw_alloc(k, op->nvec(), mo, mi, precision);
    if (rc) krylov_free(op);  // a later call with the same sizes must not take it for a complete workspace
    return rc;
}

// ---- launch helpers ------------------------------------------------------------------------------
template <typename C>
static void norm2(KrylovWork *k, const C *w, double *nrm2, const int *g, cudaStream_t st)
{
    // kernels on one stream run one after another, so any level's counter serves
    g2_launch(k_norm2_fused<C>, k->nparts, kVT, 0, st, w, k->N, k->part, nrm2, k->Lo.counter, g); g2_count_launches(1);
}

// Arnoldi step j on level L with basis V (j + 1 columns) and vector w
template <typename C>
static int arnoldi_step1(KrylovWork *k, Level &L, C *V, int j, C *w, double tol, const int *gate, cudaStream_t st)
{
    Multi<C> mm{};
    mm.V[0] = V;
    mm.w[0] = w;
    mm.part[0] = k->part;
    mm.L[0] = L;
    mm.gate[0] = gate;
    return arnoldi_step(mm, 1, k->N, k->nparts, j, tol, k->err, st);
}
template <typename C> static int apply_prec(IeOp *op, const C *in, C *out, cudaStream_t st, const int *gate);
template <> int apply_prec<double2>(IeOp *op, const double2 *in, double2 *out, cudaStream_t st, const int *gate)
{
    return ie_apply_device64(op, in, out, st, gate);
}
template <> int apply_prec<float2>(IeOp *op, const float2 *in, float2 *out, cudaStream_t st, const int *gate)
{
    return ie_apply_device32(op, in, out, st, gate);
}

// Inner GMRES (seq_fgmres.F90:142-152 -> gmres.F90:110-213 with MaxIt = 1, x0 = b = v): x = M(v)
template <typename CI>
static int inner_solve(IeOp *op, KrylovWork *k, const CI *v, const CI *x0, CI *x, double tol, bool true_residual,
                       cudaStream_t st)
{
    Level &L = k->Li;
    const size_t N = k->N;
    const int g = vec_grid(N);
    CI *Vi = reinterpret_cast<CI *>(k->Vi), *ri = reinterpret_cast<CI *>(k->ri), *wi = reinterpret_cast<CI *>(k->wi);
    const int *solver = L.flags + F_SOLVER, *krylov = L.flags + F_KRYLOV;
    Starts<CI> s{};
    s.v[0] = v;
    s.x0[0] = x0;
    s.x[0] = x;
    s.r[0] = ri;
    s.V[0] = Vi;
    s.part[0] = k->part;
    s.L[0] = L;
    int rc = krylov_begin(s, 1, N, k->nparts, k->err, st);
    if (rc) return rc;
    rc = apply_prec<CI>(op, x0, ri, st, solver);
    if (rc) return rc;
    k->applies32 += sizeof(CI) == 8 ? 1 : 0;
    k->applies64 += sizeof(CI) == 16 ? 1 : 0;
    if ((rc = krylov_residual(s, 1, N, k->nparts, tol, k->err, st))) return rc;
    for (int j = 0; j < k->mi; j++) {
        CI *Vj = Vi + (size_t)j * N;
        rc = apply_prec<CI>(op, Vj, wi, st, krylov);
        if (rc) return rc;
        k->applies32 += sizeof(CI) == 8 ? 1 : 0;
        k->applies64 += sizeof(CI) == 16 ? 1 : 0;
        if ((rc = arnoldi_step1<CI>(k, L, Vi, j, wi, tol, krylov, st))) return rc;
    }
    // FinalActions -> ConstructCurrentSolution (gmres.F90:423-458): x = x0 + V y
    g2_launch(k_trisolve, 1, 32, 0, st, L, solver); g2_count_launches(1);
    g2_launch(k_lincomb<CI, CI>, g, kVT, 0, st, x, 1.0, x, Vi, N, L.y, L.flags + F_L, N, solver); g2_count_launches(1);
    if (true_residual) {  // gmres.F90:402-419, result unused by the outer solver
        rc = apply_prec<CI>(op, x, ri, st, solver);
        if (rc) return rc;
        k->applies32 += sizeof(CI) == 8 ? 1 : 0;
        k->applies64 += sizeof(CI) == 16 ? 1 : 0;
    }
    return G2_OK;
}

// inner solve vin -> xin (warm: starting at x0in); eager on first use, then captured once and replayed
template <typename CI>
static int inner_solve_fixed(IeOp *op, KrylovWork *k, double tol, bool true_res, bool warm, cudaStream_t st)
{
    const int q = warm ? 1 : 0;
    const CI *v = reinterpret_cast<const CI *>(k->vin);
    const CI *x0 = warm ? reinterpret_cast<const CI *>(k->x0in) : v;
    CI *x = reinterpret_cast<CI *>(k->xin);
    const char *ng = std::getenv("GIEM2G_NO_GRAPHS");
    const bool graphs = !(ng && ng[0] == '1');
    if (k->inner_exec[q] && (k->inner_tol[q] != tol || k->inner_true_res[q] != true_res ||
                             k->inner_gen[q] != op->config_gen)) {
        cudaGraphExecDestroy(k->inner_exec[q]);
        k->inner_exec[q] = nullptr;
        k->inner_uses[q] = 0;
    }
    auto credit = [&]() {
        g2_count_launches(k->inner_graph_launches[q]);
        if (sizeof(CI) == 8) k->applies32 += k->inner_graph_applies[q];
        else k->applies64 += k->inner_graph_applies[q];
    };
    if (k->inner_exec[q]) {
        G2_CUDA_CHECK(cudaGraphLaunch(k->inner_exec[q], st));
        credit();
        return G2_OK;
    }
    if (!graphs || k->inner_uses[q]++ == 0) return inner_solve<CI>(op, k, v, x0, x, tol, true_res, st);
    // capture: count what one cycle launches, then instantiate
    const int a32 = k->applies32, a64 = k->applies64;
    const long long l0 = g2_launch_total();
    cudaGraph_t graph = nullptr;
    G2_CUDA_CHECK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    int rc = inner_solve<CI>(op, k, v, x0, x, tol, true_res, st);
    cudaError_t ce = cudaStreamEndCapture(st, &graph);
    if (rc) return rc;
    if (ce != cudaSuccess) {
        g2_set_error(__FILE__, __LINE__, cudaGetErrorString(ce));
        return G2_ERR_CUDA;
    }
    k->inner_graph_applies[q] = (k->applies32 - a32) + (k->applies64 - a64);
    k->inner_graph_launches[q] = (int)(g2_launch_total() - l0);
    k->applies32 = a32;
    k->applies64 = a64;
    ce = cudaGraphInstantiate(&k->inner_exec[q], graph, 0);
    cudaGraphDestroy(graph);
    if (ce != cudaSuccess) {
        g2_set_error(__FILE__, __LINE__, cudaGetErrorString(ce));
        k->inner_exec[q] = nullptr;
        return G2_ERR_CUDA;
    }
    k->inner_tol[q] = tol;
    k->inner_true_res[q] = true_res;
    k->inner_gen[q] = op->config_gen;
    G2_CUDA_CHECK(cudaGraphLaunch(k->inner_exec[q], st));
    credit();
    return G2_OK;
}

template <typename CI>
static int outer_solve(IeOp *op, KrylovWork *k, const GIEM2G_FGMRES_CTL &ctl, GIEM2G_RESULT *info, cudaStream_t st)
{
    Level &L = k->Lo;
    const size_t N = k->N;
    const int g = vec_grid(N), M = k->mo;
    const double tol = ctl.misfit;
    const char *tr = std::getenv("GIEM2G_INNER_TRUE_RESIDUAL");
    const bool true_res = tr && tr[0] == '1';
    CI *Z = reinterpret_cast<CI *>(k->Zo);
    CI *vin = reinterpret_cast<CI *>(k->vin);
    if (!k->report) G2_CUDA_CHECK(cudaMallocHost(&k->report, sizeof(Report)));
    const double *h_scal = k->report->scal;
    auto pull = [&]() -> int {
        g2_launch(k_report, 1, 32, 0, st, L, k->err, k->report); g2_count_launches(1);
        G2_CUDA_CHECK(cudaStreamSynchronize(st));
        return k->report->err ? ie_check_device_error(op) : G2_OK;
    };
    k->history.clear();
    info->iterations = 0;
    info->bea = -1.0;
    info->be = -1.0;
    // gmres.F90:129-168
    g2_launch(k_zero_level, 1, 256, 0, st, L, k->Li.bar); g2_count_launches(1);
    norm2<double2>(k, k->b, L.scal + S_NRM2, nullptr, st);
    g2_launch(k_set_bn, 1, 1, 0, st, L); g2_count_launches(1);
    int rc = pull();
    if (rc) return rc;
    if (h_scal[S_BN] < ZERO_THRESHOLD) {
        cudaMemsetAsync(k->x, 0, sizeof(double2) * N, st);
        info->stat = 1;
        return G2_OK;
    }
    const double bn = h_scal[S_BN];
    rc = ie_apply_device64(op, k->x, k->r0, st);  // x holds x0
    if (rc) return rc;
    k->applies64++;
    g2_launch(k_axpby<double2, double2, double2>, g, kVT, 0, st, k->r0, 1.0, k->b, -1.0, k->r0, N, nullptr); g2_count_launches(1);
    g2_launch(k_axpby<double2, double2, double2>, g, kVT, 0, st, k->w, 1.0, k->r0, 0.0, (const double2 *)nullptr, N, nullptr); g2_count_launches(1);
    norm2<double2>(k, k->w, L.scal + S_NRM2, nullptr, st);
    g2_launch(k_set_beta, 1, 1, 0, st, L, tol); g2_count_launches(1);
    if ((rc = pull())) return rc;
    if (h_scal[S_BETA] / bn < tol) {
        info->stat = 1;
        info->be = h_scal[S_BETA] / bn;
        return G2_OK;
    }
    int iter = 0, L_used = 0;
    bool converged = false, hook_off = false;
    k->hook_steps = 0;
    double bea = -1.0;
    char msg[256];
    for (;;) {
        g2_launch(k_cycle_start, 1, 1, 0, st, L, nullptr); g2_count_launches(1);
        g2_launch(k_scale_by<double2>, g, kVT, 0, st, k->Vo, k->w, L.scal, S_BETA, N, nullptr); g2_count_launches(1);
        for (int j = 0; j < M; j++) {
            const double2 *Vj = k->Vo + (size_t)j * N;
            CI *Zj = Z + (size_t)j * N;
            // right preconditioner: Z_j = inner GMRES(V_j)  (gmres.F90:251, :491-506), through the fixed
            // buffers vin -> xin of the captured inner cycle.  With an outer preconditioner hook the hook's
            // output (complex128 in tmp) either starts the inner cycle (mode 1) or is Z_j itself (mode 2).
            bool hooked = false;
            if (op->precond_mode && !hook_off) {
                const int hr = op->precond_fn(op->precond_user, Vj, k->tmp, (long long)N, reinterpret_cast<void *>(st));
                if (hr == 0) hooked = true;
                else hook_off = true;
            }
            if (hooked && op->precond_mode == 2) {
                g2_launch(k_axpby<CI, double2, double2>, g, kVT, 0, st, Zj, 1.0, k->tmp, 0.0, (const double2 *)nullptr, N, nullptr); g2_count_launches(1);
            } else {
                g2_launch(k_axpby<CI, double2, double2>, g, kVT, 0, st, vin, 1.0, Vj, 0.0, (const double2 *)nullptr, N, nullptr); g2_count_launches(1);
                if (hooked) {
                    g2_launch(k_axpby<CI, double2, double2>, g, kVT, 0, st, reinterpret_cast<CI *>(k->x0in), 1.0, k->tmp, 0.0,
                                                                     (const double2 *)nullptr, N, nullptr); g2_count_launches(1);
                }
                if ((rc = inner_solve_fixed<CI>(op, k, tol, true_res, hooked, st))) return rc;
                g2_launch(k_axpby<CI, CI, CI>, g, kVT, 0, st, Zj, 1.0, reinterpret_cast<const CI *>(k->xin), 0.0, (const CI *)nullptr, N, nullptr); g2_count_launches(1);
            }
            if (sizeof(CI) == sizeof(double2)) {
                if ((rc = ie_apply_device64(op, reinterpret_cast<const double2 *>(Zj), k->w, st))) return rc;
            } else {
                g2_launch(k_axpby<double2, CI, CI>, g, kVT, 0, st, k->tmp, 1.0, Zj, 0.0, (const CI *)nullptr, N, nullptr); g2_count_launches(1);
                if ((rc = ie_apply_device64(op, k->tmp, k->w, st))) return rc;
            }
            k->applies64++;
            if ((rc = arnoldi_step1<double2>(k, L, k->Vo, j, k->w, tol, nullptr, st))) return rc;
            if ((rc = pull())) return rc;
            bea = h_scal[S_BEA];
            if (!std::isfinite(bea)) {
                g2_set_error_msg("FGMRES: non-finite Arnoldi misfit");
                return G2_ERR_NUMERIC;
            }
            // the hook must keep reducing the FP64 residual; otherwise the plain inner GMRES takes over
            if (hooked && !k->history.empty() && !(bea < kHookGain * k->history.back())) hook_off = true;
            if (hooked) k->hook_steps++;
            k->history.push_back(bea);
            info->iterations = (int)k->history.size();
            // ie_solver_module.F90:335-343 Information
            std::snprintf(msg, sizeof(msg), "FGMRES outer  iteration:%5d Arnoldy misfit: %10.3E", (int)k->history.size(), bea);
            g2_log(msg);
            L_used = j + 1;
            if (bea < tol) { converged = true; break; }
        }
        if (converged) break;
        iter++;
        if (iter >= ctl.fgmres_maxit) break;
        // PrepareRestart: x += Z y; w = V g' (gmres.F90:333-379)
        g2_launch(k_trisolve, 1, 32, 0, st, L, nullptr); g2_count_launches(1);
        g2_launch(k_lincomb<double2, CI>, g, kVT, 0, st, k->x, 1.0, k->x, Z, N, L.y, L.flags + F_L, N, nullptr); g2_count_launches(1);
        g2_launch(k_restart_g, 1, 1, 0, st, L); g2_count_launches(1);
        g2_launch(k_copy_g, 1, 64, 0, st, L); g2_count_launches(1);
        g2_launch(k_lincomb<double2, double2>, g, kVT, 0, st, k->w, 0.0, (const double2 *)nullptr, k->Vo, N, L.y,
                                                       L.flags + F_L, N, nullptr);
    }
    (void)L_used;
    // FinalActions (gmres.F90:382-421)
    g2_launch(k_trisolve, 1, 32, 0, st, L, nullptr); g2_count_launches(1);
    g2_launch(k_lincomb<double2, CI>, g, kVT, 0, st, k->x, 1.0, k->x, Z, N, L.y, L.flags + F_L, N, nullptr); g2_count_launches(1);
    if ((rc = ie_apply_device64(op, k->x, k->r0, st))) return rc;
    k->applies64++;
    g2_launch(k_axpby<double2, double2, double2>, g, kVT, 0, st, k->r0, 1.0, k->b, -1.0, k->r0, N, nullptr); g2_count_launches(1);
    norm2<double2>(k, k->r0, L.scal + S_NRM2, nullptr, st);
    if ((rc = pull())) return rc;
    const double be = std::sqrt(h_scal[S_NRM2]) / bn;
    info->iterations = (int)k->history.size();
    info->bea = bea;
    info->be = be;
    if (converged) info->stat = be >= tol ? 2 : 1;
    else info->stat = -1;
    return G2_OK;
}

int krylov_solve_device(IeOp *op, const double2 *d_Ebkg, double2 *d_Esol, const double2 *d_E0,
                        const GIEM2G_FGMRES_CTL &ctl, GIEM2G_RESULT *info)
{
    if (ctl.fgmres_buf < 1 || ctl.gmres_buf < 1 || ctl.fgmres_buf > KMAX - 1 || ctl.gmres_buf > KMAX - 1) {
        g2_set_error_msg("FGMRES buffer sizes must be in [1, 31]");
        return G2_ERR_UNSUPPORTED;
    }
    if (ctl.precision < 0 || ctl.precision > 1) return G2_ERR_ARG;
    int rc = krylov_alloc(op, ctl.fgmres_buf, ctl.gmres_buf, ctl.precision);
    if (rc) return rc;
    KrylovWork *k = reinterpret_cast<KrylovWork *>(op->krylov);
    cudaStream_t st = op->stream;
    const size_t cells = op->cells();
    const int g = vec_grid(k->N);
    k->applies32 = k->applies64 = 0;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, st);
    // SolveEquation (ie_solver_module.F90:62-80): rhs = sqrt(Re sb) E_bkg; guess = E0/a or rhs
    g2_launch(k_rhs, g, 256, 0, st, k->b, d_Ebkg, op->d_post64, (size_t)op->Nx * op->Ny, op->Nz); g2_count_launches(1);
    if (d_E0) {
        g2_launch(k_scale_asig, g, 256, 0, st, k->x, d_E0, op->d_asig64, cells, true);
        g2_count_launches(1);
    } else {
        cudaMemcpyAsync(k->x, k->b, sizeof(double2) * k->N, cudaMemcpyDeviceToDevice, st);
    }
    if (ctl.precision == 0) rc = outer_solve<double2>(op, k, ctl, info, st);
    else rc = outer_solve<float2>(op, k, ctl, info, st);
    if (rc) return rc;
    // Esol = a * chi (ie_solver_module.F90:85-97)
    g2_launch(k_scale_asig, g, 256, 0, st, d_Esol, k->x, op->d_asig64, cells, false); g2_count_launches(1);
    cudaEventRecord(e1, st);
    g2_launch(k_report, 1, 32, 0, st, k->Lo, k->err, k->report); g2_count_launches(1);
    G2_CUDA_CHECK(cudaStreamSynchronize(st));
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    info->applies_fp64 = k->applies64;
    info->applies_fp32 = k->applies32;
    info->precond_steps = k->hook_steps;
    info->device_ms = ms;
    op->mult_num += k->applies64 + k->applies32;
    op->apply_seconds += ms * 1e-3;
    return k->report->err ? ie_check_device_error(op) : G2_OK;
}

int krylov_history(IeOp *op, double *out, int max_len)
{
    KrylovWork *k = reinterpret_cast<KrylovWork *>(op->krylov);
    if (!k) return 0;
    const int n = (int)k->history.size() < max_len ? (int)k->history.size() : max_len;
    for (int i = 0; i < n; i++) out[i] = k->history[i];
    return n;
}

// ==================================================================================================
// Batched solves (several frequencies and both polarisations): n independent instances, each a full
// nested FGMRES with its own workspace, advanced in lockstep on one stream.  Per outer step the host
// launches every active instance's work, replays ONE captured inner cycle for all instances and reads
// all instances' scalars with one synchronisation.  Consecutive instances of the same operator form
// pairs whose complex64 applies share every tensor read (ie_apply_pair32).  Each instance follows
// the operations of the single solve, so its iteration count and status are those of a solve on its own; its
// sums may be split over fewer blocks (arnoldi.cu), a difference of rounding.  Converged instances are masked: their inner-cycle kernels are gated off through a
// device flag and the host stops launching their outer work.
struct BatchGroup {
    IeOp *op = nullptr;
    int first = 0, n = 0;  // instances first .. first+n-1 (n = 1 or 2)
};

struct BatchWork {
    int n = 0, mo = 0, mi = 0, precision = -1;
    std::vector<IeOp *> ops;
    std::vector<KrylovWork *> k;
    std::vector<BatchGroup> groups;
    std::vector<int> h_active;  // instances still running (each mask has its own captured inner cycle)
    double2 *d_stage = nullptr;  // host-array solves: E_bkg[n] then E_sol[n] (complex128)
    // pinned host copies of the outer levels' scalars and flags, two slots (outer step j uses slot j % 2),
    // each completed by its own event
    void *h_pin = nullptr;
    cudaEvent_t ev_pull[2] = {nullptr, nullptr};
    cudaStream_t st = nullptr;
    // One captured inner cycle per mask of active instances: a solve changes the mask as instances
    // converge, and the next solve starts from all-active again, so the graphs are kept, not re-captured.
    struct InnerGraph {
        std::vector<int> mask;
        cudaGraphExec_t exec = nullptr;
        int uses = 0, launches = 0;
        std::vector<int> applies;
    };
    std::vector<InnerGraph> graphs;
    double inner_tol = -1.0;
    std::vector<long long> cv;  // operators' configuration generations the graphs were captured with
    std::vector<std::vector<double>> history;
};

static void batch_destroy(BatchWork *b)
{
    if (!b) return;
    if (b->st) cudaStreamSynchronize(b->st);
    for (auto &gr : b->graphs)
        if (gr.exec) cudaGraphExecDestroy(gr.exec);
    for (KrylovWork *k : b->k) kw_free(k);
    if (b->h_pin) cudaFreeHost(b->h_pin);
    for (cudaEvent_t e : b->ev_pull)
        if (e) cudaEventDestroy(e);
    if (b->d_stage) cudaFree(b->d_stage);
    delete b;
}

int batch_create(IeOp *const *ops, int n, int mo, int mi, int precision, void **out)
{
    *out = nullptr;
    if (n < 1) return G2_ERR_ARG;
    if (mo < 1 || mi < 1 || mo > KMAX - 1 || mi > KMAX - 1) {
        g2_set_error_msg("FGMRES buffer sizes must be in [1, 31]");
        return G2_ERR_UNSUPPORTED;
    }
    if (precision < 0 || precision > 1) return G2_ERR_ARG;
    BatchWork *b = new BatchWork();
    b->n = n;
    b->mo = mo;
    b->mi = mi;
    b->precision = precision;
    b->st = ops[0]->stream;
    for (int i = 0; i < n; i++) {
        if (!ops[i]) { batch_destroy(b); return G2_ERR_ARG; }
        b->ops.push_back(ops[i]);
        KrylovWork *k = new KrylovWork();
        k->err = ops[i]->d_err;
        b->k.push_back(k);
        const int rc = kw_alloc(k, ops[i]->nvec(), mo, mi, precision);
        if (rc) { batch_destroy(b); return rc; }
    }
    for (int i = 0; i < n;) {
        BatchGroup g;
        g.op = ops[i];
        g.first = i;
        g.n = (i + 1 < n && ops[i + 1] == ops[i]) ? 2 : 1;
        b->groups.push_back(g);
        i += g.n;
    }
    b->h_active.assign(n, 1);
    b->history.resize(n);
    *out = b;
    return G2_OK;
}

void batch_free(void *h) { batch_destroy(reinterpret_cast<BatchWork *>(h)); }

int batch_history(void *h, int i, double *out, int max_len)
{
    BatchWork *b = reinterpret_cast<BatchWork *>(h);
    if (!b || i < 0 || i >= b->n) return 0;
    const int m = (int)b->history[i].size() < max_len ? (int)b->history[i].size() : max_len;
    for (int j = 0; j < m; j++) out[j] = b->history[i][j];
    return m;
}

// applies of the inner level: in_i -> out_i for every instance, paired where two instances share an
// operator (complex64); flag selects the gate of the single applies (F_SOLVER or F_KRYLOV)
template <typename CI, typename FIn, typename FOut>
static int batch_apply(BatchWork *b, FIn in, FOut out, int flag, cudaStream_t st, const BatchGroup *only = nullptr)
{
    for (const BatchGroup &g : b->groups) {
        if (only && &g != only) continue;
        const bool both = g.n == 2 && b->h_active[g.first] && b->h_active[g.first + 1];
        if (both && sizeof(CI) == sizeof(float2)) {
            float2 *U1 = nullptr, *Uh = nullptr;
            int rc = ie_pair_scratch(g.op, &U1, &Uh);
            if (rc) return rc;
            rc = ie_apply_pair32(g.op, reinterpret_cast<const float2 *>(in(g.first)),
                                 reinterpret_cast<const float2 *>(in(g.first + 1)),
                                 reinterpret_cast<float2 *>(out(g.first)), reinterpret_cast<float2 *>(out(g.first + 1)),
                                 st, U1, Uh);
            if (rc == G2_OK) {
                b->k[g.first]->applies32++;
                b->k[g.first + 1]->applies32++;
                continue;
            }
            if (rc != G2_ERR_UNSUPPORTED) return rc;
        }
        for (int i = g.first; i < g.first + g.n; i++) {
            if (!b->h_active[i]) continue;
            const int rc = apply_prec<CI>(g.op, in(i), out(i), st, b->k[i]->Li.flags + flag);
            if (rc) return rc;
            if (sizeof(CI) == sizeof(float2)) b->k[i]->applies32++;
            else b->k[i]->applies64++;
        }
    }
    return G2_OK;
}

// one inner GMRES cycle (x0 = b = v) for every instance: the lockstep form of inner_solve
template <typename CI>
static int batch_inner(BatchWork *b, double tol, cudaStream_t st)
{
    const int n = b->n;
    // f on runs of up to KMI active instances of one vector length
    auto starts_of = [&](auto f) -> int {
        std::vector<int> act;
        for (int i = 0; i < n; i++)
            if (b->h_active[i]) act.push_back(i);
        for (size_t c = 0; c < act.size();) {
            KrylovWork *k0 = b->k[act[c]];
            Starts<CI> s{};
            int q = 0;
            for (; c < act.size() && q < KMI; c++, q++) {
                KrylovWork *k = b->k[act[c]];
                if (k->N != k0->N || k->nparts != k0->nparts) break;
                s.v[q] = s.x0[q] = reinterpret_cast<const CI *>(k->vin);
                s.x[q] = reinterpret_cast<CI *>(k->xin);
                s.r[q] = reinterpret_cast<CI *>(k->ri);
                s.V[q] = reinterpret_cast<CI *>(k->Vi);
                s.part[q] = k->part;
                s.L[q] = k->Li;
                // a cycle enqueued after its instance converged (one outer step ahead of the host, see batch_outer)
                // does nothing; masked instances launch nothing, as each mask has its own captured cycle
                s.go[q] = k->Lo.flags + F_KRYLOV;
            }
            if (const int r = f(s, q, k0)) return r;
        }
        return G2_OK;
    };
    int rc = starts_of([&](const Starts<CI> &s, int q, KrylovWork *k) { return krylov_begin(s, q, k->N, k->nparts, k->err, st); });
    if (rc) return rc;
    auto vin = [&](int i) { return reinterpret_cast<const CI *>(b->k[i]->vin); };
    auto ri = [&](int i) { return reinterpret_cast<CI *>(b->k[i]->ri); };
    rc = batch_apply<CI>(b, vin, ri, F_SOLVER, st);
    if (rc) return rc;
    rc = starts_of([&](const Starts<CI> &s, int q, KrylovWork *k) {
        return krylov_residual(s, q, k->N, k->nparts, tol, k->err, st);
    });
    if (rc) return rc;
    // Arnoldi step j of the active instances in `act`: runs of up to KMI instances with the same vector length
    // share each launch (each instance keeps its own blocks, partials and gates)
    auto arnoldi_of = [&](const std::vector<int> &act, int j) -> int {
        for (size_t c = 0; c < act.size();) {
            KrylovWork *k0 = b->k[act[c]];
            size_t e = c + 1;
            while (e < act.size() && e - c < (size_t)KMI && b->k[act[e]]->N == k0->N && b->k[act[e]]->nparts == k0->nparts)
                e++;
            if (e - c == 1) {
                Level &L = k0->Li;
                CI *Vi = reinterpret_cast<CI *>(k0->Vi);
                const int r = arnoldi_step1<CI>(k0, L, Vi, j, reinterpret_cast<CI *>(k0->wi), tol, L.flags + F_KRYLOV, st);
                if (r) return r;
            } else {
                Multi<CI> mm{};
                for (size_t q = 0; q < e - c; q++) {
                    KrylovWork *k = b->k[act[c + q]];
                    mm.V[q] = reinterpret_cast<CI *>(k->Vi);
                    mm.w[q] = reinterpret_cast<CI *>(k->wi);
                    mm.part[q] = k->part;
                    mm.L[q] = k->Li;
                    mm.gate[q] = k->Li.flags + F_KRYLOV;
                }
                const int r = arnoldi_step(mm, (int)(e - c), k0->N, k0->nparts, j, tol, k0->err, st);
                if (r) return r;
            }
            c = e;
        }
        return G2_OK;
    };
    // Each operator group (one frequency's polarisations) runs its apply and then its Arnoldi step before the
    // next group's apply, so the group's fresh w is still in L2 when its Gram-Schmidt reads it (with all
    // applies first, a 16-instance sweep re-read every w from DRAM).  Per instance the sequence of kernels is
    // unchanged.
    for (int j = 0; j < b->mi; j++) {
        auto vj = [&](int i) { return reinterpret_cast<const CI *>(b->k[i]->Vi) + (size_t)j * b->k[i]->N; };
        auto wi = [&](int i) { return reinterpret_cast<CI *>(b->k[i]->wi); };
        for (const BatchGroup &g : b->groups) {
            std::vector<int> act;
            for (int i = g.first; i < g.first + g.n; i++)
                if (b->h_active[i]) act.push_back(i);
            if (act.empty()) continue;
            if ((rc = batch_apply<CI>(b, vj, wi, F_KRYLOV, st, &g))) return rc;
            if ((rc = arnoldi_of(act, j))) return rc;
        }
    }
    for (int i = 0; i < n; i++) {
        if (!b->h_active[i]) continue;
        KrylovWork *k = b->k[i];
        Level &L = k->Li;
        const int g = vec_grid(k->N);
        const int *solver = L.flags + F_SOLVER;
        CI *x = reinterpret_cast<CI *>(k->xin);
        g2_launch(k_trisolve, 1, 32, 0, st, L, solver); g2_count_launches(1);
        g2_launch(k_lincomb<CI, CI>, g, kVT, 0, st, x, 1.0, x, reinterpret_cast<const CI *>(k->Vi), k->N, L.y, L.flags + F_L,
                                             k->N, solver); g2_count_launches(1);
    }
    return G2_OK;
}

// the inner cycle of all instances: eager on first use, then one captured graph replayed
template <typename CI>
static int batch_inner_fixed(BatchWork *b, double tol, cudaStream_t st)
{
    std::vector<long long> cv;
    for (IeOp *op : b->ops) cv.push_back(op->config_gen);
    const char *ng = std::getenv("GIEM2G_NO_GRAPHS");
    const bool use_graphs = !(ng && ng[0] == '1');
    if (b->inner_tol != tol || b->cv != cv) {  // the captured arguments are stale: drop every graph
        for (auto &gr : b->graphs)
            if (gr.exec) cudaGraphExecDestroy(gr.exec);
        b->graphs.clear();
        b->inner_tol = tol;
        b->cv = cv;
    }
    BatchWork::InnerGraph *gr = nullptr;
    for (auto &e : b->graphs)
        if (e.mask == b->h_active) gr = &e;
    if (!gr) {
        constexpr size_t kMaxGraphs = 32;
        if (b->graphs.size() >= kMaxGraphs) {  // oldest first
            if (b->graphs.front().exec) cudaGraphExecDestroy(b->graphs.front().exec);
            b->graphs.erase(b->graphs.begin());
        }
        b->graphs.emplace_back();
        gr = &b->graphs.back();
        gr->mask = b->h_active;
        gr->applies.assign(b->n, 0);
    }
    auto credit = [&]() {
        g2_count_launches(gr->launches);
        for (int i = 0; i < b->n; i++) {
            if (sizeof(CI) == sizeof(float2)) b->k[i]->applies32 += gr->applies[i];
            else b->k[i]->applies64 += gr->applies[i];
        }
    };
    if (gr->exec) {
        G2_CUDA_CHECK(cudaGraphLaunch(gr->exec, st));
        credit();
        return G2_OK;
    }
    // first use of a mask runs eagerly (it may allocate pair scratch, which a capture cannot)
    if (!use_graphs || gr->uses++ == 0) return batch_inner<CI>(b, tol, st);
    std::vector<int> a0(b->n);
    for (int i = 0; i < b->n; i++) a0[i] = b->k[i]->applies32 + b->k[i]->applies64;
    const long long l0 = g2_launch_total();
    cudaGraph_t graph = nullptr;
    G2_CUDA_CHECK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    int rc = batch_inner<CI>(b, tol, st);
    cudaError_t ce = cudaStreamEndCapture(st, &graph);
    if (rc) return rc;
    if (ce != cudaSuccess) {
        g2_set_error(__FILE__, __LINE__, cudaGetErrorString(ce));
        return G2_ERR_CUDA;
    }
    gr->launches = (int)(g2_launch_total() - l0);
    for (int i = 0; i < b->n; i++) {
        KrylovWork *k = b->k[i];
        gr->applies[i] = k->applies32 + k->applies64 - a0[i];
        if (sizeof(CI) == sizeof(float2)) k->applies32 -= gr->applies[i];
        else k->applies64 -= gr->applies[i];
    }
    ce = cudaGraphInstantiate(&gr->exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ce != cudaSuccess) {
        g2_set_error(__FILE__, __LINE__, cudaGetErrorString(ce));
        gr->exec = nullptr;
        return G2_ERR_CUDA;
    }
    G2_CUDA_CHECK(cudaGraphLaunch(gr->exec, st));
    credit();
    return G2_OK;
}

// per-instance host copies of the outer level's scalars and flags, one synchronisation for all
struct BatchScal {
    double s[S_NSCAL];
    int f[F_NFLAGS];
};
// Copies of the outer level's scalars and flags of instances `which` into pinned slot `slot` (pageable
// destinations made every such read a staged, blocking copy), completed by the slot's event.
static int batch_pull_start(BatchWork *b, const std::vector<int> &which, int slot, cudaStream_t st)
{
    if (!b->h_pin) {
        G2_CUDA_CHECK(cudaMallocHost(&b->h_pin, 2 * sizeof(BatchScal) * b->n));
        for (cudaEvent_t &e : b->ev_pull) G2_CUDA_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    BatchScal *h = reinterpret_cast<BatchScal *>(b->h_pin) + (size_t)slot * b->n;
    for (int i : which) {
        G2_CUDA_CHECK(cudaMemcpyAsync(h[i].s, b->k[i]->Lo.scal, sizeof(h[i].s), cudaMemcpyDeviceToHost, st));
        G2_CUDA_CHECK(cudaMemcpyAsync(h[i].f, b->k[i]->Lo.flags, sizeof(h[i].f), cudaMemcpyDeviceToHost, st));
    }
    G2_CUDA_CHECK(cudaEventRecord(b->ev_pull[slot], st));
    return G2_OK;
}
static int batch_pull_finish(BatchWork *b, const std::vector<int> &which, int slot, std::vector<BatchScal> &h)
{
    G2_CUDA_CHECK(cudaEventSynchronize(b->ev_pull[slot]));
    const BatchScal *p = reinterpret_cast<const BatchScal *>(b->h_pin) + (size_t)slot * b->n;
    for (int i : which) h[i] = p[i];
    return G2_OK;
}
static std::vector<int> active_list(const BatchWork *b)
{
    std::vector<int> a;
    for (int i = 0; i < b->n; i++)
        if (b->h_active[i]) a.push_back(i);
    return a;
}
// per-instance host copies of the active instances' scalars and flags, one synchronisation for all
static int batch_pull(BatchWork *b, std::vector<BatchScal> &h, cudaStream_t st)
{
    const std::vector<int> act = active_list(b);
    int rc = batch_pull_start(b, act, 0, st);
    if (!rc) rc = batch_pull_finish(b, act, 0, h);
    if (rc) return rc;
    for (IeOp *op : b->ops) {
        const int e = ie_check_device_error(op);
        if (e) return e;
    }
    return G2_OK;
}

// The same copies into pinned slot `slot` without waiting, so the host can enqueue more work before it waits
// (batch_outer's outer step j + 1).
static int batch_pull_async(BatchWork *b, int slot, cudaStream_t st)
{
    return batch_pull_start(b, active_list(b), slot, st);
}
static int batch_pull_wait(BatchWork *b, int slot, std::vector<BatchScal> &h)
{
    return batch_pull_finish(b, active_list(b), slot, h);
}

// FinalActions of instance i (gmres.F90:382-421) after the host learned that it stops
template <typename CI>
static void batch_final_launch(BatchWork *b, int i, cudaStream_t st, int &rc)
{
    KrylovWork *k = b->k[i];
    Level &L = k->Lo;
    const int g = vec_grid(k->N);
    CI *Z = reinterpret_cast<CI *>(k->Zo);
    g2_launch(k_trisolve, 1, 32, 0, st, L, nullptr); g2_count_launches(1);
    g2_launch(k_lincomb<double2, CI>, g, kVT, 0, st, k->x, 1.0, k->x, Z, k->N, L.y, L.flags + F_L, k->N, nullptr); g2_count_launches(1);
    if ((rc = ie_apply_device64(b->ops[i], k->x, k->r0, st))) return;
    k->applies64++;
    g2_launch(k_axpby<double2, double2, double2>, g, kVT, 0, st, k->r0, 1.0, k->b, -1.0, k->r0, k->N, nullptr); g2_count_launches(1);
    norm2<double2>(k, k->r0, L.scal + S_NRM2, nullptr, st);
}

template <typename CI>
static int batch_outer(BatchWork *b, const GIEM2G_FGMRES_CTL &ctl, GIEM2G_RESULT *info, cudaStream_t st)
{
    const int n = b->n, M = b->mo;
    const double tol = ctl.misfit;
    std::vector<BatchScal> h(n);
    std::vector<double> bn(n, 0.0), bea(n, -1.0);
    std::vector<int> iter(n, 0), converged(n, 0), finishing(n, 0);
    int rc = G2_OK;
    char msg[256];
    for (int i = 0; i < n; i++) {
        b->history[i].clear();
        b->h_active[i] = 1;
        info[i].iterations = 0;
        info[i].bea = -1.0;
        info[i].be = -1.0;
        info[i].stat = -1;
    }
    // gmres.F90:129-168 for every instance, with one host read: the initial residual is gated on the device
    // flag k_set_bn clears for a zero right-hand side, so the host need not read ||b|| before launching it
    for (int i = 0; i < n; i++) {
        KrylovWork *k = b->k[i];
        const int g = vec_grid(k->N);
        const int *solver = k->Lo.flags + F_SOLVER;
        g2_launch(k_zero_level, 1, 256, 0, st, k->Lo, k->Li.bar); g2_count_launches(1);
        norm2<double2>(k, k->b, k->Lo.scal + S_NRM2, nullptr, st);
        g2_launch(k_set_bn, 1, 1, 0, st, k->Lo); g2_count_launches(1);
        if ((rc = ie_apply_device64(b->ops[i], k->x, k->r0, st, solver))) return rc;
        g2_launch(k_axpby<double2, double2, double2>, g, kVT, 0, st, k->r0, 1.0, k->b, -1.0, k->r0, k->N, solver); g2_count_launches(1);
        g2_launch(k_axpby<double2, double2, double2>, g, kVT, 0, st, k->w, 1.0, k->r0, 0.0, (const double2 *)nullptr, k->N, solver); g2_count_launches(1);
        norm2<double2>(k, k->w, k->Lo.scal + S_NRM2, solver, st);
        g2_launch(k_set_beta, 1, 1, 0, st, k->Lo, tol); g2_count_launches(1);
    }
    if ((rc = batch_pull(b, h, st))) return rc;
    for (int i = 0; i < n; i++) {
        KrylovWork *k = b->k[i];
        bn[i] = h[i].s[S_BN];
        if (bn[i] < ZERO_THRESHOLD) {
            cudaMemsetAsync(k->x, 0, sizeof(double2) * k->N, st);
            info[i].stat = 1;
            b->h_active[i] = 0;
            continue;
        }
        k->applies64++;
    }
    for (int i = 0; i < n; i++) {
        if (!b->h_active[i]) continue;
        if (h[i].s[S_BETA] / bn[i] < tol) {
            info[i].stat = 1;
            info[i].be = h[i].s[S_BETA] / bn[i];
            b->h_active[i] = 0;
        }
    }
    auto any_active = [&]() {
        for (int i = 0; i < n; i++)
            if (b->h_active[i]) return true;
        return false;
    };
    while (any_active()) {
        for (int i = 0; i < n; i++) {
            if (!b->h_active[i]) continue;
            KrylovWork *k = b->k[i];
            g2_launch(k_cycle_start, 1, 1, 0, st, k->Lo, nullptr); g2_count_launches(1);
            g2_launch(k_scale_by<double2>, vec_grid(k->N), kVT, 0, st, k->Vo, k->w, k->Lo.scal, S_BETA, k->N, nullptr); g2_count_launches(1);
        }
        bool cycle_done = false;
        // Outer step j of every active instance.  Its kernels are gated by the instance's outer Krylov flag,
        // which the Arnoldi tail of step j - 1 clears when the instance converged (or its cycle ended): step
        // j + 1 is enqueued before the host reads step j's misfits, so the GPU does not wait for the host
        // between steps, and an instance that converged at step j does nothing in step j + 1.  The arithmetic
        // of the instances that go on is unchanged.
        auto enqueue_step = [&](int j) -> int {
            for (int i = 0; i < n; i++) {
                if (!b->h_active[i]) continue;
                KrylovWork *k = b->k[i];
                const int *go = k->Lo.flags + F_KRYLOV;
                g2_launch(k_axpby<CI, double2, double2>, vec_grid(k->N), kVT, 0, st, 
                    reinterpret_cast<CI *>(k->vin), 1.0, k->Vo + (size_t)j * k->N, 0.0, (const double2 *)nullptr, k->N,
                    go); g2_count_launches(1);
            }
            int r = batch_inner_fixed<CI>(b, tol, st);
            if (r) return r;
            // per operator group: the FP64 applies, then the group's outer Arnoldi step (w still in L2), with
            // the group's instances sharing each CGS and scaling launch
            for (const BatchGroup &gr : b->groups) {
                std::vector<int> act;
                for (int i = gr.first; i < gr.first + gr.n; i++) {
                    if (!b->h_active[i]) continue;
                    act.push_back(i);
                    KrylovWork *k = b->k[i];
                    const int g = vec_grid(k->N);
                    const int *go = k->Lo.flags + F_KRYLOV;
                    CI *Zj = reinterpret_cast<CI *>(k->Zo) + (size_t)j * k->N;
                    g2_launch(k_axpby<CI, CI, CI>, g, kVT, 0, st, Zj, 1.0, reinterpret_cast<const CI *>(k->xin), 0.0, (const CI *)nullptr, k->N, go); g2_count_launches(1);
                    if (sizeof(CI) == sizeof(double2)) {
                        if ((r = ie_apply_device64(b->ops[i], reinterpret_cast<const double2 *>(Zj), k->w, st, go))) return r;
                    } else {
                        g2_launch(k_axpby<double2, CI, CI>, g, kVT, 0, st, k->tmp, 1.0, Zj, 0.0, (const CI *)nullptr, k->N, go); g2_count_launches(1);
                        if ((r = ie_apply_device64(b->ops[i], k->tmp, k->w, st, go))) return r;
                    }
                }
                if (act.size() == 1) {
                    KrylovWork *k0 = b->k[act[0]];
                    const int *go = k0->Lo.flags + F_KRYLOV;
                    if ((r = arnoldi_step1<double2>(k0, k0->Lo, k0->Vo, j, k0->w, tol, go, st))) return r;
                } else if (act.size() == 2 && b->k[act[0]]->N == b->k[act[1]]->N &&
                           b->k[act[0]]->nparts == b->k[act[1]]->nparts) {
                    Multi<double2> mm{};
                    for (size_t q = 0; q < act.size(); q++) {
                        KrylovWork *k = b->k[act[q]];
                        mm.V[q] = k->Vo;
                        mm.w[q] = k->w;
                        mm.part[q] = k->part;
                        mm.L[q] = k->Lo;
                        mm.gate[q] = k->Lo.flags + F_KRYLOV;
                    }
                    KrylovWork *k0 = b->k[act[0]];
                    if ((r = arnoldi_step(mm, 2, k0->N, k0->nparts, j, tol, k0->err, st))) return r;
                } else {
                    for (int i : act) {
                        KrylovWork *k = b->k[i];
                        const int *go = k->Lo.flags + F_KRYLOV;
                        if ((r = arnoldi_step1<double2>(k, k->Lo, k->Vo, j, k->w, tol, go, st))) return r;
                    }
                }
            }
            return G2_OK;
        };
        // Running ahead is skipped when an instance is expected to converge at step j (its last misfit times
        // its last reduction factor within kAheadMargin of the tolerance): a step enqueued after that keeps the
        // pair's shared complex64 applies for an instance that would otherwise run its single applies.
        auto near_tol = [&]() {
            constexpr double kAheadMargin = 4.0;
            for (int i = 0; i < n; i++) {
                if (!b->h_active[i] || b->history[i].empty()) continue;
                const std::vector<double> &hs = b->history[i];
                const double last = hs.back();
                const double r = hs.size() > 1 && hs[hs.size() - 2] > 0.0 ? std::min(1.0, last / hs[hs.size() - 2]) : 1.0;
                if (last * r < kAheadMargin * tol) return true;
            }
            return false;
        };
        bool ahead = false;  // step j was enqueued ahead, during step j - 1
        for (int j = 0; j < M && !cycle_done; j++) {
            if (!ahead && (rc = enqueue_step(j))) return rc;
            if ((rc = batch_pull_async(b, j & 1, st))) return rc;
            ahead = j + 1 < M && !near_tol();
            if (ahead && (rc = enqueue_step(j + 1))) return rc;
            if ((rc = batch_pull_wait(b, j & 1, h))) return rc;
            // an instance still active here ran step j (it had not converged at step j - 1)
            for (int i = 0; i < n; i++)
                if (b->h_active[i]) b->k[i]->applies64++;
            for (int i = 0; i < n; i++) {
                if (!b->h_active[i]) continue;
                bea[i] = h[i].s[S_BEA];
                if (!std::isfinite(bea[i])) {
                    g2_set_error_msg("FGMRES: non-finite Arnoldi misfit");
                    return G2_ERR_NUMERIC;
                }
                b->history[i].push_back(bea[i]);
                std::snprintf(msg, sizeof(msg), "FGMRES outer  iteration:%5d Arnoldy misfit: %10.3E  (instance %d)",
                              (int)b->history[i].size(), bea[i], i);
                g2_log(msg);
                if (bea[i] < tol) {
                    converged[i] = 1;
                    finishing[i] = 1;
                    b->h_active[i] = 0;
                }
            }
            if (!any_active()) cycle_done = true;
        }
        // end of the cycle for the instances still running: restart or give up (gmres.F90:186-212)
        for (int i = 0; i < n; i++) {
            if (!b->h_active[i]) continue;
            KrylovWork *k = b->k[i];
            const int g = vec_grid(k->N);
            iter[i]++;
            if (iter[i] >= ctl.fgmres_maxit) {
                finishing[i] = 1;
                b->h_active[i] = 0;
                continue;
            }
            g2_launch(k_trisolve, 1, 32, 0, st, k->Lo, nullptr); g2_count_launches(1);
            g2_launch(k_lincomb<double2, CI>, g, kVT, 0, st, k->x, 1.0, k->x, reinterpret_cast<const CI *>(k->Zo), k->N,
                                                      k->Lo.y, k->Lo.flags + F_L, k->N, nullptr); g2_count_launches(1);
            g2_launch(k_restart_g, 1, 1, 0, st, k->Lo); g2_count_launches(1);
            g2_launch(k_copy_g, 1, 64, 0, st, k->Lo); g2_count_launches(1);
            g2_launch(k_lincomb<double2, double2>, g, kVT, 0, st, k->w, 0.0, (const double2 *)nullptr, k->Vo, k->N, k->Lo.y,
                                                           k->Lo.flags + F_L, k->N, nullptr); g2_count_launches(1);
        }
        // instances that stopped in this cycle: final actions now (their own kernels only)
        for (int i = 0; i < n; i++) {
            if (!finishing[i]) continue;
            batch_final_launch<CI>(b, i, st, rc);
            if (rc) return rc;
        }
        bool any_fin = false;
        for (int i = 0; i < n; i++) any_fin = any_fin || finishing[i];
        if (any_fin) {
            // read the true residuals of the instances that finished (pull reads active ones only)
            std::vector<int> fin;
            for (int i = 0; i < n; i++)
                if (finishing[i]) fin.push_back(i);
            if ((rc = batch_pull_start(b, fin, 0, st)) || (rc = batch_pull_finish(b, fin, 0, h))) return rc;
            for (int i = 0; i < n; i++) {
                if (!finishing[i]) continue;
                const double be = std::sqrt(h[i].s[S_NRM2]) / bn[i];
                info[i].iterations = (int)b->history[i].size();
                info[i].bea = bea[i];
                info[i].be = be;
                info[i].stat = converged[i] ? (be >= tol ? 2 : 1) : -1;
                finishing[i] = 0;
            }
        }
    }
    return G2_OK;
}

int batch_solve_device(void *h, const double2 *const *d_Ebkg, double2 *const *d_Esol, const double2 *const *d_E0,
                       const GIEM2G_FGMRES_CTL &ctl, GIEM2G_RESULT *info)
{
    BatchWork *b = reinterpret_cast<BatchWork *>(h);
    if (!b) return G2_ERR_STATE;
    if (ctl.fgmres_buf != b->mo || ctl.gmres_buf != b->mi || (ctl.precision >= 0 && ctl.precision != b->precision)) {
        g2_set_error_msg("batched solve: buffer sizes or precision differ from the batch's");
        return G2_ERR_ARG;
    }
    cudaStream_t st = b->st;
    for (IeOp *op : b->ops)
        if (op->stream != st) G2_CUDA_CHECK(cudaStreamSynchronize(op->stream));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, st);
    for (int i = 0; i < b->n; i++) {
        IeOp *op = b->ops[i];
        KrylovWork *k = b->k[i];
        k->applies32 = k->applies64 = 0;
        const int g = vec_grid(k->N);
        // SolveEquation (ie_solver_module.F90:62-80): rhs = sqrt(Re sb) E_bkg; guess = E0/a or rhs
        g2_launch(k_rhs, g, 256, 0, st, k->b, d_Ebkg[i], op->d_post64, (size_t)op->Nx * op->Ny, op->Nz); g2_count_launches(1);
        if (d_E0 && d_E0[i]) {
            g2_launch(k_scale_asig, g, 256, 0, st, k->x, d_E0[i], op->d_asig64, op->cells(), true); g2_count_launches(1);
        } else {
            G2_CUDA_CHECK(cudaMemcpyAsync(k->x, k->b, sizeof(double2) * k->N, cudaMemcpyDeviceToDevice, st));
        }
    }
    int rc = b->precision == 0 ? batch_outer<double2>(b, ctl, info, st) : batch_outer<float2>(b, ctl, info, st);
    if (rc) return rc;
    for (int i = 0; i < b->n; i++) {
        IeOp *op = b->ops[i];
        KrylovWork *k = b->k[i];
        g2_launch(k_scale_asig, vec_grid(k->N), 256, 0, st, d_Esol[i], k->x, op->d_asig64, op->cells(), false); g2_count_launches(1);
    }
    cudaEventRecord(e1, st);
    G2_CUDA_CHECK(cudaStreamSynchronize(st));
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    for (int i = 0; i < b->n; i++) {
        info[i].applies_fp64 = b->k[i]->applies64;
        info[i].applies_fp32 = b->k[i]->applies32;
        info[i].device_ms = ms;
        b->ops[i]->mult_num += b->k[i]->applies64 + b->k[i]->applies32;
    }
    for (IeOp *op : b->ops) {
        const int e = ie_check_device_error(op);
        if (e) return e;
    }
    return G2_OK;
}

int batch_stage(void *h, double2 **d_stage, size_t *N)
{
    BatchWork *b = reinterpret_cast<BatchWork *>(h);
    if (!b) return G2_ERR_STATE;
    size_t nmax = 0;
    for (IeOp *op : b->ops) nmax = op->nvec() > nmax ? op->nvec() : nmax;
    if (!b->d_stage) G2_CUDA_CHECK(cudaMalloc(&b->d_stage, sizeof(double2) * nmax * 3 * b->n));
    *d_stage = b->d_stage;
    *N = nmax;
    return G2_OK;
}

int batch_size(void *h) { return h ? reinterpret_cast<BatchWork *>(h)->n : 0; }
IeOp *batch_op(void *h, int i) { return reinterpret_cast<BatchWork *>(h)->ops[i]; }
