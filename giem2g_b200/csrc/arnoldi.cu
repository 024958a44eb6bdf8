// One Arnoldi step of up to KMI lockstep instances in one cooperative launch: the dots of the first Gram-Schmidt pass, the
// correction passes, V_{j+1} = w / ||w|| and the Givens update (gmres.F90:263-326), with a grid barrier per pass.
//
// As a launch per sweep (dots, four passes of which usually one or two do anything, scaling) a step of a small grid took
// about 25 us, nearly all of it ramps, tails and last-block reductions.  Here every block keeps its part of the vectors
// for the whole step, reduces all partial sums of a pass itself (a fixed order, so the result does not depend on the
// schedule) and takes the pass decision with the others.  blockIdx.y is the instance; the barrier joins the blocks of one
// instance.  The launch is cooperative, so all blocks are resident; the waits are bounded (2 s, error code 51).
// Whole solves, launches per sweep -> one launch with its barriers, the last scalar step beside the scaling and the scaling
// four words at a time: FP64 32x32x8 3.31 -> 2.30 ms, mixed pairs 128x128x32 2 ms of 66 (bound by the sweeps' HBM and L2
// traffic); with the correction sweep backwards, the cycle start in two launches and sums in FP64 beyond 16 elements 2.0 ms
// and, of such a pair's 60 ms, 11.3.
#include <atomic>
#include <type_traits>
#include <utility>
#include "krylov_dev.cuh"

namespace {

// All blocks of an instance.  Block 0 arrives with 2^31 - (n - 1), the others with 1: n arrivals flip the word's top bit
// and leave the rest as it was, so nothing is reset and launches of any grid can follow one another.  One release, one
// L2 round trip and an acquiring poll: about 2 k clocks with 48 blocks, where an arrival counter with a generation word
// between full fences had taken 6.4-7.7 k, 3.5 us in each of the step's two or three barriers.
G2_D bool grid_barrier(unsigned *bar, unsigned n, int *err)
{
    __shared__ bool ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = true;
        const unsigned add = blockIdx.x == 0 ? 0x80000000u - (n - 1) : 1u;
        unsigned old, cur;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(bar), "r"(add) : "memory");
        unsigned long long t0 = 0, t1;
        for (int spin = 0;; spin++) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(bar) : "memory");
            if ((cur ^ old) & 0x80000000u) break;
            if ((spin & 255) != 255) continue;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
            if (t0 == 0) t0 = t1;
            if (t1 - t0 > 2000000000ull) {
                atomicCAS(err, 0, 51);
                ok = false;
                break;
            }
        }
    }
    __syncthreads();
    return ok;
}

// end of Arnoldi step j (gmres.F90:283-326): column j of H from the summed dots hc, H(j+1,j) = ||w||, the rotations, the
// Arnoldi misfit and the exit test, by the lanes of one warp; cs, sn, g and the scalars were fetched when the step began.
struct Finish {
    double cs[KMAX], bn;
    double2 sn[KMAX], g[2];
    int iter;
};
G2_D void finish_load(Finish &f, const Level &L, int j)
{
    const int t = threadIdx.x;
    if (t < j) {
        f.cs[t] = L.cs[t];
        f.sn[t] = L.sn[t];
    }
    if (t >= 32 && t < 34) f.g[t - 32] = L.H[hix(j + t - 32, L.m, L.m)];
    if (t == 64) f.bn = L.scal[S_BN];
    if (t == 65) f.iter = L.flags[F_ITER];
}
G2_D void finish_step(Finish &f, double2 *hc, Level &L, int j, double nrm, double tol)
{
    const int m = L.m, lane = threadIdx.x & 31;
    const double dnormw = sqrt(nrm);
    if (lane == 0) {
        double2 h = hc[0];
        for (int i = 0; i < j; i++) {
            double2 nx = hc[i + 1];
            zrot1(h, nx, f.cs[i], f.sn[i]);
            hc[i] = h;
            h = nx;
        }
        // netlib ZROTG of (h, ||w||); the second argument is real and not negative
        double2 hn = make_double2(dnormw, 0.0), sn;
        double c;
        const double ah = cabs_(h);
        if (ah == 0.0) {
            c = 0.0;
            sn = make_double2(1.0, 0.0);
        } else {
            const double scale = ah + dnormw, a1 = ah / scale, b1 = dnormw / scale, norm = scale * sqrt(a1 * a1 + b1 * b1);
            const double2 alpha = cdivr(h, ah);
            c = ah / norm;
            sn = cdivr(make_double2(alpha.x * dnormw, alpha.y * dnormw), norm);
        }
        zrot1(f.g[0], f.g[1], c, sn);
        zrot1(h, hn, c, sn);
        hc[j] = h;
        hc[j + 1] = make_double2(0.0, 0.0);
        const double bea = cabs_(f.g[1]) / f.bn;
        if (bea < tol || j + 1 >= m) L.flags[F_KRYLOV] = 0;
        L.scal[S_BEA] = bea;
        L.cs[j] = c;
        L.sn[j] = sn;
        L.H[hix(j, m, m)] = f.g[0];
        L.H[hix(j + 1, m, m)] = f.g[1];
        L.scal[S_NRM2] = nrm;
        L.flags[F_ITER] = f.iter + 1;
        L.flags[F_L] = j + 1;
    }
    __syncwarp();
    for (int i = lane; i <= j + 1; i += 32) L.H[hix(i, j, m)] = hc[i];
}

// v = f(w): rounds of U words per thread, loads first.  FIN: in block 0, where the first warp finishes the step meanwhile,
// the other seven take its words too.
template <bool FIN, typename T, typename F>
G2_D void scale_rows(const T *w, T *v, size_t n, size_t S, F f)
{
    constexpr int U = 4;
    const bool first = FIN && blockIdx.x == 0;
    const size_t rows = (n + S - 1) / S, T0 = blockIdx.x * (size_t)kVT + threadIdx.x;
    const size_t rounds = first ? (rows * kVT + kVT - 33) / (kVT - 32) : rows;
    auto at = [&](size_t r) {
        const size_t q = threadIdx.x - 32 + (kVT - 32) * r;
        return first ? (q % kVT) + (q / kVT) * S : T0 + r * S;
    };
    for (size_t r = 0; r < rounds; r += U) {
        T x[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (at(r + u) < n) x[u] = w[at(r + u)];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (at(r + u) < n) v[at(r + u)] = f(x[u]);
    }
}

// Sums of a complex64 sweep: a thread adds up to kChain elements in FP32, then that to FP64 sums of its own in shared
// memory.  (A thread's part of a vector is 83 elements for a pair of 128x128x32 and 498 for one of 256x256x48; in one FP32
// chain its error would grow with it.)
constexpr int kChain = 16;
template <typename C, int K> constexpr size_t sums_bytes()
{
    return sizeof(C) == sizeof(float2) ? (K + 1) * kVT * sizeof(double2) : 0;
}

template <typename C, int K>
__global__ void __launch_bounds__(kVT) k_arnoldi(Multi<C> mm, size_t N, double tol, int *err)
{
    pdl_wait();
    const int y = blockIdx.y;
    if (mm.gate[y] && *mm.gate[y] == 0) return;
    using R = typename RealOf<C>::T;
    using W = typename Wide<C>::T;
    constexpr int E = Wide<C>::E, j = K - 1;
    __shared__ double2 hs[KMAX + 1], hn[KMAX + 1], hsum[KMAX + 1];
    __shared__ double nrm;
    __shared__ Finish fin;
    Level L = mm.L[y];
    if (blockIdx.x == 0) finish_load(fin, L, j);
    C *V = mm.V[y], *w = mm.w[y];
    const size_t S = (size_t)gridDim.x * kVT, t0 = blockIdx.x * (size_t)kVT + threadIdx.x;
    const size_t Nw = wide_words<C>(N, N), ldw = N / E;
    const W *Vw = reinterpret_cast<const W *>(V);
    W *ww = reinterpret_cast<W *>(w);
    const size_t set = (size_t)gridDim.x * (KMAX + 1);
    R ax[K + 1], ay[K + 1];
    extern __shared__ __align__(16) double2 sums[];  // [K + 1][kVT]
    int added;  // elements in ax, ay
    bool kept;  // the thread has sums in shared memory
    auto zero = [&] {
#pragma unroll
        for (int k = 0; k <= K; k++) ax[k] = ay[k] = R(0);
        added = 0;
    };
    auto clear = [&] {
        zero();
        kept = false;
    };
    auto total = [&](int k) {
        double2 v = make_double2(ax[k], ay[k]);
        if constexpr (sums_bytes<C, K>() > 0)
            if (kept) {
                const double2 s = sums[k * kVT + threadIdx.x];
                v.x += s.x;
                v.y += s.y;
            }
        return v;
    };
    auto count = [&](int n) {  // after n more elements
        if constexpr (sums_bytes<C, K>() > 0) {
            added += n;
            if (added + n <= kChain) return;
#pragma unroll
            for (int k = 0; k <= K; k++) sums[k * kVT + threadIdx.x] = total(k);
            kept = true;
            zero();
        }
    };
    auto dots = [&](const C &a, const C *b) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            ax[k] += b[k].x * a.x + b[k].y * a.y;
            ay[k] += b[k].x * a.y - b[k].y * a.x;
        }
    };
    auto dots_of = [&](const C &a, size_t i) {  // the basis values of element i from memory
#pragma unroll
        for (int k = 0; k < K; k++) {
            const C b = V[(size_t)k * N + i];
            ax[k] += b.x * a.x + b.y * a.y;
            ay[k] += b.x * a.y - b.y * a.x;
        }
    };
    // U words per thread and round, every load of the round first; HOLD: the K basis values fit the registers
    constexpr bool HOLD = SweepU<K, W>::v > 0;
    constexpr int U = HOLD ? SweepU<K, W>::v : 1, KH = HOLD ? K : 1;
    clear();
    size_t i = t0;
    if constexpr (HOLD) {
        auto round = [&](auto nu) {
            constexpr int NU = decltype(nu)::value;
            W wv[NU], v[KH][NU];
#pragma unroll
            for (int u = 0; u < NU; u++) wv[u] = ww[i + u * S];
#pragma unroll
            for (int k = 0; k < KH; k++)
#pragma unroll
                for (int u = 0; u < NU; u++) v[k][u] = Vw[(size_t)k * ldw + i + u * S];
#pragma unroll
            for (int u = 0; u < NU; u++)
#pragma unroll
                for (int e = 0; e < E; e++) {
                    C b[KH];
#pragma unroll
                    for (int k = 0; k < KH; k++) b[k] = part_of(v[k][u], e);
                    dots(part_of(wv[u], e), b);
                }
            count(NU * E);
        };
        for (; i + (U - 1) * S < Nw; i += U * S) round(std::integral_constant<int, U>());
        for (; i < Nw; i += S) round(std::integral_constant<int, 1>());
    }
    for (i = HOLD ? Nw * E + t0 : t0; i < N; i += S) {
        dots_of(w[i], i);
        count(1);
    }
    block_reduce_store<K>(total, mm.part[y]);
    if (!grid_barrier(L.bar, gridDim.x, err)) return;
    reduce_partials(mm.part[y], gridDim.x, K, hs, nullptr);
    if (threadIdx.x < K) hsum[threadIdx.x] = hs[threadIdx.x];
    __syncthreads();
    for (int p = 1;; p++) {
        // w -= V hs; dots and norm of the new w
        clear();
        auto take = [&](C &a, const C &b, int k) {
            const R hx = (R)hs[k].x, hy = (R)hs[k].y;
            a.x -= b.x * hx - b.y * hy;
            a.y -= b.x * hy + b.y * hx;
        };
        i = t0;
        if constexpr (HOLD) {
            auto round = [&](auto nu) {
                constexpr int NU = decltype(nu)::value;
                W wv[NU], v[KH][NU];
#pragma unroll
                for (int u = 0; u < NU; u++) wv[u] = ww[i + u * S];
#pragma unroll
                for (int k = 0; k < KH; k++)
#pragma unroll
                    for (int u = 0; u < NU; u++) v[k][u] = Vw[(size_t)k * ldw + i + u * S];
#pragma unroll
                for (int u = 0; u < NU; u++) {
#pragma unroll
                    for (int e = 0; e < E; e++) {
                        C a = part_of(wv[u], e), b[KH];
#pragma unroll
                        for (int k = 0; k < KH; k++) {
                            b[k] = part_of(v[k][u], e);
                            take(a, b[k], k);
                        }
                        ax[K] += a.x * a.x + a.y * a.y;
                        dots(a, b);
                        set_part(wv[u], e, a);
                    }
                    ww[i + u * S] = wv[u];
                }
                count(NU * E);
            };
            // backwards after the forward sweep before it, whose last words are still in L2 (odd p): pairs 128x128x32, steps
            // of 10, 7 and 4 vectors 154 -> 142, 93 -> 82, 60 -> 53 us
            const size_t full = Nw > t0 ? ((Nw - t0 + S - 1) / S) / U : 0;
            if (p & 1) {
                for (i = t0 + full * U * S; i < Nw; i += S) round(std::integral_constant<int, 1>());
                for (size_t r = full; r-- > 0;) {
                    i = t0 + r * U * S;
                    round(std::integral_constant<int, U>());
                }
            } else {
                for (; i + (U - 1) * S < Nw; i += U * S) round(std::integral_constant<int, U>());
                for (; i < Nw; i += S) round(std::integral_constant<int, 1>());
            }
        }
        for (i = HOLD ? Nw * E + t0 : t0; i < N; i += S) {
            C a = w[i];
#pragma unroll
            for (int k = 0; k < K; k++) take(a, V[(size_t)k * N + i], k);
            w[i] = a;
            ax[K] += a.x * a.x + a.y * a.y;
            dots_of(a, i);
            count(1);
        }
        double2 *part = mm.part[y] + (p & 1) * set;  // the other set may still be read by a slower block
        block_reduce_store<K>(total, part);
        if (!grid_barrier(L.bar, gridDim.x, err)) return;
        reduce_partials(part, gridDim.x, K, hn, &nrm);
        // gmres.F90:277-280
        double dl = 0.0;
        for (int k = 0; k < K; k++) dl += hs[k].x * hs[k].x + hs[k].y * hs[k].y;
        if (2.0 * sqrt(nrm) > sqrt(dl) || p > N_IGS) break;
        __syncthreads();
        if (threadIdx.x < K) {
            hsum[threadIdx.x].x += hn[threadIdx.x].x;
            hsum[threadIdx.x].y += hn[threadIdx.x].y;
            hs[threadIdx.x] = hn[threadIdx.x];
        }
        __syncthreads();
    }
    // every block has read its gate, a flag that the step's end may clear: all of them passed the barriers above
    if (blockIdx.x == 0 && threadIdx.x < 32) return finish_step(fin, hsum, L, j, nrm, tol);
    const double inv = 1.0 / sqrt(nrm);
    if (HOLD && Nw)
        scale_rows<true>(ww, reinterpret_cast<W *>(V) + (size_t)K * ldw, Nw, S, [&](W x) {
#pragma unroll
            for (int e = 0; e < E; e++) set_part(x, e, scaled(part_of(x, e), inv));
            return x;
        });
    else scale_rows<true>(w, V + (size_t)K * N, N, S, [&](C x) { return scaled(x, inv); });
}

// ---- start of an inner cycle -----------------------------------------------------------------------
// Two launches, one before and one after the apply that forms A x0, where a launch per operation (reset, norm, scalars,
// copy; difference, norm, scalars, column g, scaling) had taken nine of 2-4 us each on a small grid.  A thread sums the
// words of a round in the vector's precision and the rounds in FP64.
template <typename C>
__global__ void __launch_bounds__(kVT) k_begin(Starts<C> s, size_t N, int *err)
{
    pdl_wait();
    using R = typename RealOf<C>::T;
    using W = typename Wide<C>::T;
    constexpr int E = Wide<C>::E, U = 4;
    const int y = blockIdx.y;
    Level L = s.L[y];
    const C *v = s.v[y], *x0 = s.x0[y];
    C *x = s.x[y];
    const size_t S = (size_t)gridDim.x * kVT, t0 = blockIdx.x * (size_t)kVT + threadIdx.x, Nw = wide_words<C>(N, N);
    double sum = 0.0;
    const W *vw = reinterpret_cast<const W *>(v);
    for (size_t i = t0; i < Nw; i += U * S) {
        R r = R(0);
        W a[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i + u * S < Nw) a[u] = vw[i + u * S];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i + u * S < Nw)
#pragma unroll
                for (int e = 0; e < E; e++) {
                    const C c = part_of(a[u], e);
                    r += c.x * c.x + c.y * c.y;
                }
        sum += r;
    }
    for (size_t i = Nw * E + t0; i < N; i += S) sum += v[i].x * v[i].x + v[i].y * v[i].y;
    block_reduce_store<0>([&](int) { return make_double2(sum, 0.0); }, s.part[y]);
    if (!grid_barrier(L.bar, gridDim.x, err)) return;
    __shared__ double nrm;
    reduce_partials(s.part[y], gridDim.x, 0, nullptr, &nrm);
    const double bn = sqrt(nrm);
    const bool zero = bn < ZERO_THRESHOLD;
    const W *xw = reinterpret_cast<const W *>(x0);
    for (size_t i = t0; i < Nw; i += U * S) {
        W a[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i + u * S < Nw) a[u] = zero ? W() : xw[i + u * S];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i + u * S < Nw) reinterpret_cast<W *>(x)[i + u * S] = a[u];
    }
    for (size_t i = Nw * E + t0; i < N; i += S) x[i] = zero ? C() : x0[i];
    if (blockIdx.x != 0) return;
    for (int i = threadIdx.x; i < (L.m + 1) * (L.m + 1); i += kVT) L.H[i] = make_double2(0.0, 0.0);
    if (threadIdx.x == 0) {
        L.scal[S_NRM2] = nrm;
        L.scal[S_BN] = bn;
        L.flags[F_SOLVER] = L.flags[F_KRYLOV] = zero || (s.go[y] && *s.go[y] == 0) ? 0 : 1;
        L.flags[F_ITER] = 0;
        L.flags[F_L] = 0;
    }
}

template <typename C>
__global__ void __launch_bounds__(kVT) k_residual(Starts<C> s, size_t N, double tol, int *err)
{
    pdl_wait();
    using R = typename RealOf<C>::T;
    using W = typename Wide<C>::T;
    constexpr int E = Wide<C>::E, U = 4;
    const int y = blockIdx.y;
    Level L = s.L[y];
    if (L.flags[F_SOLVER] == 0) return;
    const double bn = L.scal[S_BN];
    const C *v = s.v[y];
    C *r = s.r[y];
    const size_t S = (size_t)gridDim.x * kVT, t0 = blockIdx.x * (size_t)kVT + threadIdx.x, Nw = wide_words<C>(N, N);
    double sum = 0.0;
    R round = R(0);
    auto diff = [&](C b, C a) {
        b.x -= a.x;
        b.y -= a.y;
        round += b.x * b.x + b.y * b.y;
        return b;
    };
    auto add_round = [&] {
        sum += round;
        round = R(0);
    };
    const W *vw = reinterpret_cast<const W *>(v);
    W *rw = reinterpret_cast<W *>(r);
    for (size_t i = t0; i < Nw; i += U * S) {
        W a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i + u * S < Nw) {
                a[u] = rw[i + u * S];
                b[u] = vw[i + u * S];
            }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i + u * S < Nw) {
#pragma unroll
                for (int e = 0; e < E; e++) set_part(a[u], e, diff(part_of(b[u], e), part_of(a[u], e)));
                rw[i + u * S] = a[u];
            }
        add_round();
    }
    for (size_t i = Nw * E + t0; i < N; i += S) {
        r[i] = diff(v[i], r[i]);
        add_round();
    }
    block_reduce_store<0>([&](int) { return make_double2(sum, 0.0); }, s.part[y]);
    if (!grid_barrier(L.bar, gridDim.x, err)) return;
    __shared__ double nrm;
    reduce_partials(s.part[y], gridDim.x, 0, nullptr, &nrm);
    const double beta = sqrt(nrm), inv = 1.0 / beta;
    const bool done = beta / bn < tol;
    if (!done && Nw)
        scale_rows<false>(rw, reinterpret_cast<W *>(s.V[y]), Nw, S, [&](W a) {
#pragma unroll
            for (int e = 0; e < E; e++) set_part(a, e, scaled(part_of(a, e), inv));
            return a;
        });
    else if (!done) scale_rows<false>(r, s.V[y], N, S, [&](C a) { return scaled(a, inv); });
    if (blockIdx.x != 0) return;
    const int m = L.m;
    if (!done && threadIdx.x <= m) L.H[hix(threadIdx.x, m, m)] = make_double2(threadIdx.x ? 0.0 : beta, 0.0);
    if (threadIdx.x == 0) {
        L.scal[S_NRM2] = nrm;
        L.scal[S_BETA] = beta;
        if (done) L.flags[F_SOLVER] = 0;
        L.flags[F_KRYLOV] = done ? 0 : 1;
        L.flags[F_L] = 0;
    }
}

int sms()
{
    static const int n = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v > 0 ? v : 1;
    }();
    return n;
}

// a cooperative launch of `kernel` for n instances: as many blocks each as are resident together, up to nparts
template <typename... P, typename... A>
int launch(void (*kernel)(P...), int per_sm, size_t smem, size_t words, int n, int nparts, cudaStream_t st, A &&...args)
{
    const size_t need = (words + kVT - 1) / kVT;
    int g = per_sm * sms() / n;
    g = g < nparts ? g : nparts;
    g = (size_t)g < need ? g : (int)need;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(g < 1 ? 1 : g, n);
    cfg.blockDim = dim3(kVT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    G2_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
    g2_count_launches(1);
    return G2_OK;
}
// resident blocks per SM; kept once the calls have succeeded
template <typename F> int per_sm_of(F kernel, size_t smem, std::atomic<int> &kept, int *out)
{
    if (!(*out = kept.load())) {
        if (smem)
            G2_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        G2_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, kernel, kVT, smem));
        if (*out < 1) *out = 1;
        kept = *out;
    }
    return G2_OK;
}
template <typename C, int K>
int launch_step(const Multi<C> &mm, int n, size_t N, int nparts, double tol, int *err, cudaStream_t st)
{
    constexpr size_t smem = sums_bytes<C, K>();
    static std::atomic<int> kept{0};
    int per_sm;
    if (const int rc = per_sm_of(k_arnoldi<C, K>, smem, kept, &per_sm)) return rc;
    return launch(k_arnoldi<C, K>, per_sm, smem, N / Wide<C>::E + 1, n, nparts, st, mm, N, tol, err);
}
template <typename C>
int dispatch(const Multi<C> &mm, int n, size_t N, int nparts, int j, double tol, int *err, cudaStream_t st)
{
    switch (j + 1) {
#define G2_K(k) \
    case k: return launch_step<C, k>(mm, n, N, nparts, tol, err, st)
        G2_K(1);
        G2_K(2);
        G2_K(3);
        G2_K(4);
        G2_K(5);
        G2_K(6);
        G2_K(7);
        G2_K(8);
        G2_K(9);
        G2_K(10);
        G2_K(11);
        G2_K(12);
        G2_K(13);
        G2_K(14);
        G2_K(15);
        G2_K(16);
        G2_K(17);
        G2_K(18);
        G2_K(19);
        G2_K(20);
        G2_K(21);
        G2_K(22);
        G2_K(23);
        G2_K(24);
        G2_K(25);
        G2_K(26);
        G2_K(27);
        G2_K(28);
        G2_K(29);
        G2_K(30);
        G2_K(31);
#undef G2_K
    }
    return G2_ERR_UNSUPPORTED;
}

}  // namespace

int arnoldi_step(const Multi<float2> &mm, int n, size_t N, int nparts, int j, double tol, int *err, cudaStream_t st)
{
    return dispatch(mm, n, N, nparts, j, tol, err, st);
}
int arnoldi_step(const Multi<double2> &mm, int n, size_t N, int nparts, int j, double tol, int *err, cudaStream_t st)
{
    return dispatch(mm, n, N, nparts, j, tol, err, st);
}

template <typename C> int krylov_begin(const Starts<C> &s, int n, size_t N, int nparts, int *err, cudaStream_t st)
{
    static std::atomic<int> kept{0};
    int per_sm;
    if (const int rc = per_sm_of(k_begin<C>, 0, kept, &per_sm)) return rc;
    return launch(k_begin<C>, per_sm, 0, N / Wide<C>::E + 1, n, nparts, st, s, N, err);
}
template <typename C>
int krylov_residual(const Starts<C> &s, int n, size_t N, int nparts, double tol, int *err, cudaStream_t st)
{
    static std::atomic<int> kept{0};
    int per_sm;
    if (const int rc = per_sm_of(k_residual<C>, 0, kept, &per_sm)) return rc;
    return launch(k_residual<C>, per_sm, 0, N / Wide<C>::E + 1, n, nparts, st, s, N, tol, err);
}
template int krylov_begin(const Starts<float2> &, int, size_t, int, int *, cudaStream_t);
template int krylov_begin(const Starts<double2> &, int, size_t, int, int *, cudaStream_t);
template int krylov_residual(const Starts<float2> &, int, size_t, int, double, int *, cudaStream_t);
template int krylov_residual(const Starts<double2> &, int, size_t, int, double, int *, cudaStream_t);
