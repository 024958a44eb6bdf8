// Spectral transform of the Green's tensor, FP64, on the GPU.
//
// Restates CalcFFTofIETensorGeneral / CALC_FFT_OF_TENSOR_COMPONENT (Integral_Equation_Module.F90:319-471)
// together with the mirrored distributed FFT (Distributed_FFT.F90:384-414, 507-551):
//   - the spatial lags g(lx,ly), lx<Nx, ly<Ny, are extended to a 2Nx x 2Ny circulant with the component
//     parities (sx,sy): xx(+,+) xy(-,-) yy(+,+) zz(+,+) xz(-,+) yz(+,-); lags Nx and Ny are set to zero;
//   - forward 2-D DFT (exp(-i...)), unnormalised;
//   - y-Nyquist correction G(.,ky) -= (-1)^ky G(.,Ny) on every kx, then x-Nyquist correction
//     G(kx,.) -= (-1)^kx G(Nx,.) with the alternating sign starting at +1 for kx = 0;
//   - keep kx<Nx, ky<Ny.
// With these corrections the 2Nx x 2Ny circular convolution restricted to the physical grid is the exact
// block-Toeplitz product, for even Nx and Ny.
// Pass A transforms along x (lines over lx for each (ly, element)), pass B along y with both corrections.
// Elements of a unit are interleaved in shared memory so global loads/stores are coalesced.
#include <vector>
#include "common.cuh"
#include "ie_internal.h"

namespace {

constexpr int kThreads = 256;
constexpr int TE = 16;  // tensor elements per CTA

G2_D void elem_parity(int e, int P, int Nz, double &sx, double &sy)
{
    if (e < 4 * P) {
        const int comp = e / P;  // xx, xy, yy, zz
        sx = sy = (comp == 1) ? -1.0 : 1.0;
    } else {
        const int comp = (e - 4 * P) / (Nz * Nz);  // xz, yz
        sx = comp == 0 ? -1.0 : 1.0;
        sy = comp == 0 ? 1.0 : -1.0;
    }
}

// pass A: spatial [lx][ly][T] -> S1 [kx 0..Nx][ly][T]
__global__ void __launch_bounds__(kThreads) k_tensor_x(const double2 *__restrict__ g, double2 *__restrict__ S1,
                                                       const double2 *__restrict__ tw, int Nx, int Ny, int Nz)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *s = reinterpret_cast<double2 *>(smem_raw);
    const int P = Nz * (Nz + 1) / 2, T = 4 * P + 2 * Nz * Nz;
    const int L = 2 * Nx, lg = ilog2(L);
    const int ly = blockIdx.x, e0 = blockIdx.y * TE;
    const int ne = min(TE, T - e0);
    for (int i = threadIdx.x; i < L * TE; i += blockDim.x) s[i] = make_double2(0.0, 0.0);
    __syncthreads();
    for (int i = threadIdx.x; i < Nx * TE; i += blockDim.x) {
        const int lx = i / TE, t = i - lx * TE;
        if (t >= ne) continue;
        double sx, sy;
        elem_parity(e0 + t, P, Nz, sx, sy);
        const double2 v = g[((size_t)lx * Ny + ly) * T + e0 + t];
        s[bitrev(lx, lg) * TE + t] = v;
        if (lx > 0) s[bitrev(L - lx, lg) * TE + t] = make_double2(sx * v.x, sx * v.y);
    }
    __syncthreads();
    smem_fft<double2, true>(s, lg, TE, 1, TE, tw, false);
    for (int i = threadIdx.x; i < (Nx + 1) * TE; i += blockDim.x) {
        const int kx = i / TE, t = i - kx * TE;
        if (t < ne) S1[((size_t)kx * Ny + ly) * T + e0 + t] = s[kx * TE + t];
    }
}

// an element's place in a unit of the FP64 or the complex64 tensor
template <bool F64> G2_D int place(ushort4 p, int layout) { return layout == L_TILED ? (F64 ? p.x : p.y) : (F64 ? p.z : p.w); }

// pass B: S1 [kx][ly][T] -> out [kx][ky][T] (kx < Nx) or nyq [ky][T] (kx == Nx, when corr == nullptr)
__global__ void __launch_bounds__(kThreads) k_tensor_y(const double2 *__restrict__ S1, double2 *__restrict__ out,
                                                       const double2 *__restrict__ nyq, const double2 *__restrict__ tw,
                                                       const ushort4 *__restrict__ pos, int layout, int Nx, int Ny,
                                                       int Nz, int kx_base)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *s = reinterpret_cast<double2 *>(smem_raw);
    const int P = Nz * (Nz + 1) / 2, T = 4 * P + 2 * Nz * Nz;
    const int L = 2 * Ny, lg = ilog2(L);
    const int kx = kx_base + blockIdx.x, e0 = blockIdx.y * TE;
    const int ne = min(TE, T - e0);
    for (int i = threadIdx.x; i < L * TE; i += blockDim.x) s[i] = make_double2(0.0, 0.0);
    __syncthreads();
    for (int i = threadIdx.x; i < Ny * TE; i += blockDim.x) {
        const int ly = i / TE, t = i - ly * TE;
        if (t >= ne) continue;
        double sx, sy;
        elem_parity(e0 + t, P, Nz, sx, sy);
        const double2 v = S1[((size_t)kx * Ny + ly) * T + e0 + t];
        s[bitrev(ly, lg) * TE + t] = v;
        if (ly > 0) s[bitrev(L - ly, lg) * TE + t] = make_double2(sy * v.x, sy * v.y);
    }
    __syncthreads();
    smem_fft<double2, true>(s, lg, TE, 1, TE, tw, false);
    for (int i = threadIdx.x; i < Ny * TE; i += blockDim.x) {
        const int ky = i / TE, t = i - ky * TE;
        if (t >= ne) continue;
        const double2 ny = s[Ny * TE + t];
        const double sgn = (ky & 1) ? -1.0 : 1.0;
        double2 v = make_double2(s[ky * TE + t].x - sgn * ny.x, s[ky * TE + t].y - sgn * ny.y);
        if (nyq == nullptr) {
            out[(size_t)ky * T + e0 + t] = v;  // x-Nyquist row (plain layout, scratch)
        } else {
            const double sx = (kx & 1) ? -1.0 : 1.0;
            const double2 c = nyq[(size_t)ky * T + e0 + t];
            out[((size_t)kx * Ny + ky) * T + place<true>(pos[e0 + t], layout)] =
                make_double2(v.x - sx * c.x, v.y - sx * c.y);
        }
    }
}

// the complex64 copy of the FP64 tensor, each in its layout
__global__ void k_to_c64(const double2 *__restrict__ a, int la, float2 *__restrict__ b, int lb,
                         const ushort4 *__restrict__ pos, size_t units, int T)
{
    const size_t n = units * T;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t u = i / T;
        const ushort4 p = pos[i - u * T];
        const double2 v = a[u * T + place<true>(p, la)];
        b[u * T + place<false>(p, lb)] = make_float2((float)v.x, (float)v.y);
    }
}
// units of a from layout la to the other one, into b; b may be a (a block holds its unit in shared memory, 217 KB at most)
template <typename C>
__global__ void __launch_bounds__(512) k_relayout(const C *a, C *b, int la, const ushort4 *__restrict__ pos, size_t units,
                                                  int T)
{
    constexpr bool F64 = sizeof(C) == sizeof(double2);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *s = reinterpret_cast<C *>(smem_raw);
    for (size_t u = blockIdx.x; u < units; u += gridDim.x) {
        for (int e = threadIdx.x; e < T; e += blockDim.x) s[e] = a[u * T + e];
        __syncthreads();
        for (int e = threadIdx.x; e < T; e += blockDim.x) {
            const ushort4 p = pos[e];
            b[u * T + place<F64>(p, 1 - la)] = s[place<F64>(p, la)];
        }
        __syncthreads();
    }
}

}  // namespace

// positions of a unit's elements in the tensors (they depend on Nz alone)
static int make_positions(IeOp *op)
{
    if (op->d_pos) return G2_OK;
    const int T = op->Tunit(), Nz = op->Nz;
    std::vector<ushort4> h(T);
    for (int e = 0; e < T; e++)
        h[e] = make_ushort4((unsigned short)unit_pos<true>(e, Nz), (unsigned short)unit_pos<false>(e, Nz),
                            (unsigned short)plain_pos<true>(e, Nz), (unsigned short)plain_pos<false>(e, Nz));
    ushort4 *d = nullptr;
    G2_CUDA_CHECK(cudaMalloc(&d, T * sizeof(ushort4)));
    cudaError_t e = cudaMemcpyAsync(d, h.data(), T * sizeof(ushort4), cudaMemcpyHostToDevice, op->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(op->stream);
    if (e != cudaSuccess) cudaFree(d);
    G2_CUDA_CHECK(e);
    op->d_pos = d;
    return G2_OK;
}

template <typename C> static int relayout(IeOp *op, const C *a, C *b, int la)
{
    const int T = op->Tunit(), smem = (int)(T * sizeof(C));
    G2_CUDA_CHECK(cudaFuncSetAttribute(k_relayout<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const unsigned grid = (unsigned)(op->units() < 592 ? op->units() : 592);
    k_relayout<C><<<grid, 512, smem, op->stream>>>(a, b, la, op->d_pos, op->units(), T);
    G2_CUDA_CHECK(cudaGetLastError());
    g2_count_launches(1);
    return G2_OK;
}
// one precision's tensors t; need: the layouts that its contractions read
template <typename C> static int sync_layouts(IeOp *op, C *(&t)[2], const bool (&need)[2], bool alloc, bool *moved)
{
    const size_t bytes = op->units() * op->Tunit() * sizeof(C);
    if (!t[0] && !t[1]) {
        if (!alloc) return G2_OK;
        C *n[2] = {nullptr, nullptr};
        for (int l = 0; l < 2; l++)
            if (need[l] && cudaMalloc(&n[l], bytes) != cudaSuccess) {
                if (n[0]) cudaFree(n[0]);
                g2_set_error(__FILE__, __LINE__, cudaGetErrorString(cudaGetLastError()));
                return G2_ERR_NOMEM;
            }
        t[0] = n[0];
        t[1] = n[1];
        return G2_OK;
    }
    for (int l = 0; l < 2; l++) {
        const int o = 1 - l;
        if (!need[l] || t[l]) continue;
        if (need[o] || op->captured) {  // both layouts from now on
            C *n = nullptr;
            if (cudaMalloc(&n, bytes) != cudaSuccess) {
                g2_set_error(__FILE__, __LINE__, cudaGetErrorString(cudaGetLastError()));
                return G2_ERR_NOMEM;
            }
            int rc = relayout(op, t[o], n, o);
            if (!rc && cudaStreamSynchronize(op->stream) != cudaSuccess) rc = G2_ERR_CUDA;
            if (rc) {
                cudaFree(n);
                return rc;
            }
            t[l] = n;
        } else {
            const int rc = relayout(op, t[o], t[o], o);
            if (rc) return rc;
            t[l] = t[o];
            t[o] = nullptr;
            // a batch reads the tensors on its first operator's stream
            G2_CUDA_CHECK(cudaStreamSynchronize(op->stream));
        }
        *moved = true;
    }
    for (int l = 0; l < 2; l++)
        if (!need[l] && t[l] && t[1 - l] && !op->captured) {
            cudaFree(t[l]);
            t[l] = nullptr;
            *moved = true;
        }
    return G2_OK;
}

int ie_sync_layouts(IeOp *op, bool alloc)
{
    const bool mma[3] = {ie_uses_mma(op, 0), ie_uses_mma(op, 1), ie_uses_mma(op, 2)};
    const bool need64[2] = {mma[0], !mma[0]}, need32[2] = {mma[1] || mma[2], !mma[1] || !mma[2]};
    bool moved = false;
    int rc = sync_layouts(op, op->d_tensor64, need64, alloc, &moved);
    if (!rc) rc = sync_layouts(op, op->d_tensor32, need32, alloc, &moved);
    if (moved) op->config_gen++;  // captured graphs of the solvers hold the tensors' addresses
    return rc;
}

int ie_tensor_spectrum(IeOp *op, cudaStream_t st)
{
    const int Nx = op->Nx, Ny = op->Ny, Nz = op->Nz, T = op->Tunit();
    if (!op->d_spatial) return G2_ERR_STATE;
    int rcp = make_positions(op);
    if (!rcp) rcp = ie_sync_layouts(op, true);  // before the spatial tensor goes
    if (rcp) return rcp;
    double2 *S1 = nullptr, *nyq = nullptr;
    int rca = g2_pool_alloc(&op->pool, (void **)&S1, (size_t)(Nx + 1) * Ny * T * sizeof(double2), st);
    if (!rca) rca = g2_pool_alloc(&op->pool, (void **)&nyq, (size_t)Ny * T * sizeof(double2), st);
    if (rca) {
        g2_pool_free(S1, st);
        return rca;
    }
    const int l64 = op->d_tensor64[L_TILED] ? L_TILED : L_PLAIN, l32 = op->d_tensor32[L_TILED] ? L_TILED : L_PLAIN;
    double2 *t64 = op->d_tensor64[l64];
    float2 *t32 = op->d_tensor32[l32];
    const size_t smx = (size_t)2 * Nx * TE * sizeof(double2), smy = (size_t)2 * Ny * TE * sizeof(double2);
    G2_CUDA_CHECK(cudaFuncSetAttribute(k_tensor_x, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    G2_CUDA_CHECK(cudaFuncSetAttribute(k_tensor_y, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    const int eb = (T + TE - 1) / TE;
    k_tensor_x<<<dim3(Ny, eb), kThreads, smx, st>>>(op->d_spatial, S1, op->d_twx64, Nx, Ny, Nz);
    k_tensor_y<<<dim3(1, eb), kThreads, smy, st>>>(S1, nyq, nullptr, op->d_twy64, op->d_pos, l64, Nx, Ny, Nz, Nx);
    k_tensor_y<<<dim3(Nx, eb), kThreads, smy, st>>>(S1, t64, nyq, op->d_twy64, op->d_pos, l64, Nx, Ny, Nz, 0);
    k_to_c64<<<1184, 256, 0, st>>>(t64, l64, t32, l32, op->d_pos, op->units(), T);
    cudaError_t le = cudaGetLastError();
    if (le == cudaSuccess && op->d_tensor64[1 - l64] && relayout(op, t64, op->d_tensor64[1 - l64], l64)) le = cudaErrorUnknown;
    if (le == cudaSuccess && op->d_tensor32[1 - l32] && relayout(op, t32, op->d_tensor32[1 - l32], l32)) le = cudaErrorUnknown;
    g2_pool_free(S1, st);
    g2_pool_free(nyq, st);
    G2_CUDA_CHECK(le);
    // the reference transforms the kernel buffer in place (G_symm and G_symmT alias it), so the
    // spatial tensor does not outlive the transform there either
    g2_pool_free(op->d_spatial, st);
    op->d_spatial = nullptr;
    G2_CUDA_CHECK(cudaStreamSynchronize(st));
    op->have_spatial = false;
    return G2_OK;
}
