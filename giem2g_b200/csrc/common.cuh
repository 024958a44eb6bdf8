// Common device helpers: complex arithmetic on double2/float2 and error handling.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>

#define G2_HD __host__ __device__ __forceinline__
#define G2_D __device__ __forceinline__

template <typename R> struct Cplx;
template <> struct Cplx<double> { using T = double2; };
template <> struct Cplx<float> { using T = float2; };

G2_HD double2 mk(double a, double b) { return make_double2(a, b); }
G2_HD float2 mk(float a, float b) { return make_float2(a, b); }

template <typename C> G2_HD C czero();
template <> G2_HD double2 czero<double2>() { return make_double2(0.0, 0.0); }
template <> G2_HD float2 czero<float2>() { return make_float2(0.f, 0.f); }

G2_HD double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
G2_HD double2 operator-(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
G2_HD float2 operator+(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
G2_HD float2 operator-(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
G2_HD double2 cmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
G2_HD float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
G2_HD double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
G2_HD float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
G2_HD double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
G2_HD float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
// acc += a*b
G2_HD void cfma(double2 &acc, double2 a, double2 b)
{
    acc.x = fma(a.x, b.x, acc.x);
    acc.x = fma(-a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y);
    acc.y = fma(a.y, b.x, acc.y);
}
G2_HD void cfma(float2 &acc, float2 a, float2 b)
{
    acc.x = fmaf(a.x, b.x, acc.x);
    acc.x = fmaf(-a.y, b.y, acc.x);
    acc.y = fmaf(a.x, b.y, acc.y);
    acc.y = fmaf(a.y, b.x, acc.y);
}
// complex division a/b (Smith's algorithm)
G2_HD double2 cdiv(double2 a, double2 b)
{
    if (fabs(b.x) >= fabs(b.y)) {
        double r = b.y / b.x, d = b.x + b.y * r;
        return make_double2((a.x + a.y * r) / d, (a.y - a.x * r) / d);
    } else {
        double r = b.x / b.y, d = b.y + b.x * r;
        return make_double2((a.x * r + a.y) / d, (a.y * r - a.x) / d);
    }
}

template <typename C> G2_HD C to_c(double2 v);
template <> G2_HD double2 to_c<double2>(double2 v) { return v; }
template <> G2_HD float2 to_c<float2>(double2 v) { return make_float2((float)v.x, (float)v.y); }

G2_HD int ilog2(int n)
{
    int l = 0;
    while ((1 << l) < n) l++;
    return l;
}
G2_D int bitrev(int v, int bits) { return (int)(__brev((unsigned)v) >> (32 - bits)); }

// In-place radix-2 DIT FFT of `nlines` lines of length L = 2^log2L held in shared memory.
// Element i of line l lives at s[l*ls + i*es]; the data must already be in bit-reversed order.
// tw[j] = exp(-2*pi*i*j/L) for j < L/2 (forward); inverse uses the conjugates.  Unnormalised.
// LINE_FAST selects the thread->butterfly mapping (line index fastest when lines are interleaved).
template <typename C, bool LINE_FAST>
G2_D void smem_fft(C *s, int log2L, int nlines, int ls, int es, const C *__restrict__ tw, bool inverse)
{
    const int L = 1 << log2L, half = L >> 1;
    const int nb = nlines * half;
    for (int lh = 0; lh < log2L; lh++) {
        const int h = 1 << lh;
        const int tshift = log2L - 1 - lh;  // twiddle index j * (L/(2h))
        for (int b = threadIdx.x; b < nb; b += blockDim.x) {
            int line, k;
            if (LINE_FAST) { line = b % nlines; k = b / nlines; }
            else { k = b & (half - 1); line = b >> (log2L - 1); }
            const int j = k & (h - 1);
            const int i0 = ((k >> lh) << (lh + 1)) + j;
            C w = tw[j << tshift];
            if (inverse) w.y = -w.y;
            C *p0 = s + line * ls + i0 * es;
            C *p1 = p0 + h * es;
            C a = *p0, bb = cmul(*p1, w);
            *p0 = a + bb;
            *p1 = a - bb;
        }
        __syncthreads();
    }
}

// Device layout of a spectral tensor unit (the tensor-core contraction's): the six blocks in the packed order of
// the spatial tensor, each stored as 8 x 8 tiles so that a warp's fragment reads (8 rows x 4 columns, or the
// transpose) hit distinct shared-memory banks.  Inside a tile element (r, c) sits at c * h + (r ^ f(c)), h the
// tile's rows (plain c * h + r in a tile of fewer than 8 rows); f spreads 4 x 4 elements over the 16 8-byte banks
// of complex64, and 2 x 4 and 4 x 2 elements over the 8 16-byte banks of complex128.  Row-major 8 x 8 storage
// without f cost 4 to 8 wavefronts where 2 (complex64) or 4 (complex128) suffice.
//   full blocks (xz, yz): tiles by row strips;  symmetric blocks: upper tiles, column of tiles by column of tiles,
//   the tile on the diagonal packed (lo + hi (hi + 1) / 2).  Every element is stored once: T elements per unit.
template <bool F64> G2_HD int tile_xor(int c) { return F64 ? ((c & 1) << 2) ^ (c & 2) : (c & 2) << 1; }
template <bool F64> G2_HD int full_pos(int r, int c, int N)
{
    const int I = r >> 3, J = c >> 3, h = N - 8 * I < 8 ? N - 8 * I : 8;
    return 8 * I * N + h * 8 * J + (c & 7) * h + ((r & 7) ^ (h == 8 ? tile_xor<F64>(c & 7) : 0));
}
template <bool F64> G2_HD int sym_pos(int i, int j, int N)
{
    const int lo = i < j ? i : j, hi = i < j ? j : i, I = lo >> 3, J = hi >> 3;
    const int w = N - 8 * J < 8 ? N - 8 * J : 8, base = 36 * J + 32 * J * (J - 1);
    if (I < J) return base + I * 8 * w + (hi & 7) * 8 + ((lo & 7) ^ tile_xor<F64>(hi & 7));
    const int a = lo & 7, b = hi & 7;
    return base + J * 8 * w + a + b * (b + 1) / 2;
}
// position of the spatial tensor's element e (packed upper xx, xy, yy, zz; column-major xz, yz) in a unit
template <bool F64> G2_HD int unit_pos(int e, int Nz)
{
    const int P = Nz * (Nz + 1) / 2;
    if (e < 4 * P) {
        const int blk = e / P, p = e - blk * P;
        int j = 0;
        while ((j + 1) * (j + 2) / 2 <= p) j++;
        return blk * P + sym_pos<F64>(p - j * (j + 1) / 2, j, Nz);
    }
    const int li = e - 4 * P, blk = li / (Nz * Nz), rc = li - blk * Nz * Nz;
    return 4 * P + blk * Nz * Nz + full_pos<F64>(rc % Nz, rc / Nz, Nz);
}

// Layout of the units that the other contraction kernels read: packed upper blocks as they are, and
// the full (xz, yz) Nz x Nz blocks column-major with the row index XOR-swizzled by
// the low bits of the column, so lane-parallel reads of a row and of a column both hit distinct
// shared-memory banks.  W = 1 is plain column-major.
G2_HD int asw(int r, int c, int N, int W) { return c * N + (r ^ (c & (W - 1))); }
// swizzle widths used for the FP64 and FP32 device tensors
__host__ __device__ constexpr int asw_width64(int Nz) { return (Nz % 8 == 0) ? 8 : 1; }
__host__ __device__ constexpr int asw_width32(int Nz) { return (Nz % 16 == 0) ? 16 : ((Nz % 8 == 0) ? 8 : 1); }

// position of the spatial tensor's element e in a unit of that layout
template <bool F64> G2_HD int plain_pos(int e, int Nz)
{
    const int P4 = 2 * Nz * (Nz + 1);
    if (e < P4) return e;
    const int li = e - P4, blk = li / (Nz * Nz), rc = li - blk * Nz * Nz;
    return P4 + blk * Nz * Nz + asw(rc % Nz, rc / Nz, Nz, F64 ? asw_width64(Nz) : asw_width32(Nz));
}

#define G2_CUDA_CHECK(expr)                                                                    \
    do {                                                                                       \
        cudaError_t e_ = (expr);                                                               \
        if (e_ != cudaSuccess) {                                                               \
            g2_set_error(__FILE__, __LINE__, cudaGetErrorString(e_));                          \
            return G2_ERR_CUDA;                                                                \
        }                                                                                      \
    } while (0)

void g2_set_error(const char *file, int line, const char *msg);

// Programmatic dependent launch for the solver's chains of short kernels.  pdl_wait() is the first statement of every
// kernel launched with g2_launch: it returns when the preceding kernel of the stream has completed and its writes are
// visible (so, by induction over the chain, everything before it too).  The wait also lets the next kernel's blocks be
// set up while this one runs: a complex128 apply of 32x32x8, five kernels, fell from 29 to 21.5 us.
G2_D void pdl_wait_only()  // the next kernel starts when this one ends
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
G2_D void pdl_wait()
{
    pdl_wait_only();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... P, typename... A>
inline cudaError_t g2_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
