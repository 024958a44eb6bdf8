// Green's-tensor contraction on the tensor cores, for every Nz the operator accepts.
//
// At each unit (q, r) the six blocks act on the four points (+-kx, +-ky) with the reference's sign table
// (apply_ie_operator_module.F90:278-291).  Multiplying the y component by sx m and the z component by sx, on
// the way in and on the way out, takes every sign but one out of the table:
//     out_x = xx Ux + xy Uy + xz Uz,   out_y = xy Ux + yy Uy + yz Uz,   out_z = -(xz^T Ux + yz^T Uy) + zz Uz,
// the same 3Nz x 3Nz matrix M for every point (and for every vector that shares the tensor).  So a unit is one
// product of M with the 4 NP points' columns, and the tensor cores can do it:
//   * rows m of the A operand are the points' real and imaginary parts (V^T), columns n of the B operand the rows
//     of M, eight at a time; a complex product is four real ones, acc_R = V Re(M)^T and acc_I = V Im(M)^T, whose
//     rows combine into the outputs;
//   * complex128: mma.m8n8k4.f64, rows (point, part);
//   * complex64: mma.m16n8k8.tf32 with each operand split into two TF32 numbers, x = hi + lo.  The hi hi products of
//     one block and z'-tile start from zero and are added to the FP32 accumulator with a rounded add (the tensor core
//     truncates when it accumulates, which would bias a long sum); the hi lo and lo hi products, 2^-11 smaller,
//     accumulate in the tensor core.  Two vectors (NP = 2) fill the 16 rows with 8 points' parts; one vector (NP = 1)
//     fills them with 4 points' parts, hi in rows 0-7 and lo in rows 8-15, so two instructions do the four products.
//     Up to 12 z the operands are split into three numbers, which hold every bit: an FP32 sum that short has a smaller
//     error than two numbers leave (the last bit of lo, for NP = 2 the lo lo products), and the launch is bound elsewhere
//     (128x128x8: 22 and 26 us where two numbers take 16 and 19).
// Error of a unit's products against 80-bit sums, FP32 FMA kernels (plain or contract.cu's) -> this one, single / pair:
// random units Nz = 8 1.1e-7 / 1.4e-7 -> 0.6e-7 / 0.6e-7, Nz = 13 1.00e-7 -> 0.94e-7 / 1.03e-7, Nz = 32 1.20e-7 / 1.43e-7
// -> 1.02e-7 / 1.12e-7, Nz = 48 1.7e-7 -> 1.1e-7 / 1.2e-7; a layered background's tensor (Nz = 32) 1.09e-7 / 1.29e-7 ->
// 0.92e-7 / 1.01e-7; one non-zero component 0.95e-7 / 1.01e-7 -> 0.88e-7 / 0.98e-7; coherent signs 0.63e-7 / 0.82e-7 ->
// 0.69e-7 / 0.70e-7; one non-zero layer 0.74e-7 -> 0.88e-7 / 0.98e-7.
// M's elements are read straight from the packed unit in shared memory: their offsets depend on the lane alone, so every
// lane keeps its offsets in registers for the whole kernel; padded columns point at a zero.  The spectrum has a row pitch
// of 4 mod 8 elements, which spreads the points' columns over the shared-memory banks.  complex128 warps own eight rows
// of M (padded within (x, y) and within z, so that the sign of out_z is one per tile); complex64 warps own the x, y and
// z rows of eight z, which lets one split of an xy tile serve two products.
// What bounds it at 128x128x32 (16384 units): complex128 HBM (tensor and spectrum twice, 1.29 GB: 200 us at the measured
// copy rate, 218 us measured); paired complex64 the TF32 pipe (864 instructions of 8-9 clocks per SM partition and unit,
// 110 us) plus the splits' instructions, which overlap with it only in part (178 us; the FP32 kernels of contract.cu
// take 180 to 293 us); single complex64 the same splits for half the products (142 us).
//
// Persistent CTAs with a ring of stages (one unit each, tensor with an L2 evict_first hint, and its spectrum).  NG
// groups of W warps take the units round-robin.  No barrier joins the warps: each waits for the stage, reads it,
// releases it and stores its own rows.  All waits are bounded (2 s, error codes 41 to 43).  The kernels do not let their
// dependents start early: with k_by's blocks waiting from the first wave on, k_by and k_bx after it took 52 and 33 us
// instead of 29 and 24 (complex128, 128x128x32; whole apply 343 -> 321 us, 64x128x27 151 -> 144, pair 277 -> 275).
#include <atomic>
#include <cstdint>
#include "common.cuh"
#include "ie_internal.h"
#include "tma.cuh"

namespace {

constexpr int kSmemMax = 232448;  // dynamic shared memory of one CTA

// complex128 shapes: KT1 tiles of 8 over the 2Nz (x, y) rows and columns, KT2 over the Nz z ones; one row tile per
// warp, W warps per unit, NG groups of them.
template <int KT1, int KT2, int NG_> struct MmaCfg64 {
    static constexpr int KT = KT1 + KT2, W = KT, NG = NG_, NTHREADS = NG * W * 32 + 32;  // and the producer
};
// complex64 shapes: KZ tiles of 8 z; a warp owns the x, y and z rows of one tile, W warps per unit.
template <int KZ, int NG_> struct MmaCfg32 {
    static constexpr int W = KZ, NG = NG_, NTHREADS = NG * W * 32;
};

struct MmaArgs {
    int Nz, Ny, pitch, nstage, stage_bytes;  // pitch: elements per spectrum row
    long long nunits;
};

G2_D void dmma(double (&c)[2], double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}
// d = a b + d over a k-tile of 8, or of 4 (a[0], a[1] and b0 only)
template <bool HALF> G2_D void tmma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    if constexpr (HALF)
        asm("mma.sync.aligned.m16n8k4.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(b0));
    else
        asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
G2_D float2 add2(float2 a, float2 b)
{
    union U { float2 f; unsigned long long u; } ua, ub, uc;
    ua.f = a;
    ub.f = b;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(uc.u) : "l"(ua.u), "l"(ub.u));
    return uc.f;
}
// d = a b
template <bool HALF> G2_D void tmma_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    if constexpr (HALF)
        asm("mma.sync.aligned.m16n8k4.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(b0), "f"(0.f));
    else
        asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// x = hi + lo: hi rounded to TF32 (11 significant bits), lo the exact rest, whose last bit or two the tensor core
// drops (2^-23 |x| at most, of either sign)
G2_D void split(float x, uint32_t &hi, uint32_t &lo)
{
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}
// x = hi + lo + rest exactly: lo rounded to TF32 too, the rest the last bit or two
G2_D void split3(float x, uint32_t &hi, uint32_t &lo, uint32_t &rest)
{
    uint32_t r;
    split(x, hi, r);
    split(__uint_as_float(r), lo, rest);
}
template <typename T> G2_D T at(const void *p, uint32_t bytes)
{
    return *reinterpret_cast<const T *>(reinterpret_cast<const char *>(p) + bytes);
}

// offset of M(row, k) in the packed unit; rows and k are (tile, index in tile) of the complex128 tiling
template <int KT1>
G2_D int mma_offset(int rt, int rn, int kt, int kn, int Nz, int P, int zero)
{
    int rc, rz, kc, kz;
    if (rt < KT1) {
        const int j = rt * 8 + rn;
        if (j >= 2 * Nz) return zero;
        rc = j >= Nz ? 1 : 0;
        rz = j - rc * Nz;
    } else {
        rc = 2;
        rz = (rt - KT1) * 8 + rn;
        if (rz >= Nz) return zero;
    }
    if (kt < KT1) {
        const int j = kt * 8 + kn;
        if (j >= 2 * Nz) return zero;
        kc = j >= Nz ? 1 : 0;
        kz = j - kc * Nz;
    } else {
        kc = 2;
        kz = (kt - KT1) * 8 + kn;
        if (kz >= Nz) return zero;
    }
    if (rc < 2 && kc < 2) return (rc + kc) * P + sym_pos<true>(rz, kz, Nz);
    if (rc == 2 && kc == 2) return 3 * P + sym_pos<true>(rz, kz, Nz);
    return rc < 2 ? 4 * P + rc * Nz * Nz + full_pos<true>(rz, kz, Nz) : 4 * P + kc * Nz * Nz + full_pos<true>(kz, rz, Nz);
}

// Spin (bounded, 2 s) until the stage's tag is ticket it; on timeout records `code` in *err.
G2_D bool wait_tag(const volatile int *tag, int it, int *err, int code)
{
    if (*tag == it) return true;
    const uint64_t t0 = globaltimer_ns();
    while (*tag != it) {
        if (globaltimer_ns() - t0 > 2000000000ull) {
            atomicCAS(err, 0, code);
            return false;
        }
    }
    return true;
}

// The stage ring: NG groups of W warps over the CTA's units; body(g, u, unit, release) works on one staged unit by one
// warp (g, u: its tensor and spectrum) and calls release() after its last shared-memory read.
// PROD: one more warp refills the stages.  Otherwise the warp that releases a stage last refills it: at 12 consumer
// warps of 168 registers a 13th warp would cost a fourth of the registers.
template <typename C, int W, int NG, bool PROD, class Body>
G2_D void mma_ring(unsigned char *smem, const C *G, C *Uhat, const MmaArgs &a, int u_elems, int T, int *err, Body body)
{
    const int nst = a.nstage, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, grp = warp / W;
    const uint32_t tbytes = (uint32_t)(T * sizeof(C)), ubytes = (uint32_t)(u_elems * sizeof(C));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + (size_t)nst * a.stage_bytes);
    uint64_t *empty = full + nst;                          // PROD
    int *out_cnt = reinterpret_cast<int *>(full + nst);    // else: warps that are done with the stage's unit
    volatile int *tag = out_cnt + nst;                     // and the ticket the stage holds or is being filled with
    if (tid == 0) {
        for (int s = 0; s < nst; s++) {
            mbar_init(&full[s], 1);
            if (PROD) {
                mbar_init(&empty[s], W);
            } else {
                out_cnt[s] = 0;
                tag[s] = s;
            }
        }
        fence_mbar_init();
    }
    for (int s = tid; s < nst; s += blockDim.x)  // the zero that padded entries of M point at
        reinterpret_cast<C *>(smem + (size_t)s * a.stage_bytes)[T + u_elems] = czero<C>();
    __syncthreads();
    const long long first = blockIdx.x, stride = gridDim.x;
    const int my_n = first < a.nunits ? (int)((a.nunits - 1 - first) / stride + 1) : 0;
    auto fill = [&](int slot, int it) {
        const long long unit = first + it * stride;
        unsigned char *st = smem + (size_t)slot * a.stage_bytes;
        mbar_arrive_expect_tx(&full[slot], tbytes + ubytes);
        bulk_g2s(st, G + unit * (long long)T, tbytes, &full[slot], l2_policy_evict_first());
        bulk_g2s(st + tbytes, Uhat + unit * (long long)u_elems, ubytes, &full[slot], l2_policy_evict_normal());
    };
    if (tid == (PROD ? NG * W * 32 : 0))
        for (int s = 0; s < nst && s < my_n; s++) fill(s, s);
    if (PROD && warp == NG * W) {
        if (lane == 0) {
            int slot = 0, round = 1, issued = min(nst, my_n);
            for (int it = nst; it < my_n; it++) {
                if (!mbar_wait_bounded(&empty[slot], (round - 1) & 1, err, 42)) {
                    // give up: every issued copy must land before the CTA may exit
                    for (int d = issued - nst; d < issued; d++) mbar_wait_bounded(&full[d % nst], (d / nst) & 1, err, 43);
                    return;
                }
                fill(slot, it);
                issued++;
                if (++slot == nst) {
                    slot = 0;
                    round++;
                }
            }
        }
        return;
    }
    int slot = grp % nst, round = grp / nst;
    for (int it = grp; it < my_n; it += NG) {
        // A parity wait cannot tell this round of the stage from the one before the last.  With a producer the stages
        // are a multiple of the groups, so this group has waited for the last round itself; without, the stage's tag
        // says that the last round is over.
        const bool ok = (PROD || wait_tag(&tag[slot], it, err, 42)) && mbar_wait_bounded(&full[slot], round & 1, err, 41);
        if (!__all_sync(0xffffffffu, ok)) {
            if (!PROD)  // give up: copies in flight must land before the CTA may exit
                for (int s = 0; s < nst; s++) mbar_wait_bounded(&full[s], (tag[s] / nst) & 1, err, 43, 200000000ull);
            return;
        }
        const unsigned char *g = smem + (size_t)slot * a.stage_bytes;
        body(g, g + tbytes, first + it * stride, [&] {
            __syncwarp();
            if (lane != 0) return;
            if (PROD) {
                mbar_arrive(&empty[slot]);
                return;
            }
            if (W > 1) {
                __threadfence_block();
                if (atomicAdd(&out_cnt[slot], 1) != W - 1) return;
                out_cnt[slot] = 0;
                __threadfence_block();
            }
            if (it + nst < my_n) {
                fill(slot, it + nst);
                tag[slot] = it + nst;
            }
        });
        for (slot += NG; slot >= nst; slot -= nst) round++;
    }
}

// a Nyquist point of the unit (they are kept zero)
G2_D bool is_nyquist(long long unit, int Ny, int slot_pt)
{
    const int q = (int)(unit / Ny), r = (int)(unit - (long long)q * Ny);
    return (q == 0 && (slot_pt & 2)) || (r == 0 && (slot_pt & 1));
}

// Lanes l and l ^ 4 hold the real (comp 0) and imaginary (comp 1) rows of one point: from their rows' products with
// Re M (r) and Im M (i), the complex output's part comp
template <typename R> G2_D R complex_part(R r, R i, int comp)
{
    const R p = __shfl_xor_sync(0xffffffffu, i, 4);
    return comp ? r + p : r - p;
}
// v0, v1: the lane's parts of outputs j and j + 1; comp 0 stores j, comp 1 stores j + 1
template <typename C, typename R> G2_D void store_pair(C *row, int j, R v0, R v1, bool ok, int comp)
{
    const R x = __shfl_xor_sync(0xffffffffu, comp ? v0 : v1, 4);
    if (ok) row[j + comp] = comp ? C{x, v1} : C{v0, x};
}

// ---- complex128 ------------------------------------------------------------------------------------------------
template <int KT1, int KT2, int NG_>
__global__ void __launch_bounds__(MmaCfg64<KT1, KT2, NG_>::NTHREADS, 1)
    k_contract_mma64(const double2 *__restrict__ G, double2 *__restrict__ Uhat, MmaArgs a, int *err, const int *gate)
{
    using Cfg = MmaCfg64<KT1, KT2, NG_>;
    constexpr int KT = Cfg::KT, W = Cfg::W;
    // A sum in one chain of FMAs has 1.2 to 1.5 times the error of the FP64 kernels it takes the place of.  Two chains (the
    // k halves of each tile) have a smaller one; blocks of four tiles, each added to the total, a smaller one still.
    // Time of one chain / two / blocks, 128x128: Nz = 20 91 / 91 / 99 us, 27 171 / 171 / 179, 32 216 / 219 / 218,
    // 40 313 / 329 / 331, 48 606 / 623 / 632, 57 964 / 1007 / 966: blocks where they cost no more than two chains.  Error on
    // random units: Nz = 32 3.3e-16 / 2.4e-16 / 2.1e-16 (contract.cu 2.2e-16), 48 4.0e-16 / 2.9e-16 / 2.1e-16 (3.1e-16).
    constexpr bool BLOCKED = KT == 12 || KT == 23;
    extern __shared__ __align__(128) unsigned char smem[];
    const int Nz = a.Nz, P = Nz * (Nz + 1) / 2, T = 4 * P + 2 * Nz * Nz, u_elems = 4 * a.pitch;
    const int lane = threadIdx.x & 31, rt = (threadIdx.x >> 5) % W;
    const int kl = lane & 3, nl = lane >> 2, pt = nl >> 1, comp = nl & 1;
    const double sz = (pt & 2) ? -1.0 : 1.0, sy = (pt & 1) ? -sz : sz;  // sx, sx m
    uint32_t off[KT];  // element offsets of the two k halves
#pragma unroll
    for (int kt = 0; kt < KT; kt++)
        off[kt] = (uint32_t)mma_offset<KT1>(rt, nl, kt, kl, Nz, P, T + u_elems) |
                  (uint32_t)mma_offset<KT1>(rt, nl, kt, kl + 4, Nz, P, T + u_elems) << 16;
    pdl_wait_only();  // the offsets above need nothing of the kernels before this one
    if (gate && *gate == 0) return;
    mma_ring<double2, W, NG_, true>(smem, G, Uhat, a, u_elems, T, err,
                              [&](const unsigned char *g, const unsigned char *us, long long unit, auto release) {
        const double *u = reinterpret_cast<const double *>(us) + 2 * pt * a.pitch + comp;
        double ar[2] = {0.0, 0.0}, ai[2] = {0.0, 0.0}, br[2] = {0.0, 0.0}, bi[2] = {0.0, 0.0};
#pragma unroll
        for (int kt = 0; kt < KT; kt++) {
            if (kt == KT1 && rt >= KT1) {  // the transposed blocks of out_z
                ar[0] = -ar[0];
                ar[1] = -ar[1];
                ai[0] = -ai[0];
                ai[1] = -ai[1];
                if constexpr (!BLOCKED) {
                    br[0] = -br[0];
                    br[1] = -br[1];
                    bi[0] = -bi[0];
                    bi[1] = -bi[1];
                }
            }
#pragma unroll
            for (int h = 0; h < 2; h++) {
                int k = (kt < KT1 ? kt : kt - KT1) * 8 + 4 * h + kl;
                double s;
                if (kt < KT1) {
                    // padded k read a row that exists (M is zero there); the first tiles lie in x for every Nz
                    if (kt == KT1 - 1) k = min(k, 2 * Nz - 1);
                    s = kt * 8 + 8 <= 4 * (KT1 - 1) + 1 || k < Nz ? 1.0 : sy;
                } else {
                    if (kt == KT - 1) k = min(k, Nz - 1);
                    k += 2 * Nz;
                    s = sz;
                }
                const double x = u[2 * k] * s;
                const double2 e = at<double2>(g, 16u * (h ? off[kt] >> 16 : off[kt] & 0xffffu));
                if (BLOCKED || h) {
                    dmma(br, x, e.x);
                    dmma(bi, x, e.y);
                } else {
                    dmma(ar, x, e.x);
                    dmma(ai, x, e.y);
                }
            }
            if (kt == KT - 1 || (BLOCKED && (kt % 4 == 3 || kt == KT1 - 1))) {
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    ar[q] += br[q];
                    ai[q] += bi[q];
                    br[q] = bi[q] = 0.0;
                }
            }
        }
        release();
        const int j = rt < KT1 ? rt * 8 + 2 * kl : 2 * Nz + (rt - KT1) * 8 + 2 * kl, lim = rt < KT1 ? 2 * Nz : 3 * Nz;
        double g0 = sz, g1 = sz;
        if (rt < KT1) {
            g0 = j < Nz ? 1.0 : sy;
            g1 = j + 1 < Nz ? 1.0 : sy;
        }
        if (is_nyquist(unit, a.Ny, pt)) ar[0] = ar[1] = ai[0] = ai[1] = 0.0;
        store_pair(Uhat + unit * (long long)u_elems + pt * a.pitch, j, complex_part(ar[0], ai[0], comp) * g0,
                   complex_part(ar[1], ai[1], comp) * g1, j + comp < lim, comp);
    });
}

// ---- complex64 -------------------------------------------------------------------------------------------------
// one real row component's sums: hi hi (FP32, rounded adds), the smaller products (in the tensor core)
template <int NP> struct Acc32 {
    float2 r[NP], i[NP];
    float sr[4], si[4];
    float2 tr, ti;  // NP = 1: lo hi sums
    G2_D void clear()
    {
#pragma unroll
        for (int k = 0; k < NP; k++) r[k] = i[k] = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 4; k++) sr[k] = si[k] = 0.f;
        tr = ti = make_float2(0.f, 0.f);
    }
};
// A fragment of one component of V (k-tile of 8 or 4); t: the third parts (TERMS = 3)
template <int NP, int TERMS> struct Vfrag {
    uint32_t h[4], l[4], t[TERMS == 3 ? 4 : 1];
};
template <int NP, int TERMS, bool HALF>
G2_D Vfrag<NP, TERMS> load_v(const float2 *u, int k0, int k1, float s, int comp)
{
    Vfrag<NP, TERMS> v{};
    // part q of the fragment's word (NP = 2), or of its words q and q + 1 (NP = 1: rows 0-7 hi, rows 8-15 lo)
    auto put = [&](int q, float x) {
        uint32_t h, l, t = 0u;
        if constexpr (TERMS == 3) split3(x * s, h, l, t);
        else split(x * s, h, l);
        v.h[q] = h;
        if constexpr (NP == 2) v.l[q] = l;
        else v.h[q + 1] = l;
        if constexpr (TERMS == 3) v.t[q] = t;
    };
    if constexpr (NP == 2) {
        const float2 u0 = u[k0];
        put(0, u0.x);
        put(1, u0.y);
        if constexpr (!HALF) {
            const float2 u1 = u[k1];
            put(2, u1.x);
            put(3, u1.y);
        }
    } else {
        put(0, reinterpret_cast<const float *>(u + k0)[comp]);
        if constexpr (!HALF) put(2, reinterpret_cast<const float *>(u + k1)[comp]);
    }
    return v;
}
template <int NP, int TERMS> G2_D Vfrag<NP, TERMS> negate(const Vfrag<NP, TERMS> &v)
{
    Vfrag<NP, TERMS> w{};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        w.h[k] = v.h[k] ^ 0x80000000u;
        w.l[k] = v.l[k] ^ 0x80000000u;
        if constexpr (TERMS == 3) w.t[k] = v.t[k] ^ 0x80000000u;
    }
    return w;
}
template <int TERMS> struct Mfrag {
    uint32_t rh[2], rl[2], ih[2], il[2], rt[TERMS == 3 ? 2 : 1], it[TERMS == 3 ? 2 : 1];
};
template <int TERMS, bool HALF> G2_D Mfrag<TERMS> load_m(const unsigned char *g, uint32_t o0, uint32_t o1)
{
    Mfrag<TERMS> m{};
    auto put = [&](int q, float2 e) {
        if constexpr (TERMS == 3) {
            split3(e.x, m.rh[q], m.rl[q], m.rt[q]);
            split3(e.y, m.ih[q], m.il[q], m.it[q]);
        } else {
            split(e.x, m.rh[q], m.rl[q]);
            split(e.y, m.ih[q], m.il[q]);
        }
    };
    put(0, at<float2>(g, o0));
    if constexpr (!HALF) put(1, at<float2>(g, o1));
    return m;
}
// The hi hi sums of one product over one z'-tile.  They start from zero and a rounded add takes them into Acc32, so a
// product is truncated once, at its own size; a part of the tensor or of the vector that is small or zero costs nothing.
// truncation: what that takes off on average, half a unit in the last place of a mantissa m of density 1 / (m ln 2),
// 2^-24 E[1 / m] = 2^-24 / (2 ln 2) = 4.3e-8.  It is added with the smaller products, before the last rounding.  Measured
// loss: random units and vectors 3.4e-8, one non-zero component 3.5e-8, a layered background's tensor 3.6e-8, coherent
// signs 4.0e-8; a vector with one non-zero layer loses nothing, since the sum of one product is exact, and gains it.  Sums
// of up to 12 z have part tiles whose few products leave fewer bits to lose: 2.4e-8 (Nz = 4) to 3.5e-8 (Nz = 8).
template <int TERMS> constexpr float truncation = TERMS == 3 ? 3.3e-8f : 4.3e-8f;
template <int NP> struct Sum32 {
    float r[4], i[4];
};
// s = hi hi part, c += smaller parts of V M^T for one tile
template <int NP, int TERMS, bool HALF>
G2_D void product(Sum32<NP> &s, Acc32<NP> &c, const Vfrag<NP, TERMS> &v, const Mfrag<TERMS> &m)
{
    tmma_zero<HALF>(s.r, v.h, m.rh[0], m.rh[1]);
    tmma_zero<HALF>(s.i, v.h, m.ih[0], m.ih[1]);
    tmma<HALF>(c.sr, v.h, m.rl[0], m.rl[1]);
    tmma<HALF>(c.si, v.h, m.il[0], m.il[1]);
    if constexpr (NP == 2) {
        tmma<HALF>(c.sr, v.l, m.rh[0], m.rh[1]);
        tmma<HALF>(c.si, v.l, m.ih[0], m.ih[1]);
    }
    if constexpr (TERMS == 3) {
        if constexpr (NP == 2) {
            tmma<HALF>(c.sr, v.l, m.rl[0], m.rl[1]);
            tmma<HALF>(c.si, v.l, m.il[0], m.il[1]);
        }
        tmma<HALF>(c.sr, v.h, m.rt[0], m.rt[1]);
        tmma<HALF>(c.si, v.h, m.it[0], m.it[1]);
        tmma<HALF>(c.sr, v.t, m.rh[0], m.rh[1]);
        tmma<HALF>(c.si, v.t, m.ih[0], m.ih[1]);
    }
}
template <int NP> G2_D void take(Acc32<NP> &c, const Sum32<NP> &s)
{
    c.r[0] = add2(c.r[0], make_float2(s.r[0], s.r[1]));
    c.i[0] = add2(c.i[0], make_float2(s.i[0], s.i[1]));
    if constexpr (NP == 2) {
        c.r[1] = add2(c.r[1], make_float2(s.r[2], s.r[3]));
        c.i[1] = add2(c.i[1], make_float2(s.i[2], s.i[3]));
    } else {
        c.tr = add2(c.tr, make_float2(s.r[2], s.r[3]));
        c.ti = add2(c.ti, make_float2(s.i[2], s.i[3]));
    }
}
// A lane's tensor offsets for one z'-tile: the symmetric, the full and the transposed full tile, two k halves each;
// 32-bit byte offsets, or 16-bit element offsets in pairs where the registers are short (PACK).
template <bool PACK> struct Offs {
    uint32_t v[PACK ? 3 : 6];
    G2_D void set(int i, int e0, int e1)
    {
        if constexpr (PACK) {
            v[i] = (uint32_t)e0 | (uint32_t)e1 << 16;
        } else {
            v[2 * i] = (uint32_t)sizeof(float2) * e0;
            v[2 * i + 1] = (uint32_t)sizeof(float2) * e1;
        }
    }
    G2_D uint32_t lo(int i) const { return PACK ? (v[i] & 0xffffu) * (uint32_t)sizeof(float2) : v[2 * i]; }
    G2_D uint32_t hi(int i) const { return PACK ? (v[i] >> 16) * (uint32_t)sizeof(float2) : v[2 * i + 1]; }
};
// All nine products of z-tile (rows) and z'-tile (columns).  LAST: the tile may hold padded k, whose offsets point at
// the zero z0 in every block (padded rows repeat the last row; they are not stored).  pb, fb: bytes of a symmetric and
// of a full block.
template <int NP, int TERMS, bool HALF, bool LAST, bool PACK>
G2_D void tile_products(Acc32<NP> (&acc)[3], const unsigned char *g, const float2 *u, int k0, int k1, int Nz, float sy,
                        float sz, int comp, const Offs<PACK> &of, uint32_t z0, uint32_t pb, uint32_t fb)
{
    const uint32_t o[6] = {of.lo(0), of.hi(0), of.lo(1), of.hi(1), of.lo(2), of.hi(2)};
    const uint32_t p0 = LAST && o[0] == z0 ? 0u : pb, p1 = LAST && o[1] == z0 ? 0u : pb;
    const uint32_t f0 = LAST && o[2] == z0 ? 0u : fb, f1 = LAST && o[3] == z0 ? 0u : fb;
    const uint32_t t0 = f0, t1 = f1;
    const Vfrag<NP, TERMS> vx = load_v<NP, TERMS, HALF>(u, k0, k1, 1.f, comp);
    const Vfrag<NP, TERMS> vy = load_v<NP, TERMS, HALF>(u + Nz, k0, k1, sy, comp);
    const Vfrag<NP, TERMS> vz = load_v<NP, TERMS, HALF>(u + 2 * Nz, k0, k1, sz, comp);
    Sum32<NP> s, t;
    auto mul = [&](Sum32<NP> &d, Acc32<NP> &a, const Vfrag<NP, TERMS> &v, uint32_t e0, uint32_t e1) {
        product<NP, TERMS, HALF>(d, a, v, load_m<TERMS, HALF>(g, e0, e1));
    };
    {
        const Mfrag<TERMS> m = load_m<TERMS, HALF>(g, o[0] + p0, o[1] + p1);  // xy
        product<NP, TERMS, HALF>(s, acc[0], vy, m);
        product<NP, TERMS, HALF>(t, acc[1], vx, m);
    }
    take(acc[0], s);
    take(acc[1], t);
    mul(s, acc[0], vx, o[0], o[1]);
    mul(t, acc[1], vy, o[0] + 2 * p0, o[1] + 2 * p1);
    take(acc[0], s);
    take(acc[1], t);
    mul(s, acc[0], vz, o[2], o[3]);
    mul(t, acc[1], vz, o[2] + f0, o[3] + f1);
    take(acc[0], s);
    take(acc[1], t);
    mul(s, acc[2], vx, o[4], o[5]);
    mul(t, acc[2], vy, o[4] + t0, o[5] + t1);
    take(acc[2], s);
    take(acc[2], t);
    mul(s, acc[2], negate(vz), o[0] + 3 * p0, o[1] + 3 * p1);  // acc[2] = -out_z
    take(acc[2], s);
}

// KZ tiles of 8 z; HALF: the last one holds at most 4
template <int NP, int KZ, bool HALF, int NG_>
__global__ void __launch_bounds__(MmaCfg32<KZ, NG_>::NTHREADS, 1)
    k_contract_mma32(const float2 *__restrict__ G, float2 *__restrict__ Uhat, MmaArgs a, int *err, const int *gate)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const int Nz = a.Nz, P = Nz * (Nz + 1) / 2, T = 4 * P + 2 * Nz * Nz, u_elems = 4 * NP * a.pitch;
    const int lane = threadIdx.x & 31, rt = (threadIdx.x >> 5) % KZ;
    const int kl = lane & 3, nl = lane >> 2;
    const int pt = NP == 2 ? nl : nl >> 1, comp = NP == 2 ? 0 : nl & 1, slot_pt = pt / NP;
    const float sz = (slot_pt & 2) ? -1.f : 1.f, sy = (slot_pt & 1) ? -sz : sz;  // sx, sx m
    const uint32_t z0 = sizeof(float2) * (T + u_elems), pb = sizeof(float2) * P, fb = sizeof(float2) * Nz * Nz;
    constexpr bool PACK = KZ >= 5;
    constexpr int TERMS = KZ == 1 || (KZ == 2 && HALF) ? 3 : 2;  // Nz <= 12
    Offs<PACK> off[KZ];
    {
        const int z = min(rt * 8 + nl, Nz - 1), zero = T + u_elems;
#pragma unroll
        for (int kt = 0; kt < KZ; kt++) {
            const int k0 = kt * 8 + kl, k1 = k0 + 4;
            off[kt].set(0, k0 < Nz ? sym_pos<false>(z, k0, Nz) : zero, k1 < Nz ? sym_pos<false>(z, k1, Nz) : zero);
            off[kt].set(1, k0 < Nz ? 4 * P + full_pos<false>(z, k0, Nz) : zero,
                        k1 < Nz ? 4 * P + full_pos<false>(z, k1, Nz) : zero);
            off[kt].set(2, k0 < Nz ? 4 * P + full_pos<false>(k0, z, Nz) : zero,
                        k1 < Nz ? 4 * P + full_pos<false>(k1, z, Nz) : zero);
        }
    }
    pdl_wait_only();
    if (gate && *gate == 0) return;
    mma_ring<float2, KZ, NG_, false>(smem, G, Uhat, a, u_elems, T, err,
                              [&](const unsigned char *g, const unsigned char *us, long long unit, auto release) {
        const float2 *u = reinterpret_cast<const float2 *>(us) + pt * a.pitch;
        Acc32<NP> acc[3];
#pragma unroll
        for (int c = 0; c < 3; c++) acc[c].clear();
#pragma unroll
        for (int kt = 0; kt < KZ - 1; kt++)
            tile_products<NP, TERMS, false, false, PACK>(acc, g, u, kt * 8 + kl, kt * 8 + kl + 4, Nz, sy, sz, comp, off[kt], z0, pb, fb);
        // padded k read an element that exists (M is zero there)
        tile_products<NP, TERMS, HALF, true, PACK>(acc, g, u, min((KZ - 1) * 8 + kl, Nz - 1), min((KZ - 1) * 8 + kl + 4, Nz - 1),
                                            Nz, sy, sz, comp, off[KZ - 1], z0, pb, fb);
        release();
        float2 *row = Uhat + unit * (long long)u_elems + pt * a.pitch;
        const int z = rt * 8 + 2 * kl;
        auto total = [](float hi, float small) { return hi + fmaf(hi, truncation<TERMS>, small); };
        if (is_nyquist(unit, a.Ny, slot_pt))
#pragma unroll
            for (int c = 0; c < 3; c++) acc[c].clear();
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const Acc32<NP> &q = acc[c];
            const float s = c == 0 ? 1.f : (c == 1 ? sy : -sz);
            float2 *dst = row + c * Nz;
            if constexpr (NP == 2) {
                if (z < Nz)
                    dst[z] = make_float2(total(q.r[0].x - q.i[1].x, q.sr[0] - q.si[2]) * s,
                                         total(q.r[1].x + q.i[0].x, q.sr[2] + q.si[0]) * s);
                if (z + 1 < Nz)
                    dst[z + 1] = make_float2(total(q.r[0].y - q.i[1].y, q.sr[1] - q.si[3]) * s,
                                             total(q.r[1].y + q.i[0].y, q.sr[3] + q.si[1]) * s);
            } else {
                const float v0 = total(complex_part(q.r[0].x, q.i[0].x, comp),
                                       complex_part(q.sr[0] + (q.sr[2] + q.tr.x), q.si[0] + (q.si[2] + q.ti.x), comp));
                const float v1 = total(complex_part(q.r[0].y, q.i[0].y, comp),
                                       complex_part(q.sr[1] + (q.sr[3] + q.tr.y), q.si[1] + (q.si[3] + q.ti.y), comp));
                store_pair(dst, z, v0 * s, v1 * s, z + comp < Nz, comp);
            }
        }
    });
}

int mma_sms()
{
    static const int n = [] {
        int dev = 0, v = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
        return v > 0 ? v : 1;
    }();
    return n;
}

// stages that fit, at most 16
template <typename C> constexpr int stage_bytes_of(int nz, int pts, int pitch)
{
    return (int)(((2 * nz * (2 * nz + 1) + pts * pitch + 1) * sizeof(C) + 127) / 128 * 128);
}
constexpr int stages_of(int bytes)
{
    const int n = (kSmemMax - 512) / (bytes + 16);
    return n > 16 ? 16 : n;
}

// all shared memory for a kernel, asked for until the call has succeeded once
template <class K> int allow_smem(K kern, std::atomic<bool> &ready)
{
    if (!ready) {
        G2_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
        ready = true;
    }
    return G2_OK;
}

template <typename C, class K>
int launch_mma(K kern, int nthreads, int multiple, int pts, const void *G, void *Uhat, int Nx, int Ny, int Nz, int *err,
               cudaStream_t st, const int *gate)
{
    MmaArgs a;
    a.Nz = Nz;
    a.Ny = Ny;
    a.pitch = ie_spectrum_pitch(Nz);
    a.nunits = (long long)Nx * Ny;
    a.stage_bytes = stage_bytes_of<C>(Nz, pts, a.pitch);
    a.nstage = stages_of(a.stage_bytes) / multiple * multiple;
    if (a.nstage < 1) return G2_ERR_UNSUPPORTED;
    const int sm = a.nstage * (a.stage_bytes + 16);
    const int grid = (int)(a.nunits < mma_sms() ? a.nunits : mma_sms());
    g2_launch(kern, grid, nthreads, sm, st, reinterpret_cast<const C *>(G), reinterpret_cast<C *>(Uhat), a, err, gate);
    G2_CUDA_CHECK(cudaGetLastError());
    return G2_OK;
}
template <int KT1, int KT2, int NG>
int launch_mma64(const void *G, void *U, int Nx, int Ny, int Nz, int *err, cudaStream_t st, const int *gate)
{
    auto kern = k_contract_mma64<KT1, KT2, NG>;
    static std::atomic<bool> ready{false};
    if (const int rc = allow_smem(kern, ready)) return rc;
    return launch_mma<double2>(kern, MmaCfg64<KT1, KT2, NG>::NTHREADS, NG, 4, G, U, Nx, Ny, Nz, err, st, gate);
}
template <int NP, int KZ, bool HALF, int NG>
int launch_mma32(const void *G, void *U, int Nx, int Ny, int Nz, int *err, cudaStream_t st, const int *gate)
{
    auto kern = k_contract_mma32<NP, KZ, HALF, NG>;
    static std::atomic<bool> ready{false};
    if (const int rc = allow_smem(kern, ready)) return rc;
    return launch_mma<float2>(kern, MmaCfg32<KZ, NG>::NTHREADS, 1, 4 * NP, G, U, Nx, Ny, Nz, err, st, gate);
}
// groups for about `want` warps, at most `most`
constexpr int pick_ng(int W, int want, int most)
{
    const int n = want / W < 1 ? 1 : want / W;
    return n < most ? n : (most < 1 ? 1 : most);
}
template <int KT1, int KT2> constexpr int ng64()
{
    constexpr int nz = 4 * KT1 < 57 ? 4 * KT1 : 57;  // the shape's largest
    return pick_ng(KT1 + KT2, 24, stages_of(stage_bytes_of<double2>(nz, 4, 3 * nz + 7)) / 2);
}
template <int NP, int KZ> constexpr int ng32()
{
    constexpr int nz = 8 * KZ < 57 ? 8 * KZ : 57;
    return pick_ng(KZ, KZ == 1 ? 16 : 12, stages_of(stage_bytes_of<float2>(nz, 4 * NP, 3 * nz + 7)));
}

int dispatch64(const void *G, void *U, int Nx, int Ny, int Nz, int *err, cudaStream_t st, const int *gate)
{
#define G2_M(K1, K2) \
    case K1: return launch_mma64<K1, K2, ng64<K1, K2>()>(G, U, Nx, Ny, Nz, err, st, gate)
    switch ((2 * Nz + 7) / 8) {
        G2_M(1, 1);
        G2_M(2, 1);
        G2_M(3, 2);
        G2_M(4, 2);
        G2_M(5, 3);
        G2_M(6, 3);
        G2_M(7, 4);
        G2_M(8, 4);
        G2_M(9, 5);
        G2_M(10, 5);
        G2_M(11, 6);
        G2_M(12, 6);
        G2_M(13, 7);
        G2_M(14, 7);
        G2_M(15, 8);
    default: return G2_ERR_UNSUPPORTED;
    }
#undef G2_M
}
template <int NP>
int dispatch32(const void *G, void *U, int Nx, int Ny, int Nz, int *err, cudaStream_t st, const int *gate)
{
#define G2_M(K) \
    case 2 * K: return launch_mma32<NP, K, true, ng32<NP, K>()>(G, U, Nx, Ny, Nz, err, st, gate); \
    case 2 * K + 1: return launch_mma32<NP, K, false, ng32<NP, K>()>(G, U, Nx, Ny, Nz, err, st, gate)
    switch ((Nz + 3) / 4 + 1) {  // quarter tiles of 4 z, in pairs
        G2_M(1);
        G2_M(2);
        G2_M(3);
        G2_M(4);
        G2_M(5);
        G2_M(6);
        G2_M(7);
        G2_M(8);
    default: return G2_ERR_UNSUPPORTED;
    }
#undef G2_M
}

}  // namespace

int ie_spectrum_pitch(int Nz) { return 3 * Nz + ((4 - 3 * Nz) % 8 + 8) % 8; }

int ie_contract_mma(int form, const void *G, void *Uhat, int Nx, int Ny, int Nz, int *err, cudaStream_t st,
                    const int *gate)
{
    if (form == 0) return dispatch64(G, Uhat, Nx, Ny, Nz, err, st, gate);
    if (form == 1) return dispatch32<1>(G, Uhat, Nx, Ny, Nz, err, st, gate);
    return dispatch32<2>(G, Uhat, Nx, Ny, Nz, err, st, gate);
}
