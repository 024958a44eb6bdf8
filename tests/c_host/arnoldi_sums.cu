// Sums of the Krylov kernels of libgiem2g_b200 on vectors of one repeated value, whose exact sums are known and whose
// roundings do not average out: prints the relative error of ||w||^2 after an Arnoldi step on a zero basis, and of ||v||
// after the cycle start.   arnoldi_sums <elements> <basis vectors> <instances> <re> <im>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "krylov_dev.cuh"

#define CHECK(x)                                                                         \
    do {                                                                                 \
        const cudaError_t e_ = (x);                                                      \
        if (e_ != cudaSuccess) {                                                         \
            std::printf("%s:%d %s\n", __FILE__, __LINE__, cudaGetErrorString(e_));       \
            return 1;                                                                    \
        }                                                                                \
    } while (0)

__global__ void fill(float2 *p, size_t n, float2 v)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) p[i] = v;
}

template <typename T> T *alloc(size_t n)
{
    T *p = nullptr;
    if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess || cudaMemset(p, 0, n * sizeof(T)) != cudaSuccess) std::exit(2);
    return p;
}

int main(int argc, char **argv)
{
    if (argc != 6) return 3;
    const size_t N = std::strtoull(argv[1], nullptr, 10);
    const int K = std::atoi(argv[2]), n = std::atoi(argv[3]), nparts = 296, m = 31;
    const float2 v = make_float2((float)std::atof(argv[4]), (float)std::atof(argv[5]));
    if (K < 1 || K > m || n < 1 || n > KMI) return 3;
    Multi<float2> mm{};
    Starts<float2> st{};
    int *err = alloc<int>(1);
    for (int y = 0; y < n; y++) {
        Level L;
        L.m = m;
        L.H = alloc<double2>((m + 1) * (m + 1));
        L.cs = alloc<double>(m + 1);
        L.sn = alloc<double2>(m + 1);
        L.y = alloc<double2>(KMAX + 1);
        L.scal = alloc<double>(S_NSCAL);
        L.flags = alloc<int>(F_NFLAGS);
        L.counter = alloc<unsigned>(1);
        L.bar = alloc<unsigned>(1);
        mm.L[y] = st.L[y] = L;
        mm.V[y] = alloc<float2>(N * (K + 1));
        mm.w[y] = alloc<float2>(N);
        mm.part[y] = st.part[y] = alloc<double2>(2 * (size_t)nparts * (KMAX + 1));
        fill<<<1184, 256>>>(mm.w[y], N, v);
        st.v[y] = st.x0[y] = mm.w[y];
        st.x[y] = st.r[y] = mm.V[y] + N * K;  // overwritten by the step
        st.V[y] = mm.V[y];
    }
    CHECK(cudaDeviceSynchronize());
    const double exact = (double)N * ((double)v.x * v.x + (double)v.y * v.y);
    if (krylov_begin(st, n, N, nparts, err, (cudaStream_t)0)) return 4;
    CHECK(cudaDeviceSynchronize());
    double worst = 0.0, worst_bn = 0.0, bn, nrm;
    for (int y = 0; y < n; y++) {
        CHECK(cudaMemcpy(&bn, mm.L[y].scal + S_BN, sizeof(double), cudaMemcpyDeviceToHost));
        worst_bn = std::fmax(worst_bn, std::fabs(bn * bn / exact - 1.0));
    }
    if (arnoldi_step(mm, n, N, nparts, K - 1, 0.0, err, (cudaStream_t)0)) return 4;
    CHECK(cudaDeviceSynchronize());
    for (int y = 0; y < n; y++) {
        CHECK(cudaMemcpy(&nrm, mm.L[y].scal + S_NRM2, sizeof(double), cudaMemcpyDeviceToHost));
        worst = std::fmax(worst, std::fabs(nrm / exact - 1.0));
    }
    int e = 0;
    CHECK(cudaMemcpy(&e, err, sizeof(int), cudaMemcpyDeviceToHost));
    std::printf("%d %.6e %.6e\n", e, worst, worst_bn);
    return 0;
}
