// Test program: the FP64 step's short quotients (divide_by, quotient, divide_all and the ranges in
// which they are taken, clip_b200/csrc/lattice.cuh) against plain division on the device, and the
// update with the short forms against the update without.  Two results agree when they are the
// same double, zeros of either sign and NaNs among themselves.  Prints one line per check and
// exits non-zero if any differs.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "lattice.cuh"

using namespace clipb;

__device__ bool same(double a, double b) { return a == b || (a != a && b != b); }

// every value over the constants and over every density
__global__ void by_constants(const double* v, int n, int* bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = v[i], m = fabs(x);
    if (!(m == 0.0 || (m >= 0x1p-950 && m < 0x1p950))) return;
    if (!same(divide_by<6>(x), x / 6.0) || !same(divide_by<36>(x), x / 36.0) || !same(divide_by<72>(x), x / 72.0) ||
        !same(divide_by<144>(x), x / 144.0))
        atomicAdd(bad, 1);
}
__global__ void by_density(const double* v, int n, const double* rho, int m, int* bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int k = 0; k < m; ++k) {
        double a[3] = {v[i], v[(i + 1) % n], -v[(i + 7) % n]};
        const double want[3] = {a[0] / rho[k], a[1] / rho[k], a[2] / rho[k]};
        divide_all<3, double>(a, rho[k], all_in_range<3, 500>(a));
        for (int d = 0; d < 3; ++d)
            if (!same(a[d], want[d])) atomicAdd(bad, 1);
    }
}
template <int E>
__device__ bool range_ok(double x) {
    const double m = fabs(x);
    return in_range<E>(x) == (m == 0.0 || (m >= ldexp(1.0, -E) && m < ldexp(1.0, E)));
}
__global__ void ranges(const double* v, int n, int* bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && !(range_ok<100>(v[i]) && range_ok<200>(v[i]) && range_ok<500>(v[i]))) atomicAdd(bad, 1);
}

// One update per node, state = Q f, DIM u, c, mu, DIM grad c.
template <int DIM>
__global__ void update(Phys<double> P, const double* state, int n, int* bad, int* taken) {
    constexpr int Q = Lat<DIM>::Q, S = Q + 2 * DIM + 2;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* s = state + (long long)i * S;
    const double c = s[Q + DIM], mu = s[Q + DIM + 1];
    double f[Q], dc[3] = {0.0, 0.0, 0.0};
    for (int q = 0; q < Q; ++q) f[q] = s[q];
    for (int d = 0; d < DIM; ++d) dc[d] = s[Q + DIM + 2 + d];
    double u[2][3], p[2], rho[2], out[2][Q];
    for (int k = 0; k < 2; ++k) {
        for (int d = 0; d < DIM; ++d) u[k][d] = s[Q + d];
        const bool in = k && all_in_range<Q, 500>(f) && all_in_range<DIM, 200>(u[k]);
        if (in) atomicAdd(taken, 1);
        macroscopic<DIM, double>(P, f, c, mu, dc, u[k], p[k], rho[k], in);
        collide_f<DIM, double>(P, f, c, mu, dc, rho[k], p[k], u[k], out[k], in);
    }
    for (int d = 0; d < DIM; ++d)
        if (!same(u[0][d], u[1][d])) atomicAdd(bad, 1);
    for (int q = 0; q < Q; ++q)
        if (!same(out[0][q], out[1][q])) atomicAdd(bad, 1);
}

static int *g_bad, g_fail = 0;
static void report(const char* name, int n) {
    int bad[2] = {-1, -1};
    const cudaError_t e = cudaMemcpy(bad, g_bad, sizeof(bad), cudaMemcpyDeviceToHost);
    cudaMemset(g_bad, 0, sizeof(bad));
    std::printf("%s: %d of %d differ, short form %d (%s)\n", name, bad[0], n, bad[1], cudaGetErrorString(e));
    if (e != cudaSuccess || bad[0]) g_fail = 1;
}
static double* device(const std::vector<double>& v) {
    double* d = nullptr;
    if (cudaMalloc(&d, v.size() * sizeof(double)) != cudaSuccess) return nullptr;
    cudaMemcpy(d, v.data(), v.size() * sizeof(double), cudaMemcpyHostToDevice);
    return d;
}

template <int DIM>
static void updates(std::mt19937_64& rng) {
    constexpr int Q = Lat<DIM>::Q, S = Q + 2 * DIM + 2, N = 1 << 16;
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    Phys<double> P{};
    P.RhoL = 0.001, P.RhoH = 1.0, P.drho = 0.999, P.drho3 = 0.333;
    P.tauL = 0.3, P.tauH = 0.05, P.dtau = -0.25, P.kappa = 0.01, P.beta4 = 0.2, P.mobility = 0.02, P.W = 4.0;
    P.g[1] = -1e-6;
    std::vector<double> st((size_t)N * S);
    for (int i = 0; i < N; ++i) {
        double* s = st.data() + (size_t)i * S;
        // ordinary states, with zeros among them, and ever smaller ones down to the ranges' ends
        const int kind = i % 8, down = kind < 4 ? 0 : -(int)(rng() % 560);
        for (int q = 0; q < Q; ++q) s[q] = kind == 0 ? 0.0 : std::ldexp(0.1 * U(rng), down);
        for (int d = 0; d < DIM; ++d) s[Q + d] = kind < 2 ? 0.0 : std::ldexp(0.05 * U(rng), down / 3);
        // c over and beyond [0, 1]; now and then where the density is zero or nearly so
        s[Q + DIM] = i % 97 == 0 ? -P.RhoL / P.drho : 0.5 + 0.6 * U(rng);
        s[Q + DIM + 1] = 0.01 * U(rng);
        for (int d = 0; d < DIM; ++d) s[Q + DIM + 2 + d] = kind == 1 ? 0.0 : std::ldexp(0.2 * U(rng), down / 2);
    }
    double* d = device(st);
    update<DIM><<<N / 128, 128>>>(P, d, N, g_bad, g_bad + 1);
    report(DIM == 2 ? "2D update" : "3D update", N * (Q + DIM));
    cudaFree(d);
}

int main() {
    if (cudaMalloc(&g_bad, 2 * sizeof(int)) != cudaSuccess || cudaMemset(g_bad, 0, 2 * sizeof(int)) != cudaSuccess) {
        std::printf("no device\n");
        return 2;
    }
    std::mt19937_64 rng(3);
    std::vector<double> v = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, -2.2250738585072014e-308, 1.7976931348623157e308};
    for (int e : {-950, -500, -200, -100, -1, 0, 1, 100, 200, 500, 949})
        for (double m : {1.0, std::nextafter(1.0, 0.0), std::nextafter(1.0, 2.0), 1.5, std::nextafter(2.0, 0.0)})
            for (double sg : {1.0, -1.0}) v.push_back(sg * std::ldexp(m, e));
    for (int i = 0; i < 100000; ++i) {
        const double m = i % 3 ? 1.0 + std::ldexp((double)(rng() >> 12), -52) : (double)(1 + rng() % 4096);
        v.push_back((rng() & 1 ? 1.0 : -1.0) * std::ldexp(m, (int)(rng() % 1100) - (i % 2 ? 600 : 550)));
    }
    std::vector<double> rho = {1.0, 0.001, 1.0 / 3.0, 0.0, -0.0, INFINITY, NAN, 0x1p-100, std::nextafter(0x1p-100, 0.0), 0x1p100,
                               std::nextafter(0x1p100, 0.0), std::nextafter(1.0, 0.0), std::nextafter(1.0, 2.0), -0.002};
    for (int i = 0; i < 40; ++i) rho.push_back(std::ldexp(1.0 + std::ldexp((double)(rng() >> 12), -52), -(int)(rng() % 12)));
    const int n = (int)v.size(), blocks = (n + 127) / 128;
    double *dv = device(v), *dr = device(rho);
    if (!dv || !dr) return 2;
    by_constants<<<blocks, 128>>>(dv, n, g_bad);
    report("by constants", n);
    by_density<<<blocks, 128>>>(dv, n, dr, (int)rho.size(), g_bad);
    report("by density", 3 * n * (int)rho.size());
    ranges<<<blocks, 128>>>(dv, n, g_bad);
    report("ranges", n);
    updates<2>(rng);
    updates<3>(rng);
    return g_fail;
}
