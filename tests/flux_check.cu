/*
 * A point's own flux as the sweep evaluates it (state_flux) against the
 * general form with the operators (state_flux_general), bit for bit, in the
 * global axes: random densities, pressures and directions, Mach numbers from 0
 * to 4 (every piece of erf up to 3.4); the three axes' half-range terms in other
 * axes (axes_core); the reconstruction's limiter and primitive state; and the
 * quotient and root that start from the quotient's
 * approximation against the operators.  Prints the counts and returns 1 if any
 * differs or too few states were taken.
 */
#include <cstdint>
#include <cstdio>

#include <cuda_runtime.h>

#include "../3d-mfcfd_b200/csrc/mfcfd_publish.cuh"

using namespace mfcfd;

__device__ double rnd(uint64_t &s) {
    s += 0x9e3779b97f4a7c15ull;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return (double)((z ^ (z >> 31)) >> 11) * 0x1p-53;
}
__device__ bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }
__device__ bool same(float a, float b) { return __float_as_int(a) == __float_as_int(b); }

// out: states taken, components that differ, quotients or roots that differ
template <typename R>
__global__ void check(int n, unsigned long long *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t s = 77 + 1000003ull * i;
    const double rho = exp2(20 * rnd(s) - 10), p = rho * exp2(6 * rnd(s) - 3);
    const double u = 4 * rnd(s) * sqrt(1.4 * p / rho), z = 2 * rnd(s) - 1, f = 6.283185307179586 * rnd(s);
    const double w = sqrt(1 - z * z), axis = rnd(s);
    double v[3] = {u * w * cos(f), u * w * sin(f), u * z};
    if (axis < 0.2) v[1] = 0.0;                   // along a plane of the axes
    if (axis < 0.1) v[2] = axis < 0.05 ? -0.0 : 0.0;
    const R U[5] = {(R)rho, (R)(rho * v[0]), (R)(rho * v[1]), (R)(rho * v[2]),
                    (R)(2.5 * p + 0.5 * rho * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]))};
    FrameT<R> G;
    for (int r = 0; r < 3; ++r) { G.t1[r] = r == 0; G.t2[r] = r == 1; G.n[r] = r == 2; }
    int taken = 0, wrong = 0;
    for (int k = 0; k < 30; ++k) {
        bool ok = true;
        const R a = state_flux(k / 5, k % 5, U, ok);
        if (!ok) continue;
        ++taken;
        if (!same(a, state_flux_general(k / 5, k % 5, U, G, G))) ++wrong;
    }
    atomicAdd(out, (unsigned long long)taken);
    if (wrong) atomicAdd(out + 1, (unsigned long long)wrong);
    // the three axes' terms in turned axes
    FrameT<R> H;
    for (int r = 0; r < 3; ++r) { H.t1[r] = (R)(r == 1 ? 0.6 : r == 2 ? 0.8 : 0); H.t2[r] = r == 0; H.n[r] = (R)(r == 1 ? 0.8 : r == 2 ? -0.6 : 0); }
    const R prim[5] = {(R)rho, (R)v[0], (R)v[1], (R)v[2], (R)p};
    FluxPreT<R> P, Q;
    AxisTermsT<R> A[3], B[3];
    R ysp;
    bool ok = true;
    pre_core(prim, H, P, ysp, ok);
    axes_core(P, ysp, A, ok);
    flux_pre(prim, H, Q);
    for (int a = 0; a < 3; ++a) {
        axis_terms(Q, a, B[a]);
        if (!ok || !same(A[a].B, B[a].B) || !same(A[a].Ap, B[a].Ap) || !same(A[a].An, B[a].An)) atomicAdd(out + 1, 1ull);
    }
    // q -> primitive, and the limiter near its threshold and its ratio of one
    const double be = 0.5 * rho / p;
    const R qt[5] = {(R)(log(rho) + 2.5 * log(be) - be * u * u), (R)(2 * be * v[0]), (R)(2 * be * v[1]), (R)(2 * be * v[2]),
                     (R)(-2 * be)};
    R pa[5], pb[5];
    ok = true;
    prim_core(qt, pa, ok);
    qtilde_to_primitive(qt, pb);
    for (int r = 0; ok && r < 5; ++r)
        if (r && !same(pa[r], pb[r]) || !same(pa[0], pb[0])) atomicAdd(out + 1, 1ull);
    const R q = qt[0], temp = (R)(exp2(-30 * rnd(s)) * (rnd(s) < 0.5 ? -1 : 1)), eps2 = (R)(1e-6 * rnd(s));
    const R hi = (R)(q + (rnd(s) < 0.2 ? 0 : exp2(-25 * rnd(s)))), lo = (R)(q - (rnd(s) < 0.2 ? 0 : exp2(-25 * rnd(s))));
    ok = true;
    const R phi = limiter_core(q, temp, hi, lo, eps2, ok);
    const R neg = (q - R(0.5) * temp) - q, pos = neg > R(0) ? hi - q : lo - q;
    R want = R(1);
    if (!(r_abs(neg) <= R(MF_LIM_EPS))) {
        R num = (pos * pos) + eps2, den = pos * pos + R(2) * neg * neg;
        num = num * neg + R(2) * neg * neg * pos;
        den = den + neg * pos + eps2;
        den = den * neg;
        want = num / den < R(1) ? num / den : R(1);
    }
    if (ok && !same(phi, want)) atomicAdd(out + 1, 1ull);
    if constexpr (sizeof(R) == 8) {
        double q0;
        const double qb = quot_seed(0.5 * rho, p, q0), x = MF_PI * qb;
        if (!same(qb, 0.5 * rho / p) || !same(sqrt_from(qb, rsqrt_seed(q0)), sqrt(qb)) ||
            !same(sqrt_from(x, rsqrt_seed(MF_PI * q0)), sqrt(x)))
            atomicAdd(out + 2, 1ull);
        // all-ones denominators, and numerators next to a quotient's midpoint
        const double b = __longlong_as_double(__double_as_longlong(p) | 0xfffffffffffffll);
        const double m = __longlong_as_double(__double_as_longlong(rho) | 1), h = (m - __longlong_as_double(__double_as_longlong(m) - 1)) * 0.5;
        const double c = i & 1 ? b : p, a = __fma_rn(m, c, h * c);
        if (!same(quot_seed(a, c, q0), a / c)) atomicAdd(out + 2, 1ull);
    }
}

int main() {
    const int n = 1 << 20;
    unsigned long long *out = nullptr, h[6];
    if (cudaMalloc(&out, sizeof h) != cudaSuccess || cudaMemset(out, 0, sizeof h) != cudaSuccess) return 2;
    check<double><<<n / 256, 256>>>(n, out);
    check<float><<<n / 256, 256>>>(n, out + 3);
    if (cudaMemcpy(h, out, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    cudaFree(out);
    std::printf("FP64 taken %llu wrong %llu, quotients and roots wrong %llu; FP32 taken %llu wrong %llu\n", h[0], h[1], h[2], h[3],
                h[4]);
    return h[1] || h[2] || h[4] || h[0] < 25ull * n || h[3] < 25ull * n ? 1 : 0;
}
