// rcp64, sqrt64 and sqrt_rsqrt64 (sph_pair64.cuh) on the device against extended precision on the host: every binary
// exponent, both ends of the range that takes the short iterations, denormals, zero, infinity and NaN.  Prints the
// largest error of each, in units of 2^-53 of the result.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "../../fdps_sph_gb300/csrc/sph_pair64.cuh"

__global__ void k_roots(int n, const double *x, double *rcp, double *root, double *r, double *y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    rcp[i] = sph::rcp64(x[i]);
    root[i] = sph::sqrt64(x[i]);
    sph::sqrt_rsqrt64(x[i], r[i], y[i]);
}

static int bad = 0;

struct Worst {
    const char *name;
    double limit, err = 0.0, at = 0.0;
    void add(double x, double got, long double want) {
        if (std::isnan(want) ? std::isnan(got) : (double)want == got) return;
        const double e = std::isfinite(got) ? (double)(fabsl((long double)got - want) / fabsl(want)) * 0x1p53 : INFINITY;
        if (!(e <= err)) err = e, at = x;
    }
    void print() {
        std::printf("%s %.3f at %a%s\n", name, err, at, err <= limit ? "" : " ABOVE ITS LIMIT");
        bad += !(err <= limit);
    }
};

int main() {
    std::vector<double> x;
    std::mt19937_64 rng(7);
    for (int e = -1074; e <= 1023; ++e)
        for (int k = 0; k < 400; ++k) {
            const double m = 1.0 + (double)(rng() >> 12) * 0x1p-52;
            x.push_back(std::ldexp(k == 0 ? 1.0 : (k == 1 ? 2.0 - 0x1p-52 : m), e));
        }
    for (double edge : {0x1p-767, 0x1p768, 0x1p-1022})
        for (double v : {std::nextafter(edge, 0.0), edge, std::nextafter(edge, INFINITY)}) x.push_back(v);
    for (double v : {0.0, -0.0, (double)INFINITY, (double)NAN, -1.0, -0x1p-1074, 0x1p-1074}) x.push_back(v);
    const int n = (int)x.size();
    double *d[5];
    std::vector<double> out[4];
    for (auto &p : d)
        if (cudaMalloc((void **)&p, n * sizeof(double)) != cudaSuccess) return 2;
    cudaMemcpy(d[0], x.data(), n * sizeof(double), cudaMemcpyHostToDevice);
    k_roots<<<(n + 255) / 256, 256>>>(n, d[0], d[1], d[2], d[3], d[4]);
    for (int k = 0; k < 4; ++k) {
        out[k].resize(n);
        if (cudaMemcpy(out[k].data(), d[k + 1], n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    }
    // one rounding is 1 unit at most (of a result just above a power of two).  The reciprocal and the root of
    // sqrt_rsqrt64 add the iteration's own error and its products' roundings; sqrt64 ends on the exact residual.
    Worst rcp{"rcp64", 2.0}, root{"sqrt64", 1.01}, r{"sqrt_rsqrt64 root", 2.0}, y{"sqrt_rsqrt64 reciprocal root", 2.0};
    for (int i = 0; i < n; ++i) {
        const long double v = x[i];
        // 1 / x is denormal or infinite for the largest and smallest x: the double's own division, rounded once
        const double q = 1.0 / x[i];
        if (std::isnormal(q)) rcp.add(x[i], out[0][i], 1.0L / v);
        else rcp.add(x[i], out[0][i], q);
        if (x[i] < 0.0) {
            if (!std::isnan(out[1][i]) || !std::isnan(out[2][i])) root.err = INFINITY, root.at = x[i];
            continue;
        }
        root.add(x[i], out[1][i], sqrtl(v));
        r.add(x[i], out[2][i], sqrtl(v));
        if (x[i] > 0.0 || std::isnan(x[i])) y.add(x[i], out[3][i], 1.0L / sqrtl(v));
        else if (out[3][i] != 0.0) y.err = INFINITY, y.at = x[i];   // (a pair at one place has no direction)
    }
    rcp.print();
    root.print();
    r.print();
    y.print();
    return bad != 0;
}
