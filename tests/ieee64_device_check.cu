// csrc/ieee64.h on the device, with the device's own seeds, against its IEEE
// `/` and sqrt(): exit code 0 when every result is equal and every seed is
// within the 2^-19 that the proofs assume.  Operands: random and rounding-
// critical significands, exponents over the whole accepted range (quotients
// between 2^-1000 and 2^1000), neighbours of powers of two.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "ieee64.h"

struct Case {
    double a, d, x;
};

__device__ unsigned long long bad[5];
__device__ double worst[2];

__device__ bool same(double p, double q) { return __double_as_longlong(p) == __double_as_longlong(q) || p == q; }
__device__ void note(double e, int k) {  // non-negative doubles order like their bits
    atomicMax(reinterpret_cast<unsigned long long *>(worst) + k, (unsigned long long)__double_as_longlong(fabs(e)));
}

__global__ void check(const Case *c, long n) {
    using namespace tsu;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const double a = c[i].a, d = c[i].d, x = c[i].x;
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
        note(fma64(y, d, -1.0), 0);
        if (recip_ok(d)) {
            y = recip(d);
            if (!same(y, 1.0 / d)) atomicAdd(bad, 1ull);
            if (!same(quot(a, d, y), a / d)) atomicAdd(bad + 1, 1ull);
            // first quotients off by up to 2^-30
            const double off = ((double)(i % 2049) - 1024.0) * 0x1p-40;
            if (!same(quot_from(a, d, y, a / d * (1.0 + off)), a / d)) atomicAdd(bad + 2, 1ull);
            if (!same(quot(0.0, d, y), 0.0)) atomicAdd(bad + 2, 1ull);
        }
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
        note(y * sqrt(x) - 1.0, 1);
        if (!same(root(x), sqrt(x))) atomicAdd(bad + 3, 1ull);
        if (!same(root(0.0), 0.0)) atomicAdd(bad + 4, 1ull);
    }
}

static uint64_t s = 0x9e3779b97f4a7c15ull;
static uint64_t rnd() {
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return s;
}
static double value(int lo, int hi) {
    const uint64_t all = (1ull << 52) - 1;
    uint64_t m;
    switch (rnd() % 4) {
        case 0: m = (1ull << (rnd() % 52)) - 1; break;
        case 1: m = all & ~(rnd() % 64); break;
        case 2: m = rnd() % 64; break;
        default: m = rnd() & all;
    }
    const uint64_t u = ((uint64_t)(1023 + lo + (int)(rnd() % (uint64_t)(hi - lo + 1))) << 52) | m;
    double x;
    std::memcpy(&x, &u, 8);
    return x;
}

int main(int argc, char **argv) {
    const long n = argc > 1 ? std::atol(argv[1]) : 1 << 22;
    std::vector<Case> c(n);
    for (long i = 0; i < n; i++) {
        const int r = (i & 1) ? 799 : 40;
        Case &k = c[i];
        k.d = value(-r, r);
        do k.a = value(-r, r);
        while (std::abs(std::ilogb(k.a) - std::ilogb(k.d)) > 998);
        if (rnd() & 1) k.a = -k.a;
        if (rnd() & 1) k.d = -k.d;
        k.x = value(-r, r);
    }
    Case *dc = nullptr;
    if (cudaMalloc(&dc, n * sizeof(Case)) != cudaSuccess) return 2;
    if (cudaMemcpy(dc, c.data(), n * sizeof(Case), cudaMemcpyHostToDevice) != cudaSuccess) return 2;
    check<<<592, 256>>>(dc, n);
    unsigned long long b[5];
    double w[2];
    if (cudaMemcpyFromSymbol(b, bad, sizeof(b)) != cudaSuccess || cudaMemcpyFromSymbol(w, worst, sizeof(w)) != cudaSuccess)
        return 2;
    std::printf("wrong: reciprocals %llu quotients %llu, %llu roots %llu, %llu; seeds within 2^%.2f, 2^%.2f\n", b[0], b[1],
                b[2], b[3], b[4], std::log2(w[0]), std::log2(w[1]));
    return b[0] | b[1] | b[2] | b[3] | b[4] || w[0] > 0x1p-19 || w[1] > 0x1p-19;
}
