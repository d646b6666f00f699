// The quotients by a stored reciprocal (divBy, divByF), their operand ranges
// and the division by multiplication (FastDiv), compared with the plain
// operations: on the host (argument "host") what the host sets up, on the device
// (argument "device") what the kernels evaluate.  Prints one line per check and
// returns the number of those that failed.
#include "vxb_common.cuh"
#include "vxb_kernels.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <string>
#include <vector>

using namespace vxb;
using namespace vxb::detail;

namespace {

int failed = 0;

void check(const char* what, uint64_t bad, uint64_t n) {
    printf("%s: %llu of %llu differ\n", what, (unsigned long long)bad, (unsigned long long)n);
    failed += bad != 0;
}

double fromBits(uint64_t u) {
    double d;
    memcpy(&d, &u, 8);
    return d;
}

float fromBits32(uint32_t u) {
    float f;
    memcpy(&f, &u, 4);
    return f;
}

void hostChecks() {
    // The ranges: every exponent with the smallest and largest mantissa.
    uint64_t bad = 0, n = 0;
    for (uint64_t e = 0; e < 2048; ++e)
        for (uint64_t m : {uint64_t(0), (uint64_t(1) << 52) - 1})
            for (uint64_t s : {uint64_t(0), uint64_t(1) << 63}) {
                const double x = fromBits(s | (e << 52) | m);
                const bool want = std::fabs(x) >= std::ldexp(1.0, -400) && std::fabs(x) < std::ldexp(1.0, 400);
                bad += divScale(x) != want;
                bad += divReciprocal(x) != (want ? 1.0 / x : 0.0);
                ++n;
            }
    check("FP64 range", bad, n);
    bad = n = 0;
    for (uint32_t e = 0; e < 256; ++e)
        for (uint32_t m : {0u, (1u << 23) - 1u})
            for (uint32_t s : {0u, 1u << 31}) {
                const float x = fromBits32(s | (e << 23) | m);
                const bool want = std::fabs(x) >= std::ldexp(1.0f, -60) && std::fabs(x) < std::ldexp(1.0f, 60);
                bad += divScaleF(x) != want;
                bad += divReciprocalF(x) != (want ? 1.0f / x : 0.0f);
                ++n;
            }
    check("FP32 range", bad, n);
    // Divisors of 1 .. 2^27 - 1: n * mul >> 32 >> shift as the device does it.
    std::mt19937_64 rng(1);
    bad = n = 0;
    for (int k = 0; k < 4000; ++k) {
        const uint32_t d = k < 1000 ? (uint32_t)k + 1 : k < 1100 ? (1u << (1 + k % 26)) + (uint32_t)(k % 3) - 1u
                                                               : (uint32_t)(rng() % ((1u << 27) - 1u)) + 1u;
        const FastDiv f = FastDiv::of(d);
        for (int q = 0; q < 40; ++q) {
            uint32_t x = (uint32_t)(rng() & ((1u << 27) - 1u));
            if (q < 12) {
                const uint64_t at = (uint64_t)d * (q < 6 ? 1 : ((1u << 27) - 1u) / d) + (uint64_t)(q % 3) - 1u;
                x = at < (1u << 27) ? (uint32_t)at : (1u << 27) - 1u;
            }
            const uint32_t got = f.mul ? (uint32_t)(((uint64_t)x * f.mul) >> 32) >> f.shift : x;
            bad += got != x / d;
            ++n;
        }
    }
    check("FastDiv", bad, n);
}

__global__ void quotients(const double* x, const double* d, uint64_t n, unsigned long long* bad) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const double a = x[i], b = d[i];
        if (!divExact(a) || !divScale(b)) atomicAdd(bad + 1, 1ull);
        const double q = divBy(a, b, __drcp_rn(b)), want = __ddiv_rn(a, b);
        if (!(q == want)) atomicAdd(bad, 1ull);   // +0 equals -0
    }
}

__global__ void quotientsF(const float* x, const float* d, uint64_t n, unsigned long long* bad) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const float a = x[i], b = d[i];
        if (!divExactF(a) || !divScaleF(b)) atomicAdd(bad + 1, 1ull);
        const float q = divByF(a, b, __frcp_rn(b)), want = __fdiv_rn(a, b);
        if (!(q == want)) atomicAdd(bad, 1ull);
    }
}

__global__ void divisions(const uint32_t* x, const FastDiv* f, const uint32_t* d, uint64_t n, unsigned long long* bad) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        if (f[i].div(x[i]) != x[i] / d[i]) atomicAdd(bad, 1ull);
}

template <class T> T* upload(const std::vector<T>& v) {
    T* p = nullptr;
    if (cudaMalloc(&p, v.size() * sizeof(T)) != cudaSuccess ||
        cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) {
        printf("no device memory\n");
        exit(100);
    }
    return p;
}

void deviceChecks() {
    const uint64_t n = 1u << 22;
    std::mt19937_64 rng(2);
    unsigned long long* bad = upload(std::vector<unsigned long long>(2, 0ull));
    unsigned long long h[2];
    auto result = [&](const char* what, const char* range) {
        cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost);
        if (cudaGetLastError() != cudaSuccess) h[0] = ~0ull;
        check(what, h[0], n);
        if (range) check(range, h[1], n);
        cudaMemset(bad, 0, sizeof(h));
    };
    // Exponents over the whole range, a quarter of them at its ends; mantissas
    // random, with few set bits, and at the ends of the binade.
    auto mantissa = [&](uint32_t bits) -> uint64_t {
        const uint64_t top = (uint64_t(1) << bits) - 1;
        switch (rng() & 3u) {
        case 0: return rng() & top;
        case 1: return rng() & 15u;
        case 2: return top - (rng() & 15u);
        default: return ((uint64_t(1) << (rng() % bits)) | (uint64_t(1) << (rng() % bits))) & top;
        }
    };
    auto exponent = [&](int lim) { return (rng() & 3u) ? (int)(rng() % (2u * lim)) - lim : (rng() & 1u) ? -lim : lim - 1; };
    std::vector<double> x(n), d(n);
    std::vector<float> xf(n), df(n);
    for (uint64_t i = 0; i < n; ++i) {
        auto value = [&]() { return fromBits((rng() & (uint64_t(1) << 63)) | ((uint64_t)(1023 + exponent(400)) << 52) | mantissa(52)); };
        auto valueF = [&]() {
            return fromBits32((uint32_t)((rng() & 1u) << 31) | ((uint32_t)(127 + exponent(60)) << 23) | (uint32_t)mantissa(23));
        };
        x[i] = i % 1000 ? value() : i % 2000 ? 0.0 : -0.0;
        d[i] = value();
        xf[i] = i % 1000 ? valueF() : i % 2000 ? 0.0f : -0.0f;
        df[i] = valueF();
    }
    quotients<<<1024, 256>>>(upload(x), upload(d), n, bad);
    result("FP64 quotients", "FP64 operands out of range");
    quotientsF<<<1024, 256>>>(upload(xf), upload(df), n, bad);
    result("FP32 quotients", "FP32 operands out of range");
    std::vector<uint32_t> w(n), by(n);
    std::vector<FastDiv> f(n);
    for (uint64_t i = 0; i < n; ++i) {
        by[i] = (uint32_t)(rng() >> 37 >> (rng() % 27)) | 1u;
        w[i] = (uint32_t)(rng() >> 37);
        if (i % 4 == 0) w[i] = w[i] / by[i] * by[i];
        if (i % 4 == 1) w[i] = w[i] / by[i] * by[i] + by[i] - 1u < (1u << 27) ? w[i] / by[i] * by[i] + by[i] - 1u : w[i];
        f[i] = FastDiv::of(by[i]);
    }
    divisions<<<1024, 256>>>(upload(w), upload(f), upload(by), n, bad);
    result("divisions", nullptr);
}

}  // namespace

int main(int argc, char** argv) {
    if (argc > 1 && std::string(argv[1]) == "host") hostChecks();
    else deviceChecks();
    return failed;
}
