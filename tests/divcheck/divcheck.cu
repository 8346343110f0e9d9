// divcheck.cu -- csrc/bh_div.cuh against CUDA's own FP64 division and square
// root, bit for bit, with the operands and the approximations its callers
// pass (test code only; compiled by tests/test_gpu_division.py).
#include <stdint.h>
#include "bh_div.cuh"

namespace {
enum { C_RCP, C_DIV, C_SQRT, C_ISQRT, C_INV2, C_INV4, C_INV3, C_NEAR, C_N };

__device__ uint64_t mix(uint64_t& s) {   // splitmix64 (Steele, Lea & Flood 2014)
    uint64_t z = (s += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__device__ double with_exponent(uint64_t bits, int e) {   // significand of `bits`, 2^e
    return __longlong_as_double((int64_t)((bits & 0x000fffffffffffffull) | ((uint64_t)(e + 1023) << 52)));
}
// significands of several kinds: any, few bits set, near a power of two, near all ones
__device__ double operand(uint64_t& s, int e) {
    uint64_t m = mix(s), k = mix(s);
    switch (k & 7) {
    case 0: m &= mix(s) & mix(s) & mix(s); break;
    case 1: m = (k >> 8) & 15; break;
    case 2: m = ~((k >> 8) & 15); break;
    case 3: m &= ~0ull << ((k >> 8) & 63); break;
    default: break;
    }
    return with_exponent(m, e);
}
__device__ int exponent(uint64_t& s, int range) { return (int)(mix(s) % (uint64_t)(2 * range + 1)) - range; }

struct Out {
    unsigned long long* count;   // [C_N] mismatches
    double* first;               // [C_N][2] operands of one of them
};
__device__ void same(const Out& o, int c, double got, double want, double a, double b) {
    if (__double_as_longlong(got) == __double_as_longlong(want)) return;
    if (atomicAdd(o.count + c, 1ull) == 0) { o.first[2 * c] = a; o.first[2 * c + 1] = b; }
}

__device__ void check_quotient(const Out& o, double a, double b) {
    const double y = bh::rcp_any(b);
    same(o, C_RCP, y, 1.0 / b, 1.0, b);
    same(o, C_DIV, bh::div_by(a, b, y), a / b, a, b);
    same(o, C_DIV, bh::div_pos(fabs(a), fabs(b), fabs(y)), fabs(a) / fabs(b), fabs(a), fabs(b));
}
// a square root, its reciprocal, and h / x with the reciprocal's square near
// 1 / x (the lapse and the shift's factor)
__device__ void check_root(const Out& o, double x, double h) {
    double i2;
    const double s = bh::sqrt_rn(x, i2), inv = bh::rcp_refine_any(s, 2.0 * i2);
    same(o, C_SQRT, s, sqrt(x), x, 0.0);
    same(o, C_ISQRT, inv, 1.0 / sqrt(x), x, 0.0);
    same(o, C_NEAR, bh::div_by(h, x, bh::rcp_refine_any(x, inv * inv)), h / x, h, x);
}
// con2prim's chain from om = 1 - v^2 in [2^-53, 1] and xi
__device__ void check_chain(const Out& o, double om, double xi) {
    if (bh::all_ones(om)) return;
    const double z = bh::rcp_rn(om);
    if (!bh::all_ones(z)) {
        const double il2 = bh::rcp_polish(z, om), l4 = z * z;
        same(o, C_INV2, il2, 1.0 / z, om, z);
        if (!bh::all_ones(l4)) same(o, C_INV4, bh::rcp_refine(l4, il2 * il2), 1.0 / l4, om, l4);
    }
    const double X = xi * xi, xX = xi * X;
    if (!bh::all_ones(X) && !bh::all_ones(xX)) {
        const double iX = bh::rcp_rn(X);
        same(o, C_INV3, bh::rcp_refine(xX, xi * iX * iX), 1.0 / xX, xi, xX);
    }
}

__global__ void k_random(int64_t n, uint64_t seed, Out o) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
        uint64_t s = seed + (uint64_t)t * 0xd1342543de82ef95ull;
        const double sa = mix(s) & 1 ? -1.0 : 1.0, sb = mix(s) & 1 ? -1.0 : 1.0;
        double a = sa * operand(s, exponent(s, 249));
        if ((mix(s) & 63) == 0) a = sa * 0.0;
        check_quotient(o, a, sb * operand(s, exponent(s, 249)));
        check_quotient(o, sa, sb * operand(s, exponent(s, 499)));   // the ends of the range
        check_root(o, operand(s, exponent(s, 249)), sa * operand(s, exponent(s, 200)));
        check_root(o, 1.0 + operand(s, exponent(s, 30)), operand(s, exponent(s, 30)));   // 1 + 2 H, W^2
        const double om = operand(s, -1 - (int)(mix(s) % 52));
        check_chain(o, om, operand(s, exponent(s, 49)));
    }
}
// divisors b whose reciprocals lie next to a midpoint of two doubles
__global__ void k_list(const double* b, int n, uint64_t seed, Out o) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    uint64_t s = seed + t;
    const double q = with_exponent((uint64_t)__double_as_longlong(b[t]), 0);
    for (int e = -3; e <= 3; e++) {
        const double d = e < 0 ? q / (1 << -e) : q * (1 << e);
        for (int k = 0; k < 64; k++) check_quotient(o, operand(s, k - 32), d);
        check_root(o, d, operand(s, 0));
        int64_t x = __double_as_longlong(d * d);   // every x near d^2, so every one with the root d
        for (int k = -8; k <= 8; k++) check_root(o, __longlong_as_double(x + k), 1.0);
        x = __double_as_longlong(1.0 / d);
        for (int k = -8; k <= 8; k++) {            // om with 1 / om = d, where d is in its range
            const double om = __longlong_as_double(x + k);
            if (om <= 1.0) check_chain(o, om, d);
        }
        x = __double_as_longlong(cbrt(d));
        for (int k = -8; k <= 8; k++) check_chain(o, 0.75, __longlong_as_double(x + k));   // xi with xi^3 near d
        x = __double_as_longlong(1.0 / sqrt(d));
        for (int k = -8; k <= 8; k++) {            // om with om^-2 near d
            const double om = __longlong_as_double(x + k);
            if (om <= 1.0) check_chain(o, om, 1.5);
        }
    }
}
__global__ void k_roots(const double* x, int n, Out o) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    for (int e = -124; e <= 124; e++) check_root(o, x[t] * with_exponent(0, 2 * e), 1.0);
}
}  // namespace

extern "C" {
int divcheck_checks(void) { return C_N; }
int divcheck_random(int64_t n, uint64_t seed, unsigned long long* count, double* first) {
    k_random<<<148 * 16, 128>>>(n, seed, Out{count, first});
    return (int)cudaDeviceSynchronize();
}
// arguments in [1, 4) whose roots lie next to a midpoint of two doubles
int divcheck_roots(const double* x, int n, uint64_t, unsigned long long* count, double* first) {
    if (n > 0) k_roots<<<(n + 127) / 128, 128>>>(x, n, Out{count, first});
    return (int)cudaDeviceSynchronize();
}
int divcheck_list(const double* b, int n, uint64_t seed, unsigned long long* count, double* first) {
    if (n > 0) k_list<<<(n + 127) / 128, 128>>>(b, n, seed, Out{count, first});
    return (int)cudaDeviceSynchronize();
}
}
