// Checks of csrc/exact_pair.cuh on the device (test_gpu_exact_pair.py builds it
// with the flags of the exact build).  Prints "<name> <checked> <wrong>" lines.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "exact_pair.cuh"

using namespace pbf;

__device__ __forceinline__ unsigned hash(unsigned x) {  // an integer mix, for operands
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    return x ^ (x >> 16);
}

__device__ __forceinline__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// Roots of the floats with bits [lo, hi), in pairs; those whose inverse is not
// the correctly rounded one are collected.
__global__ void roots(unsigned lo, unsigned hi, unsigned long long* wrong, unsigned* odd, unsigned* nodd, unsigned cap) {
    for (unsigned b = lo + 2u * (blockIdx.x * blockDim.x + threadIdx.x); b < hi; b += 2u * gridDim.x * blockDim.x) {
        const float2 x = make_float2(__uint_as_float(b), __uint_as_float(min(b + 1u, hi - 1u)));
        float2 root, inv;
        root_and_inverse(x, root, inv);
        const float want[2] = {sqrtf(x.x), sqrtf(x.y)}, got[2] = {root.x, root.y}, iv[2] = {inv.x, inv.y};
        for (int k = 0; k < 2; ++k) {
            if (!same(want[k], got[k])) atomicAdd(wrong, 1ull);
            if (!same(iv[k], __fdiv_rn(1.0f, want[k]))) {
                const unsigned at = atomicAdd(nodd, 1u);
                if (at < cap) odd[at] = __float_as_uint(k ? x.y : x.x);
            }
        }
    }
}

// a / root for every significand of a and the root of each square in x[0, nx).
__global__ void quotients(const unsigned* x, unsigned nx, float scale, unsigned long long* wrong) {
    for (unsigned j = blockIdx.y; j < nx; j += gridDim.y) {
        float2 root, inv;
        root_and_inverse(make_float2(__uint_as_float(x[j]), __uint_as_float(x[j])), root, inv);
        for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < (1u << 22); m += gridDim.x * blockDim.x) {
            const float2 a = make_float2(scale * __uint_as_float(0x3f800000u | m),
                                         -scale * __uint_as_float(0x3f800000u | m | (1u << 22)));
            const float2 q = quotient(a, root, inv);
            if (!same(q.x, __fdiv_rn(a.x, root.x))) atomicAdd(wrong, 1ull);
            if (!same(q.y, __fdiv_rn(a.y, root.y))) atomicAdd(wrong, 1ull);
        }
    }
}

// Products, sums and sums of products, each lane like the scalar operation.
__global__ void sums(unsigned n, float one, unsigned long long* wrong) {
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float v[6];
        for (unsigned k = 0; k < 6; ++k) {  // exponents -20 to 11, both signs
            const unsigned h = hash(6u * i + k), g = hash(h + 0x9e3779b9u);
            v[k] = __uint_as_float((h & 0x807fffffu) | ((107u + (g & 31u)) << 23));
        }
        const float2 a = make_float2(v[0], v[1]), b = make_float2(v[2], v[3]), c = make_float2(v[4], v[5]);
        const float2 m = mul2(a, b), s = add2(mul2(a, b), c, one), d = sub2(a, c);
        const float2 t = add2(mul2(a, a), add2(mul2(b, b), mul2(c, c), one), one);
        bool ok = same(m.x, __fmul_rn(v[0], v[2])) && same(m.y, __fmul_rn(v[1], v[3]));
        ok = ok && same(s.x, __fadd_rn(__fmul_rn(v[0], v[2]), v[4])) && same(s.y, __fadd_rn(__fmul_rn(v[1], v[3]), v[5]));
        ok = ok && same(d.x, __fadd_rn(v[0], -v[4])) && same(d.y, __fadd_rn(v[1], -v[5]));
        ok = ok && same(t.x, __fadd_rn(__fmul_rn(v[0], v[0]),
                                       __fadd_rn(__fmul_rn(v[2], v[2]), __fmul_rn(v[4], v[4]))));
        ok = ok && same(t.y, __fadd_rn(__fmul_rn(v[1], v[1]),
                                       __fadd_rn(__fmul_rn(v[3], v[3]), __fmul_rn(v[5], v[5]))));
        if (!ok) atomicAdd(wrong, 1ull);
    }
}

#define CHECK(call)                                                             \
    do {                                                                        \
        const cudaError_t e_ = (call);                                          \
        if (e_ != cudaSuccess) {                                                \
            std::printf("error %s\n", cudaGetErrorString(e_));                  \
            return 1;                                                           \
        }                                                                       \
    } while (0)

static unsigned bits(float f) {
    unsigned u;
    static_assert(sizeof u == sizeof f, "");
    __builtin_memcpy(&u, &f, 4);
    return u;
}

int main() {
    constexpr unsigned kOdd = 1u << 20, kRandom = 4096;
    unsigned long long* wrong = nullptr;
    unsigned *odd = nullptr, *nodd = nullptr, *some = nullptr;
    CHECK(cudaMallocManaged(&wrong, 8 * 4));
    CHECK(cudaMallocManaged(&odd, 4 * kOdd));
    CHECK(cudaMallocManaged(&nodd, 4));
    CHECK(cudaMallocManaged(&some, 4 * kRandom));
    for (int k = 0; k < 4; ++k) wrong[k] = 0;
    *nodd = 0;
    const unsigned lo = bits(1e-14f), hi = bits(1.1e4f) + 1u;
    std::srand(1);
    for (unsigned k = 0; k < kRandom; ++k)
        some[k] = lo + (unsigned)(((unsigned long long)std::rand() * 2147483647ull + std::rand()) % (hi - lo));
    roots<<<4096, 256>>>(lo, hi, wrong, odd, nodd, kOdd);
    CHECK(cudaDeviceSynchronize());
    std::printf("roots %u %llu\n", hi - lo, wrong[0]);
    std::printf("inverses %u %u\n", hi - lo, *nodd);
    const unsigned n = *nodd < kOdd ? *nodd : kOdd;
    // Dividends from 1 to 2 and at the ends of the spiky kernel's range.
    const float scales[3] = {1.0f, 1e9f, 1e-21f};
    if (n)
        for (float s : scales) quotients<<<dim3(64, 64), 256>>>(odd, n, s, wrong + 1);
    for (float s : scales) quotients<<<dim3(64, 64), 256>>>(some, kRandom, s, wrong + 2);
    sums<<<4096, 256>>>(1u << 26, 1.0f, wrong + 3);
    CHECK(cudaDeviceSynchronize());
    std::printf("quotients_of_inexact_inverses %llu %llu\n", 3ull * n << 23, wrong[1]);
    std::printf("quotients %llu %llu\n", 3ull * kRandom << 23, wrong[2]);
    std::printf("sums %u %llu\n", 1u << 26, wrong[3]);
    return 0;
}
