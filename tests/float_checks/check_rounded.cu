// csrc/rounded.cuh against the IEEE operators, on the device: the root, its
// reciprocal and the reciprocal for every float that Ranges admits, the
// quotient for random operands over its ranges, half of them with a quotient
// next to a rounding boundary. Prints the disagreements of each and how much
// of the trials the ranges admit.
#include <cstdio>

#include "../../visionary-sim_gb300/csrc/rounded.cuh"

using namespace vsim::rounded;

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

__global__ void everyFloat(unsigned long long* bad) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= 0xffffffffull; i += stride) {
        const float v = __uint_as_float(uint32_t(i));
        float c, inv;
        rootAndReciprocal(v, c, inv);
        Ranges root;
        root.arguments(v, 1.0f);
        root.reciprocalOfRoot(inv);
        if (v > 0 && root.hold()) {
            const float want = __fsqrt_rn(v);
            if (!same(c, want)) atomicAdd(bad, 1ull);
            if (!same(inv, __fdiv_rn(1.0f, want))) atomicAdd(bad + 1, 1ull);
            atomicAdd(bad + 5, 1ull);
        }
        Ranges divisor;
        divisor.arguments(v, 1.0f);
        if (divisor.hold() && !same(reciprocal(v, approxReciprocal(v)), __fdiv_rn(1.0f, v))) atomicAdd(bad + 2, 1ull);
        if (divisor.hold() != (fabsf(v) >= 0x1p-20f && fabsf(v) <= 0x1p100f)) atomicAdd(bad + 2, 1ull);  // NaN: not held
    }
}

__device__ uint32_t mix(uint64_t& s) {
    s += 0x9e3779b97f4a7c15ull;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return uint32_t((z ^ (z >> 31)) >> 16);
}

__global__ void randomPairs(unsigned long long* bad, int each) {
    uint64_t s = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) * 7919 + 1;
    for (int k = 0; k < each; k++) {
        const float b = __uint_as_float((105 + mix(s) % 126) << 23 | (mix(s) & 0x7fffff));
        float a = __uint_as_float((1 + mix(s) % 253) << 23 | (mix(s) & 0x7fffff));
        if (k & 1) {
            // b times a value half an ulp from a float, rounded: quotients at
            // the edges of rounding
            const float q = __uint_as_float(127u << 23 | (mix(s) & 0x7fffff));
            a = float(double(b) * (double(q) + double(__uint_as_float(__float_as_uint(q) + 1))) * 0.5);
        }
        if (mix(s) & 1) a = -a;
        const float q = quotient(a, b, reciprocal(b, approxReciprocal(b)));
        Ranges r;
        r.arguments(1.0f, b);
        r.quotients(q, 1.0f);
        if (!r.hold()) continue;
        if (!same(q, __fdiv_rn(a, b))) atomicAdd(bad + 3, 1ull);
        atomicAdd(bad + 4, 1ull);
    }
}

int main() {
    unsigned long long* bad;
    if (cudaMallocManaged(&bad, 6 * sizeof *bad) != cudaSuccess) return 2;
    for (int i = 0; i < 6; i++) bad[i] = 0;
    everyFloat<<<2432, 256>>>(bad);
    randomPairs<<<2432, 256>>>(bad, 200);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    printf("root %llu reciprocal_root %llu reciprocal %llu quotient %llu of %llu; roots %llu\n", bad[0], bad[1], bad[2],
           bad[3], bad[4], bad[5]);
    return bad[0] || bad[1] || bad[2] || bad[3] || bad[4] < 10000000 || bad[5] < 1000000000 ? 1 : 0;
}
