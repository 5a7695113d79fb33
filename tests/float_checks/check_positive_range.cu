// csrc/rounded.cuh against the IEEE operators, on the device, over the range of
// the arguments that have to be positive: every float as a root's argument and as
// a divisor, held in [2^-58, 2^125] only; and quotients of random operands over
// more than the ranges, a third of them around the least dividends that are held
// and a third next to a rounding boundary.
#include <cstdio>

#include "../../visionary-sim_gb300/csrc/rounded.cuh"

using namespace vsim::rounded;

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

__global__ void everyFloat(unsigned long long* bad) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= 0xffffffffull; i += stride) {
        const float v = __uint_as_float(uint32_t(i));
        const bool in = v >= 0x1p-58f && v <= 0x1p125f;
        Ranges divisor, root;
        divisor.argumentAndPositive(1.0f, v);
        root.argumentAndPositive(v, 1.0f);
        if (divisor.hold() != in || root.hold() != in) atomicAdd(bad, 1ull);
        if (!in) continue;
        atomicAdd(bad + 4, 1ull);
        if (!same(reciprocal(v, approxReciprocal(v)), __fdiv_rn(1.0f, v))) atomicAdd(bad + 1, 1ull);
        float c, inv;
        rootAndReciprocal(v, c, inv);
        root.reciprocalOfRoot(inv);
        if (!root.hold()) continue;
        const float want = __fsqrt_rn(v);
        if (!same(c, want) || !same(inv, __fdiv_rn(1.0f, want))) atomicAdd(bad + 2, 1ull);
    }
}

__device__ uint32_t mix(uint64_t& s) {
    s += 0x9e3779b97f4a7c15ull;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return uint32_t((z ^ (z >> 31)) >> 16);
}

__global__ void quotients(unsigned long long* bad, int each) {
    uint64_t s = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) * 7919 + 5;
    auto of = [&](int exponent) { return __uint_as_float(uint32_t(127 + exponent) << 23 | (mix(s) & 0x7fffffu)); };
    for (int k = 0; k < each; k++) {
        float b = of(int(mix(s) % 190) - 63);
        float a = of(int(mix(s) % 237) - 110);
        if (k % 3 == 1) {  // about the least dividend
            b = of(int(mix(s) % 66) - 62);
            a = of(int(mix(s) % 6) - 103);
        }
        if (k % 3 == 2) {
            const float q = of(int(mix(s) % 100) - 50);  // half an ulp from a float, rounded
            a = float(double(b) * (double(q) + double(__uint_as_float(__float_as_uint(q) + 1))) * 0.5);
        }
        if (mix(s) & 1) a = -a;
        const float q = quotient(a, b, reciprocal(b, approxReciprocal(b)));
        Ranges r;
        r.argumentAndPositive(3.0f, b);
        r.quotients(q, 1.0f);
        if (!r.hold()) continue;
        if (!same(q, __fdiv_rn(a, b))) atomicAdd(bad + 3, 1ull);
        atomicAdd(bad + 5, 1ull);
    }
}

int main() {
    unsigned long long* bad;
    if (cudaMallocManaged(&bad, 6 * sizeof *bad) != cudaSuccess) return 2;
    for (int i = 0; i < 6; i++) bad[i] = 0;
    everyFloat<<<2432, 256>>>(bad);
    quotients<<<2432, 256>>>(bad, 200);
    if (cudaDeviceSynchronize() != cudaSuccess) return 2;
    printf("held %llu reciprocal %llu root %llu quotient %llu; floats %llu quotients %llu\n", bad[0], bad[1], bad[2],
           bad[3], bad[4], bad[5]);
    return bad[0] || bad[1] || bad[2] || bad[3] || bad[4] < 1000000000 || bad[5] < 10000000 ? 1 : 0;
}
