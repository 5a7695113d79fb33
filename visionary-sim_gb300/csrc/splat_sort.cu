// Gaussian-splat deformation (sample.wgsl:40-80 with covariance.wgsl:18-42)
// and the stable LSD radix sort behind the depth order.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>

#include "kernels.cuh"

namespace vsim {

// ------------------------------------------------------------- splats --

// Back-to-front draw key: ascending key order is descending depth.
__device__ __forceinline__ uint32_t depthKey(float depth) {
    const uint32_t bits = __float_as_uint(depth);
    const uint32_t ordered = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
    return ~ordered;
}

// One thread per splat: trilinear position and gradient F from the cell's
// eight live nodes, then Sigma' = (F R S)(F R S)^T, then the depth key. The
// embedding (cell corner node, local coordinates) was computed at bind time
// with sample.wgsl:45-51's arithmetic.
// ellipsoid.wgsl:20-91: a covariance (xx, xy, xz, yy, yz, zz) as a unit
// quaternion xyzw and three axis lengths, by four sweeps of cyclic Jacobi.
// inverseSqrt is 1 / sqrt and normalize is q / sqrt(|q|^2) with |q|^2 fused
// as dot is; every other operation rounds once -- the CPU restatement's
// evaluation, so the two agree bit for bit.
__device__ __forceinline__ void ellipsoidAxes(const float cov[6], float4& rotation, V& scale) {
    float a[9] = {cov[0], cov[1], cov[2], cov[1], cov[3], cov[4], cov[2], cov[4], cov[5]};
    float q[4] = {0.0f, 0.0f, 0.0f, 1.0f};
#pragma unroll
    for (int sweep = 0; sweep < 4; sweep++) {
#pragma unroll
        for (int p = 0; p < 3; p++) {
            const int r = (p + 1) % 3, other = (p + 2) % 3;
            const float apr = a[r * 3 + p];
            if (apr == 0.0f) continue;
            const float app = a[p * 3 + p];
            const float arr = a[r * 3 + r];
            const float theta = (arr - app) / (2.0f * apr);
            const float sign = theta >= 0.0f ? 1.0f : -1.0f;
            const float tangent = sign / (fabsf(theta) + sqrtf(theta * theta + 1.0f));
            const float cosine = 1.0f / sqrtf(tangent * tangent + 1.0f);
            const float sine = tangent * cosine;
            const float apo = a[other * 3 + p];
            const float aro = a[other * 3 + r];
            const float turnedP = cosine * apo - sine * aro;
            const float turnedR = sine * apo + cosine * aro;
            a[p * 3 + p] = app - tangent * apr;
            a[r * 3 + r] = arr + tangent * apr;
            a[r * 3 + p] = 0.0f;
            a[p * 3 + r] = 0.0f;
            a[other * 3 + p] = turnedP;
            a[p * 3 + other] = turnedP;
            a[other * 3 + r] = turnedR;
            a[r * 3 + other] = turnedR;
            const float half = -(sine / (1.0f + cosine));
            float b[4] = {0.0f, 0.0f, 0.0f, 1.0f};
            b[other] = half;
            const float prod[4] = {q[3] * b[0] + q[0] * b[3] + q[1] * b[2] - q[2] * b[1],
                                   q[3] * b[1] - q[0] * b[2] + q[1] * b[3] + q[2] * b[0],
                                   q[3] * b[2] + q[0] * b[1] - q[1] * b[0] + q[2] * b[3],
                                   q[3] * b[3] - q[0] * b[0] - q[1] * b[1] - q[2] * b[2]};
            const float length =
                sqrtf(fmaf(prod[3], prod[3], fmaf(prod[2], prod[2], fmaf(prod[1], prod[1], prod[0] * prod[0]))));
#pragma unroll
            for (int c = 0; c < 4; c++) q[c] = prod[c] / length;
        }
    }
    rotation = make_float4(q[0], q[1], q[2], q[3]);
    scale = mk(sqrtf(fmaxf(a[0], 0.0f)), sqrtf(fmaxf(a[4], 0.0f)), sqrtf(fmaxf(a[8], 0.0f)));
}

constexpr uint32_t kDeformBlock = 256;

// Stores the warp's 32 vectors, lane l's at out[3 (first + l)], as whole
// 16-byte words through 96 words of shared memory. `first` is a multiple of
// 32; vectors from `n` on are left out. The caller's next use of `words` must
// wait for the warp.
__device__ __forceinline__ void storeXyz(float* out, uint32_t first, uint32_t n, V v, float* words) {
    const uint32_t lane = threadIdx.x & 31;
    words[3 * lane] = v.x;
    words[3 * lane + 1] = v.y;
    words[3 * lane + 2] = v.z;
    __syncwarp();
    if (first + 32 <= n) {
        if (lane < 24)
            __stcs(reinterpret_cast<float4*>(out + 3 * size_t(first)) + lane, reinterpret_cast<const float4*>(words)[lane]);
    } else {
        for (uint32_t q = lane; q < 3 * (n - first); q += 32) out[3 * size_t(first) + q] = words[q];
    }
    __syncwarp();
}

template <bool AXES>
__global__ void __launch_bounds__(kDeformBlock) splatDeformKernel(const float4* __restrict__ embed,
                                                         const float4* __restrict__ quat,
                                                         const float4* __restrict__ scaleBody,
                                                         const SplatBody* __restrict__ bodies,
                                                         const float4* __restrict__ pos, uint32_t n, float vx,
                                                         float vy, float vz, float* __restrict__ means,
                                                         float2* __restrict__ cov, uint32_t* __restrict__ keys,
                                                         uint32_t* __restrict__ order,
                                                         float4* __restrict__ axesRotation,
                                                         float* __restrict__ axesScale) {
    __shared__ __align__(16) float words[kDeformBlock / 32][96];
    const uint32_t at = blockIdx.x * blockDim.x + threadIdx.x, first = at & ~31u;
    if (first >= n) return;
    // The last warp's lanes past the end go through the last splat again and
    // store nothing.
    const uint32_t i = min(at, n - 1);
    const bool mine = at < n;
    // The splat's embedding, scale and rotation do not change between
    // frames: loaded before waiting for the frame that moves the nodes.
    // The splat streams are read and written once, marked evict-first
    // (.cs), so that the node positions the corner gathers hit stay in L2.
    const float4 e = __ldcs(embed + i);
    const float4 sb = __ldcs(scaleBody + i);
    const float4 q4 = __ldcs(quat + i);
    const SplatBody B = bodies[__float_as_uint(sb.w)];
    pdlWait();
    pdlLaunchNext();
    const uint32_t node0 = __float_as_uint(e.w);
    const float local[3] = {e.x, e.y, e.z};
    const float inv = B.inv;
    V position = mk(0.0f, 0.0f, 0.0f);
    V col0 = mk(0.0f, 0.0f, 0.0f), col1 = col0, col2 = col0;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const int cx = c & 1, cy = (c >> 1) & 1, cz = (c >> 2) & 1;
        const float fx = cx ? local[0] : 1.0f - local[0];
        const float fy = cy ? local[1] : 1.0f - local[1];
        const float fz = cz ? local[2] : 1.0f - local[2];
        const float dx = cx ? 1.0f : -1.0f, dy = cy ? 1.0f : -1.0f, dz = cz ? 1.0f : -1.0f;
        const V p = xyz(pos[node0 + cx + B.nx * cy + B.nxy * cz]);
        position = position + p * (fx * fy * fz);
        const V g = mk(dx * fy * fz, dy * fx * fz, dz * fx * fy) * inv;
        col0 = col0 + p * g.x;
        col1 = col1 + p * g.y;
        col2 = col2 + p * g.z;
    }
    const M F{{col0, col1, col2}};
    const float x = q4.x, y = q4.y, z = q4.z, w = q4.w;
    const V r0 = mk(1.0f - 2.0f * (y * y + z * z), 2.0f * (x * y + z * w), 2.0f * (x * z - y * w));
    const V r1 = mk(2.0f * (x * y - z * w), 1.0f - 2.0f * (x * x + z * z), 2.0f * (y * z + x * w));
    const V r2 = mk(2.0f * (x * z + y * w), 2.0f * (y * z - x * w), 1.0f - 2.0f * (x * x + y * y));
    const V a0 = mul(F, r0) * sb.x;
    const V a1 = mul(F, r1) * sb.y;
    const V a2 = mul(F, r2) * sb.z;
    // (A A^T)(row, col) = a0[row] a0[col] + a1[row] a1[col] + a2[row] a2[col],
    // column col of A times row col of A^T, fused as M * v is.
    const float xx = fmaf(a2.x, a2.x, fmaf(a1.x, a1.x, a0.x * a0.x));
    const float xy = fmaf(a2.y, a2.x, fmaf(a1.y, a1.x, a0.y * a0.x));
    const float xz = fmaf(a2.z, a2.x, fmaf(a1.z, a1.x, a0.z * a0.x));
    const float yy = fmaf(a2.y, a2.y, fmaf(a1.y, a1.y, a0.y * a0.y));
    const float yz = fmaf(a2.z, a2.y, fmaf(a1.z, a1.y, a0.z * a0.y));
    const float zz = fmaf(a2.z, a2.z, fmaf(a1.z, a1.z, a0.z * a0.z));
    const float depth = position.x * vx + position.y * vy + position.z * vz;
    storeXyz(means, first, n, position, words[threadIdx.x >> 5]);
    if (mine) {
        __stcs(cov + 3 * size_t(i), make_float2(xx, xy));
        __stcs(cov + 3 * size_t(i) + 1, make_float2(xz, yy));
        __stcs(cov + 3 * size_t(i) + 2, make_float2(yz, zz));
        keys[i] = depthKey(depth);
    }
    (void)order;
    if (AXES) {
        const float c6[6] = {xx, xy, xz, yy, yz, zz};
        float4 rotation;
        V scale;
        ellipsoidAxes(c6, rotation, scale);
        if (mine) axesRotation[i] = rotation;
        storeXyz(axesScale, first, n, scale, words[threadIdx.x >> 5]);
    }
}

cudaError_t launchSplatDeform(cudaStream_t st, const SplatState& s, const float4* pos, uint32_t n, float vx, float vy,
                              float vz, bool axes) {
    if (n == 0) return cudaSuccess;
    // Programmatic dependent launch: the constant loads above overlap the
    // tail of the frame's last kernel.
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((n + kDeformBlock - 1) / kDeformBlock);
    cfg.blockDim = dim3(kDeformBlock);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (axes)
        return cudaLaunchKernelEx(&cfg, splatDeformKernel<true>, (const float4*)s.embed, (const float4*)s.quat,
                                  (const float4*)s.scaleBody, (const SplatBody*)s.bodies, pos, n, vx, vy, vz,
                                  s.means, s.cov, s.keys, s.order, s.axesRotation, s.axesScale);
    return cudaLaunchKernelEx(&cfg, splatDeformKernel<false>, (const float4*)s.embed, (const float4*)s.quat,
                              (const float4*)s.scaleBody, (const SplatBody*)s.bodies, pos, n, vx, vy, vz, s.means,
                              s.cov, s.keys, s.order, (float4*)nullptr, (float*)nullptr);
}

// --------------------------------------------------------- radix sort --
//
// Least-significant-digit radix sort, 8-bit digits, one sweep of the keys
// per pass -- the single-pass scan with decoupled look-back (Merrill and
// Garland, 2016) applied to radix sorting as Adinets and Merrill's
// "Onesweep" (2022) does:
//
// - one launch counts every pass's digits over all the keys at once (a
//   pass's digit totals do not depend on the order earlier passes leave);
// - then one launch per pass. Each block takes the next tile from a ticket,
//   so tiles start in order; it ranks its keys per digit (a warp its own,
//   rankKeys) and publishes the tile's count of each digit in a status word
//   (count and a flag packed in 32 bits, so one store carries both). While
//   the words of the tiles before it arrive, it sorts the tile in shared
//   memory; then each digit's thread walks back over those tiles, adding
//   their counts until it meets a word that already holds an inclusive
//   prefix, and publishes the tile's own. A tile waits only on tiles that
//   started before it, which publish their counts without waiting on
//   anything, so every walk ends. The block writes the tile out in runs that
//   are contiguous per digit.
//
// What bounds a pass is instructions, most of them the ranking's ballots (20M
// keys: 124 warp instructions per 32 keys, the ALU pipe 60 % and the
// shared-memory pipe 45 % active, 2 TB/s of DRAM). Against ranking with
// __match_any_sync, key by key with its load and its counter's round trip,
// looking back one word a trip before the tile is sorted, and two look-ups a
// key: 20M keys in 492 us where they took 746, 1M in 52 where 83.
//
// The tile: past two tiles of 4096 keys an SM the passes take several waves,
// and fewer, larger tiles are worth the longer first one (20M keys: 582 us
// with tiles of 4096 keys, 500 with 6144 and 8192, whose keys spill; 4M: 141,
// 130 and 139). Within one wave a tile's latency is the pass (1M keys: 52, 61
// and 70 us).
//
// Tiles and ranks follow input order, so each pass -- and the sort -- is
// stable. The status words, digit totals and tickets are cleared by one
// memset at the start of a sort; every other scratch word is written before
// it is read.

constexpr uint32_t kCountThreads = 256;
constexpr uint32_t kSortThreads = 512;
constexpr uint32_t kSortItems = 8;        // keys a thread while the tiles are one wave
constexpr uint32_t kSortLargeItems = 12;  // and past that
constexpr uint32_t kSortTile = kSortThreads * kSortItems;            // 4096 keys
constexpr uint32_t kSortLargeTile = kSortThreads * kSortLargeItems;  // 6144
constexpr uint32_t kSortMaxPasses = 4;
constexpr uint32_t kStatusCount = 1u << 30;     // the word holds the tile's own count
constexpr uint32_t kStatusPrefix = 2u << 30;    // the word holds the inclusive prefix
constexpr uint32_t kStatusValue = (1u << 30) - 1u;
constexpr uint32_t kLookbackSpinLimit = 1u << 22;

namespace {
constexpr size_t align256(size_t b) { return (b + 255) & ~size_t(255); }
constexpr uint32_t tilesOf(uint32_t n) { return (n + kSortTile - 1) / kSortTile; }
// Cleared at the start of a sort: the digit totals of every pass, a ticket
// per pass and the failure word; then, per pass, a status word per (tile,
// digit).
constexpr size_t kSortHeadBytes = align256(kSortMaxPasses * 256 * 4) + 256;
constexpr size_t sortClearedBytes(uint32_t n) {
    return kSortHeadBytes + align256(size_t(kSortMaxPasses) * tilesOf(n) * 256 * 4);
}
constexpr size_t sortTempBytes(uint32_t n) { return 4 * align256(size_t(n) * 4) + sortClearedBytes(n); }
}  // namespace

size_t radixSortTempBytes(uint32_t n) { return sortTempBytes(n); }

__device__ __forceinline__ uint32_t loadRelaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void storeRelaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Every pass's digit counts over all keys: per block in shared memory, then
// added into totals[pass * 256 + digit].
__global__ void __launch_bounds__(kCountThreads) sortDigitCountKernel(const uint32_t* __restrict__ keys, uint32_t n,
                                                                     uint32_t keyBits,
                                                                     uint32_t* __restrict__ totals) {
    __shared__ uint32_t bins[kSortMaxPasses * 256];
    for (uint32_t i = threadIdx.x; i < kSortMaxPasses * 256; i += kCountThreads) bins[i] = 0;
    pdlWait();  // the keys come from the kernel before
    pdlLaunchNext();
    __syncthreads();
    const uint32_t passes = (keyBits + 7) / 8;
    auto count = [&](uint32_t k) {
#pragma unroll
        for (uint32_t p = 0; p < kSortMaxPasses; p++) {
            if (p >= passes) break;
            const uint32_t bits = keyBits - 8 * p < 8 ? keyBits - 8 * p : 8;
            atomicAdd(&bins[p * 256 + ((k >> (8 * p)) & ((1u << bits) - 1u))], 1u);
        }
    };
    const uint32_t stride = gridDim.x * kCountThreads;
    // four keys per load where the keys start on a 16-byte boundary
    const uint32_t quads = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0 ? n / 4 : 0;
    const uint4* k4 = reinterpret_cast<const uint4*>(keys);
    for (uint32_t i = blockIdx.x * kCountThreads + threadIdx.x; i < quads; i += stride) {
        const uint4 q = k4[i];
        count(q.x);
        count(q.y);
        count(q.z);
        count(q.w);
    }
    for (uint32_t i = 4 * quads + blockIdx.x * kCountThreads + threadIdx.x; i < n; i += stride) count(keys[i]);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < passes * 256; i += kCountThreads)
        if (bins[i]) atomicAdd(&totals[i], bins[i]);
}

// The lanes of `active` whose 8-bit digit equals this lane's: one ballot a bit.
__device__ __forceinline__ uint32_t peersOf(uint32_t digit, uint32_t active) {
    uint32_t peers = active;
#pragma unroll
    for (uint32_t b = 0; b < 8; b++) {
        const bool bit = digit >> b & 1u;
        const uint32_t set = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? set : ~set;
    }
    return peers;
}

// Ranks a warp's keys of each digit: key r of a lane comes after the keys
// before it in (r, lane) order, and rank(r) counts those of its digit. `hist`,
// the warp's 256 counters, zero before, holds its digit counts after. The
// lowest lane of each digit adds for all of its peers, in order of r, and
// hands them the count before; in two loops, so that no key's ballots wait on
// the counters' round trip for the one before. A rank fits 16 bits, and so
// does what the second loop needs of the first: two keys share a register.
template <uint32_t ITEMS>
struct Ranks {
    uint32_t packed[(ITEMS + 1) / 2];
    __device__ __forceinline__ uint32_t operator()(uint32_t r) const { return packed[r / 2] >> 16 * (r % 2) & 0xffffu; }
    __device__ __forceinline__ void set(uint32_t r, uint32_t v) {
        packed[r / 2] = r % 2 ? (packed[r / 2] & 0xffffu) | v << 16 : (packed[r / 2] & 0xffff0000u) | v;
    }
};

template <bool FULL, uint32_t ITEMS>
__device__ __forceinline__ void rankKeys(const uint32_t (&key)[ITEMS], uint32_t first, uint32_t n, uint32_t shift,
                                         uint32_t mask, uint32_t* hist, Ranks<ITEMS>& rank) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t before[ITEMS];
#pragma unroll
    for (uint32_t r = 0; r < (ITEMS + 1) / 2; r++) rank.packed[r] = 0;
#pragma unroll
    for (uint32_t r = 0; r < ITEMS; r++) {
        const bool valid = FULL || first + r * 32 + lane < n;
        const uint32_t digit = key[r] >> shift & mask;
        const uint32_t peers = peersOf(digit, FULL ? 0xffffffffu : __ballot_sync(0xffffffffu, valid));
        before[r] = 0;
        if (valid && (peers & lt) == 0) before[r] = atomicAdd(hist + digit, uint32_t(__popc(peers)));
        // A lane past the end hands itself its zero.
        const uint32_t leader = valid ? __ffs(int(peers)) - 1 : lane;
        rank.set(r, leader | __popc(peers & lt) << 8);
        asm volatile("" : "+r"(rank.packed[r / 2]));  // packed now, not where it is read
        __syncwarp();
    }
#pragma unroll
    for (uint32_t r = 0; r < ITEMS; r++) {
        const uint32_t info = rank(r);
        rank.set(r, __shfl_sync(0xffffffffu, before[r], int(info & 31u)) + (info >> 8));
    }
}

// The exclusive scan of one value a thread over the first 256 threads of a
// block; all of its threads call it.
__device__ __forceinline__ uint32_t scanDigits(uint32_t v, uint32_t* warpSums) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= uint32_t(d)) incl += u;
    }
    if (lane == 31 && warp < 8) warpSums[warp] = incl;
    __syncthreads();
    uint32_t base = 0;
#pragma unroll
    for (uint32_t w = 0; w < 7; w++)
        if (w < warp) base += warpSums[w];
    return base + incl - v;
}

template <uint32_t ITEMS>
struct PassShared {
    uint2 pairs[kSortThreads * ITEMS];  // key, value
    uint32_t warpHist[kSortThreads / 32][256];
    uint32_t part[kSortThreads / 256][256];  // digit counts over eight warps each
    uint32_t place[256];                // what takes a key's place in the tile to its place in the output
    uint32_t warpSums[2][8];
    uint32_t tile;
};

// One pass over one tile: rank it, find its digits' global offsets by
// decoupled look-back, scatter. `status` is the pass's (tile, digit) words,
// `totals` its 256 digit counts over all keys.
template <bool FULL, uint32_t ITEMS>
__device__ __forceinline__ void sortTile(PassShared<ITEMS>& sh, uint32_t tile,
                                         const uint32_t* __restrict__ keysIn, const uint32_t* __restrict__ valsIn,
                                         uint32_t n, uint32_t shift, uint32_t mask,
                                         const uint32_t* __restrict__ totals, uint32_t* __restrict__ status,
                                         uint32_t* __restrict__ error, uint32_t* __restrict__ keysOut,
                                         uint32_t* __restrict__ valsOut) {
    constexpr uint32_t kTile = kSortThreads * ITEMS;
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t tileBase = tile * kTile;
    const uint32_t first = tileBase + warp * 32 * ITEMS;
    uint32_t key[ITEMS], val[ITEMS];
    Ranks<ITEMS> rank;
    const uint32_t* keyAt = keysIn + first + lane;
#pragma unroll
    for (uint32_t r = 0; r < ITEMS; r++) key[r] = FULL || first + r * 32 + lane < n ? keyAt[r * 32] : 0u;
    rankKeys<FULL, ITEMS>(key, first, n, shift, mask, sh.warpHist[warp], rank);
    __syncthreads();
    if (valsIn) {
        const uint32_t* valAt = valsIn + first + lane;
#pragma unroll
        for (uint32_t r = 0; r < ITEMS; r++) val[r] = FULL || first + r * 32 + lane < n ? valAt[r * 32] : 0u;
    } else {
#pragma unroll
        for (uint32_t r = 0; r < ITEMS; r++) val[r] = first + r * 32 + lane;
    }
    // Per digit, eight warps' counts a thread: the tile's count of the digit,
    // and where each warp's keys of it start in the tile.
    const uint32_t digit = t & 255, part = t >> 8;
    constexpr uint32_t kParts = kSortThreads / 256, kEach = 8;
    uint32_t of[kEach], count = 0, run = 0;
#pragma unroll
    for (uint32_t w = 0; w < kEach; w++) count += of[w] = sh.warpHist[part * kEach + w][digit];
    if (kParts > 1) {
        sh.part[part][digit] = count;
        __syncthreads();
        count = 0;
#pragma unroll
        for (uint32_t q = 0; q < kParts; q++) {
            const uint32_t c = sh.part[q][digit];
            if (q < part) run += c;
            count += c;
        }
    }
    // The first tile starts from the digit's place in the whole output, so
    // that every prefix that follows holds it.
    uint32_t before = 0;
    if (tile == 0) {
        before = scanDigits(t < 256 ? totals[t] : 0u, sh.warpSums[1]);
        if (t < 256) storeRelaxed(status + t, kStatusPrefix | (before + count));
    } else if (t < 256) {
        storeRelaxed(status + size_t(tile) * 256 + t, kStatusCount | count);
    }
    uint32_t start = scanDigits(t < 256 ? count : 0u, sh.warpSums[0]);
    if (kParts > 1) {
        if (t < 256) sh.place[t] = start;
        __syncthreads();
        start = sh.place[digit];
    }
    run += start;
#pragma unroll
    for (uint32_t w = 0; w < kEach; w++) {
        sh.warpHist[part * kEach + w][digit] = run;
        run += of[w];
    }
    __syncthreads();
    // The digits again, from a shift that the compiler takes for another:
    // kept from the ranking they would cost a register a key.
    uint32_t shiftAgain = shift;
    asm volatile("" : "+r"(shiftAgain));
#pragma unroll
    for (uint32_t r = 0; r < ITEMS; r++) {
        if (FULL || first + r * 32 + lane < n)
            sh.pairs[sh.warpHist[warp][key[r] >> shiftAgain & mask] + rank(r)] = make_uint2(key[r], val[r]);
    }
    if (t < 256) {
        // Decoupled look-back over the tiles before this one, whose words
        // have had the scatter's time to be published; several words a trip.
        constexpr uint32_t kTrip = 4;
        uint32_t polls = 0;
        bool found = tile == 0;
        for (uint32_t j = tile; !found && j > 0;) {
            uint32_t word[kTrip], taken = 0;
#pragma unroll
            for (uint32_t k = 0; k < kTrip; k++)
                word[k] = k < j ? loadRelaxed(status + size_t(j - 1 - k) * 256 + t) : 0u;
            bool more = true;
#pragma unroll
            for (uint32_t k = 0; k < kTrip; k++) {
                more = more && (word[k] & ~kStatusValue) != 0;  // else tile j - 1 - k has not published yet
                if (!more) continue;
                before += word[k] & kStatusValue;
                taken++;
                found = (word[k] & ~kStatusValue) == kStatusPrefix;
                more = !found;
            }
            j -= taken;
            if (taken == 0) {
                if (++polls > kLookbackSpinLimit) {
                    atomicOr(error, 1u);
                    break;
                }
                __nanosleep(32);
            }
        }
        if (tile > 0) storeRelaxed(status + size_t(tile) * 256 + t, kStatusPrefix | (before + count));
        sh.place[t] = before - start;
    }
    __syncthreads();
    const uint32_t held = FULL ? kTile : n - tileBase;
    uint32_t j = t;
#pragma unroll 4
    for (uint32_t r = 0; r < ITEMS; r++, j += kSortThreads) {
        if (FULL || j < held) {
            const uint2 pair = sh.pairs[j];
            const uint32_t out = sh.place[pair.x >> shiftAgain & mask] + j;
            if (keysOut) keysOut[out] = pair.x;
            valsOut[out] = pair.y;
        }
    }
}

template <uint32_t ITEMS>
__global__ void __launch_bounds__(kSortThreads, 2) sortPassKernel(const uint32_t* __restrict__ keysIn,
                                                                  const uint32_t* __restrict__ valsIn, uint32_t n,
                                                                  uint32_t shift, uint32_t mask,
                                                                  const uint32_t* __restrict__ totals,
                                                                  uint32_t* __restrict__ status,
                                                                  uint32_t* __restrict__ ticket,
                                                                  uint32_t* __restrict__ error,
                                                                  uint32_t* __restrict__ keysOut,
                                                                  uint32_t* __restrict__ valsOut) {
    extern __shared__ __align__(16) unsigned char raw[];
    auto& sh = *reinterpret_cast<PassShared<ITEMS>*>(raw);
    // The ticket counter was cleared before the sort's first launch, which
    // this one follows in stream order: safe to take before the wait.
    if (threadIdx.x == 0) sh.tile = atomicAdd(ticket, 1u);
    for (uint32_t i = threadIdx.x; i < kSortThreads / 32 * 256; i += kSortThreads) (&sh.warpHist[0][0])[i] = 0;
    pdlWait();  // the keys and totals come from the kernels before
    pdlLaunchNext();
    __syncthreads();
    const uint32_t tile = sh.tile;
    if (n - tile * (kSortThreads * ITEMS) >= kSortThreads * ITEMS)
        sortTile<true>(sh, tile, keysIn, valsIn, n, shift, mask, totals, status, error, keysOut, valsOut);
    else
        sortTile<false>(sh, tile, keysIn, valsIn, n, shift, mask, totals, status, error, keysOut, valsOut);
}

namespace {
// A sort kernel launched with programmatic dependent launch: its blocks may
// start while the kernel before finishes, and wait (pdlWait) before reading.
template <class... KArgs, class... Args>
cudaError_t pdl(void (*kernel)(KArgs...), uint32_t grid, uint32_t threads, size_t bytes, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
}  // namespace

// ------------------------------------------------ small sorts, one launch --
//
// Up to kClusterKeys keys one cluster of blocks sorts in one launch: the keys
// and their indices stay in the blocks' shared memory, and each 8-bit pass
// ranks them as sortTile does, gives every block the digit counts of every
// other over distributed shared memory and scatters straight into the block
// that holds the key's next place, key and index in one store. A block reads
// its keys into registers before the barrier that every block's scatter
// follows, so one buffer serves. Two cluster barriers a pass take the place
// of a launch and a look-back; what bounds it is the scattered stores between
// blocks, one key each. 30,011 keys in 18.8 us where the memset, count and
// four pass launches took 38.6 (100 keys: 7.1 and 20).
//
// The line: the tiles' six launches take 26 to 28.5 us at any size up to
// 50,000 keys; the cluster 17.3 at 16,384, 21.8 at 32,768 (four keys a thread)
// and 26.6 at 49,152 (six).

constexpr uint32_t kClusterThreads = 512;
constexpr uint32_t kClusterWarps = kClusterThreads / 32;
constexpr uint32_t kClusterBlocks = 16;
constexpr uint32_t kClusterItems = 6;  // keys a thread, at most
constexpr uint32_t kClusterKeys = kClusterBlocks * kClusterThreads * kClusterItems;

template <uint32_t ITEMS>
struct ClusterSortShared {
    uint2 pairs[kClusterThreads * ITEMS];  // key, index
    uint32_t warpHist[kClusterWarps][256];
    uint32_t half[kClusterThreads / 256][256];  // digit counts over eight warps each
    uint32_t counts[kClusterBlocks][256];       // every block's digit counts, written by that block
    uint32_t place[256];                        // where the block's keys of each digit start
    uint32_t warpSums[8];
};

__device__ __forceinline__ void clusterMeet() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// The address of this block's shared word `p` in block `rank` of the cluster.
__device__ __forceinline__ uint32_t inBlock(const void* p, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;"
        : "=r"(a)
        : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
    return a;
}
__device__ __forceinline__ void storeCluster(uint32_t a, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void storeCluster(uint32_t a, uint32_t x, uint32_t y) {
    asm volatile("st.shared::cluster.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}

template <uint32_t ITEMS>
__global__ void __launch_bounds__(kClusterThreads) clusterSortKernel(const uint32_t* __restrict__ keysIn, uint32_t n,
                                                                     uint32_t keyBits, uint32_t* __restrict__ order) {
    constexpr uint32_t kTile = kClusterThreads * ITEMS;
    extern __shared__ __align__(16) unsigned char raw[];
    auto& sh = *reinterpret_cast<ClusterSortShared<ITEMS>*>(raw);
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t rank = blockIdx.x, blocks = gridDim.x;  // one cluster is the whole grid
    const uint32_t first = rank * kTile + warp * 32 * ITEMS;
    uint32_t key[ITEMS], val[ITEMS];
    pdlWait();
    pdlLaunchNext();
#pragma unroll
    for (uint32_t r = 0; r < ITEMS; r++) {
        const uint32_t at = first + r * 32 + lane;
        key[r] = at < n ? keysIn[at] : 0u;
        val[r] = at;
    }
    clusterMeet();  // every block runs before another writes to it
    for (uint32_t shift = 0; shift < keyBits; shift += 8) {
        const uint32_t mask = keyBits - shift < 8 ? (1u << (keyBits - shift)) - 1u : 255u;
        // Each warp's digit counts, and every key's rank among its warp's
        // keys of the same digit.
        for (uint32_t d = lane; d < 256; d += 32) sh.warpHist[warp][d] = 0;
        __syncwarp();
        Ranks<ITEMS> rankOf;
        rankKeys<false, ITEMS>(key, first, n, shift, mask, sh.warpHist[warp], rankOf);
        __syncthreads();
        // Per digit: the counts summed over the warps, eight of them a
        // thread, each warp's turned into the sum before it.
        const uint32_t digit = t & 255, half = t >> 8;
        constexpr uint32_t kHalves = kClusterThreads / 256, kEach = kClusterWarps / kHalves;
        uint32_t of[kEach], sum = 0;
#pragma unroll
        for (uint32_t w = 0; w < kEach; w++) sum += of[w] = sh.warpHist[half * kEach + w][digit];
        sh.half[half][digit] = sum;
        __syncthreads();
        uint32_t run = 0, all = 0;
#pragma unroll
        for (uint32_t q = 0; q < kHalves; q++) {
            const uint32_t c = sh.half[q][digit];
            if (q < half) run += c;
            all += c;
        }
#pragma unroll
        for (uint32_t w = 0; w < kEach; w++) {
            sh.warpHist[half * kEach + w][digit] = run;
            run += of[w];
        }
        // The block's counts to every block: stores, whose way the barrier
        // waits for once, where loads after it would each wait for theirs.
        for (uint32_t b = half; b < blocks; b += kHalves) storeCluster(inBlock(&sh.counts[rank][digit], b), all);
        clusterMeet();  // the counts are final; every block has its keys in registers
        // The digit's keys in the blocks before this one, and in all of them.
        uint32_t before = 0, total = 0;
        if (t < 256) {
#pragma unroll
            for (uint32_t b = 0; b < kClusterBlocks; b++) {
                const uint32_t c = b < blocks ? sh.counts[b][t] : 0u;
                total += c;
                if (b < rank) before += c;
            }
        }
        before += scanDigits(total, sh.warpSums);
        if (t < 256) sh.place[t] = before;
        __syncthreads();
        const bool last = shift + 8 >= keyBits;
#pragma unroll
        for (uint32_t r = 0; r < ITEMS; r++) {
            if (first + r * 32 + lane >= n) continue;
            const uint32_t d = key[r] >> shift & mask;
            const uint32_t to = sh.place[d] + sh.warpHist[warp][d] + rankOf(r);
            if (last) {
                order[to] = val[r];
            } else {
                const uint32_t block = to / kTile, at = to % kTile;
                storeCluster(inBlock(&sh.pairs[at], block), key[r], val[r]);
            }
        }
        clusterMeet();  // the scatter has landed; no block leaves while another reads its counts
        if (last) break;
#pragma unroll
        for (uint32_t r = 0; r < ITEMS; r++) {
            const uint32_t at = warp * 32 * ITEMS + r * 32 + lane;
            key[r] = sh.pairs[at].x;
            val[r] = sh.pairs[at].y;
        }
    }
}

namespace {
// Whether the device takes the cluster sort's largest cluster (16 blocks is
// past what every device must take), asked once a device.
bool takesCluster(int device) {
    static std::atomic<int> known[64] = {};  // 0: not asked, 1: no, 2: yes
    if (device < 0 || device >= 64) return false;
    int k = known[device].load(std::memory_order_relaxed);
    if (k == 0) {
        auto kernel = clusterSortKernel<kClusterItems>;
        constexpr size_t kBytes = sizeof(ClusterSortShared<kClusterItems>);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kClusterBlocks);
        cfg.blockDim = dim3(kClusterThreads);
        cfg.dynamicSmemBytes = kBytes;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kClusterBlocks;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        const bool ok =
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBytes)) == cudaSuccess &&
            cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0;
        if (!ok) cudaGetLastError();
        k = ok ? 2 : 1;
        known[device].store(k, std::memory_order_relaxed);
    }
    return k == 2;
}

template <uint32_t ITEMS>
cudaError_t clusterSort(const uint32_t* keys, uint32_t* order, uint32_t n, uint32_t keyBits, cudaStream_t st) {
    constexpr size_t kBytes = sizeof(ClusterSortShared<ITEMS>);
    const uint32_t blocks = (n + kClusterThreads * ITEMS - 1) / (kClusterThreads * ITEMS);
    auto kernel = clusterSortKernel<ITEMS>;
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBytes))) ||
        (e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)))
        return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = kBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, keys, n, keyBits, order);
}

bool sortsInOneLaunch(uint32_t n, int device) { return n <= kClusterKeys && takesCluster(device); }
}  // namespace

uint32_t radixSortLaunches(uint32_t n, uint32_t keyBits) {
    if (n == 0) return 0;
    int device = 0;
    if (cudaGetDevice(&device) == cudaSuccess && sortsInOneLaunch(n, device)) return 1;
    return 1 + (keyBits + 7) / 8;  // the digit counts, then one launch per pass
}

cudaError_t radixSortU32(const uint32_t* keys, uint32_t* order, uint32_t n, uint32_t keyBits, void* temp,
                         size_t tempBytes, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    if (tempBytes < radixSortTempBytes(n) || n > kStatusValue || keyBits < 1 || keyBits > 32)
        return cudaErrorInvalidValue;
    char* p = static_cast<char*>(temp);
    const size_t vec = align256(size_t(n) * 4);
    uint32_t* keysA = reinterpret_cast<uint32_t*>(p);
    uint32_t* keysB = reinterpret_cast<uint32_t*>(p + vec);
    uint32_t* valsA = reinterpret_cast<uint32_t*>(p + 2 * vec);
    uint32_t* valsB = reinterpret_cast<uint32_t*>(p + 3 * vec);
    char* cleared = p + 4 * vec;
    uint32_t* totals = reinterpret_cast<uint32_t*>(cleared);
    uint32_t* tickets = totals + kSortMaxPasses * 256;
    uint32_t* error = tickets + kSortMaxPasses;
    uint32_t* status = reinterpret_cast<uint32_t*>(cleared + kSortHeadBytes);
    const uint32_t passes = (keyBits + 7) / 8;
    cudaError_t e;
    int device = 0, sms = 0;
    if ((e = cudaGetDevice(&device))) return e;
    if (sortsInOneLaunch(n, device)) {
        // The fewest keys a thread that sixteen blocks hold.
        constexpr uint32_t kOne = kClusterBlocks * kClusterThreads;
        return n <= kOne       ? clusterSort<1>(keys, order, n, keyBits, st)
               : n <= 2 * kOne ? clusterSort<2>(keys, order, n, keyBits, st)
               : n <= 4 * kOne ? clusterSort<4>(keys, order, n, keyBits, st)
                               : clusterSort<kClusterItems>(keys, order, n, keyBits, st);
    }
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device))) return e;
    const bool oneWave = (n + kSortTile - 1) / kSortTile <= 2u * uint32_t(sms);
    const uint32_t tile = oneWave ? kSortTile : kSortLargeTile, tiles = (n + tile - 1) / tile;
    if ((e = cudaMemsetAsync(cleared, 0, kSortHeadBytes + size_t(passes) * tiles * 256 * 4, st))) return e;
    // Eight blocks an SM, all that fit: the counters' round trips bound it.
    const uint32_t countGrid = std::min<uint32_t>(tiles, 8u * uint32_t(sms));
    if ((e = pdl(sortDigitCountKernel, countGrid, kCountThreads, 0, st, keys, n, keyBits, totals))) return e;
    const uint32_t* kin = keys;
    const uint32_t* vin = nullptr;
    for (uint32_t pass_ = 0; pass_ < passes; pass_++) {
        const uint32_t shift = 8 * pass_;
        const uint32_t bits = keyBits - shift < 8 ? keyBits - shift : 8;
        const uint32_t mask = (1u << bits) - 1u;
        const bool last = pass_ + 1 == passes;
        uint32_t* kout = last ? nullptr : (pass_ % 2 == 0 ? keysA : keysB);
        uint32_t* vout = last ? order : (pass_ % 2 == 0 ? valsA : valsB);
        auto pass = [&](auto kernel, size_t bytes) {
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
            if (e) return e;
            return pdl(kernel, tiles, kSortThreads, bytes, st, kin, vin, n, shift, mask,
                       (const uint32_t*)(totals + 256 * pass_), status + size_t(pass_) * tiles * 256,
                       tickets + pass_, error, kout, vout);
        };
        e = oneWave ? pass(sortPassKernel<kSortItems>, sizeof(PassShared<kSortItems>))
                    : pass(sortPassKernel<kSortLargeItems>, sizeof(PassShared<kSortLargeItems>));
        if (e) return e;
        kin = kout;
        vin = vout;
    }
    return cudaSuccess;
}

}  // namespace vsim

// ------------------------------------------------- sort without allocating --
//
// Some callers cannot allocate device memory: a host engine that owns every
// byte of the GPU through its own pool and forbids libraries to allocate
// behind its back, a real-time frame loop that may not risk cudaMalloc's
// implicit device synchronisation or an allocation stall mid-frame, or a thin
// binding handed nothing but raw device pointers. For them the sort below
// takes its scratch from a fixed array compiled into this library instead of
// from the caller: it allocates nothing and frees nothing.
//
// The array holds the scratch of kNoAllocMaxKeys keys (about 17 MiB) and lives
// on every GPU that loads the library until the process exits. Every call
// shares it, so calls whose work overlaps on the GPU -- on two streams, or from
// two threads -- race and corrupt each other's results; serialise them. The
// array keeps the last call's contents: each call first clears (with a memset
// on its stream) the words that must start at zero -- the look-back status
// words, digit totals and tile tickets -- and writes every other word before
// reading it.

namespace vsim {
namespace {

constexpr uint32_t kNoAllocMaxKeys = 1u << 20;
constexpr size_t kNoAllocScratchBytes = sortTempBytes(kNoAllocMaxKeys);

__device__ __align__(256) static unsigned char g_sortScratch[kNoAllocScratchBytes];

// In host code `g_sortScratch` names a host-side stand-in, not device memory:
// the device address comes from cudaGetSymbolAddress, looked up with the
// device current and cached per device together with the identity of the
// context it was looked up in. A device reset (cudaDeviceReset, or a primary
// context torn down and made again) reloads the module and may move the
// array; the next call sees a new context and looks the address up again.
constexpr int kMaxDevices = 64;
std::mutex g_scratchLock;
struct ScratchEntry {
    void* ptr;
    unsigned long long context;  // 0: unknown, never trusted
};
ScratchEntry g_scratchAddress[kMaxDevices] = {};

// The unique id of the calling thread's current context (cuCtxGetId), 0 when
// there is none or the driver cannot say. Reached through the runtime's
// driver entry points, so the library does not link libcuda itself.
unsigned long long currentContextId() {
    using GetCurrent = int (*)(void**);
    using GetId = int (*)(void*, unsigned long long*);
    static GetCurrent getCurrent = nullptr;
    static GetId getId = nullptr;
    static std::once_flag found;
    std::call_once(found, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &fn, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            getCurrent = reinterpret_cast<GetCurrent>(fn);
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &fn, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            getId = reinterpret_cast<GetId>(fn);
    });
    if (!getCurrent || !getId) return 0;
    void* ctx = nullptr;
    unsigned long long id = 0;
    if (getCurrent(&ctx) != 0 || !ctx || getId(ctx, &id) != 0) return 0;
    return id;
}

cudaError_t scratchAddress(void** out) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> hold(g_scratchLock);
    ScratchEntry& entry = g_scratchAddress[device];
    const unsigned long long context = currentContextId();
    if (!entry.ptr || context == 0 || entry.context != context) {
        void* ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_sortScratch);  // makes the device's context current if none was
        if (e != cudaSuccess) return e;
        entry.ptr = ptr;
        entry.context = context ? context : currentContextId();
    }
    *out = entry.ptr;
    return cudaSuccess;
}


}  // namespace

}  // namespace vsim

extern "C" int vsim_radix_sort_u32_noalloc(const uint32_t* d_keys, uint32_t* d_order, uint32_t n, uint32_t key_bits,
                                           void* stream) {
    using namespace vsim;
    clearError();
    if (key_bits < 1 || key_bits > 32) return fail(VSIM_ERR_RANGE, "key_bits must be in [1, 32]");
    if (n > kNoAllocMaxKeys)
        return fail(VSIM_ERR_CAPACITY, "vsim_radix_sort_u32_noalloc sorts at most 1048576 keys; use "
                                       "vsim_radix_sort_u32 with caller-provided scratch for more");
    if (n == 0) return VSIM_OK;
    if (!d_keys || !d_order) return fail(VSIM_ERR_INVALID, "keys or order is NULL");
    if (wordRangesOverlap(d_keys, d_order, n)) return fail(VSIM_ERR_INVALID, "keys and order overlap");
    void* scratch = nullptr;
    cudaError_t e = scratchAddress(&scratch);
    if (e != cudaSuccess) return fail(VSIM_ERR_CUDA, std::string("scratch address: ") + cudaGetErrorString(e));
    e = radixSortU32(d_keys, d_order, n, key_bits, scratch, kNoAllocScratchBytes, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return fail(VSIM_ERR_CUDA, std::string("radix sort: ") + cudaGetErrorString(e));
    return VSIM_OK;
}

