// A Gaussian cloud to an occupancy grid on the device: voxelizeCloud
// (packages/visionary-sim/src/sim/discretize/lattice/cloudVolume.js:101-397),
// the reference's "cloud" rest geometry (voxelLattice.js:208-226).
//
// The reference runs it on the CPU in JavaScript doubles. Here every step is
// a kernel whose every decision equals the one the same double arithmetic
// and order would take, so the grid is the same cell for cell. Double
// arithmetic is slow on this part, so decisions are taken in float wherever
// a proven error bound shows float gives the same answer, and in double
// only where it cannot:
//   1. bounds: each Gaussian's ellipsoid reach (materialBounds, :219-234),
//      estimated in float with a relative bound; the extremes reduced with
//      order-preserving 64-bit keys, then evaluated exactly for the few
//      Gaussians whose bracket can hold an extreme;
//   2. the grid laid out on the host from the bounds (gridForBounds,
//      voxelize.js:40-67);
//   3. stamp: a thread per Gaussian marks its centre cell and looks whether
//      its box has a cell that is still empty; those that do are tested cell
//      by cell against the ellipsoid (stampCloud, :138-178), box edges and
//      samples decided in float unless too close to call; a box that meets
//      more than two bricks of cells on an axis is walked by warps;
//   4. seal and fill (:291-306) on the cells packed 32 to a word along x:
//      6-neighbourhood dilations, the fill, as many erosions, the stamp put
//      back, the words written out as bytes once. The reference fills by
//      flooding the empty cells from the grid's faces (fillEnclosed,
//      :321-375); here the flood's set is reached by rounds of sweeps over
//      the words (an occluded fill along x, warp scans along y and z) to a
//      round that adds nothing, or, past a cap of rounds, found as the
//      face-connected components of empty cells that touch a face by a
//      concurrent union-find (x runs seeded by warp ballots, links by
//      atomicMin on roots, path halving by plain stores).
// Marking is an OR (a cell is set by any Gaussian that reaches it), and the
// components of a graph do not depend on the order edges are merged, so no
// step's result depends on thread timing.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>

#include <math_constants.h>

#include "float_bounds.cuh"
#include "frame_rows.cuh"
#include "sim_internal.cuh"

struct vsim_cloud_volume {
    int device = 0;
    cudaStream_t stream = nullptr;
    uint32_t dims[3]{};
    double origin[3]{};
    double h = 0;
    uint64_t cells = 0;
    uint64_t occupied = 0;
    uint64_t filled = 0;
    uint8_t* occupancy = nullptr;
};

namespace vsim {
namespace {

using bounds::Box;
using bounds::Ellipsoid;
using bounds::floatCellAt;
using bounds::floatTestOf;
using bounds::FloatTest;
using bounds::GridView;
using bounds::quickSample;
using bounds::sampleInside;
using bounds::hypotV8;
using bounds::kReachSlack;
using bounds::reachEstimate;

constexpr uint32_t kCloudBlock = 256;
// Caps of the union-find loops. Labels strictly fall along every walk, so
// the loops end by themselves; the caps, and the shared flag the first
// thread to reach one raises (every walk polls it), only bound the kernels'
// time on an input no test has seen.
constexpr uint32_t kFindLimit = 1u << 22;
constexpr uint32_t kUniteLimit = 1u << 16;
constexpr uint32_t kPollEvery = 1024;
// Rounds of flood sweeps before the union-find takes over (a round that
// adds nothing ends the flood; each turn of a path the sweeps' axes cannot
// follow in one round costs a round).
constexpr uint32_t kFloodRounds = 24;
std::atomic<uint32_t> floodRounds{kFloodRounds};

struct CloudInput {
    const float* pos;    // xyz per Gaussian
    const float* rot;    // quaternion x, y, z, w
    const float* scale;  // standard deviations per axis, metres
    uint32_t count;
    double sigma;
    float sigmaF;        // float(sigma)
};




// mat3.js:71-87 (mat3FromQuat), each entry rounded to float32 as its output
// array does, and the half-axes sigma * scale (cloudVolume.js:196-199).
__device__ void frameOf(const CloudInput& in, uint32_t i, Ellipsoid& e) {
    const double x = in.rot[4 * size_t(i)], y = in.rot[4 * size_t(i) + 1];
    const double z = in.rot[4 * size_t(i) + 2], w = in.rot[4 * size_t(i) + 3];
    e.col[0] = double(float(1.0 - 2.0 * (y * y + z * z)));
    e.col[1] = double(float(2.0 * (x * y + z * w)));
    e.col[2] = double(float(2.0 * (x * z - y * w)));
    e.col[3] = double(float(2.0 * (x * y - z * w)));
    e.col[4] = double(float(1.0 - 2.0 * (x * x + z * z)));
    e.col[5] = double(float(2.0 * (y * z + x * w)));
    e.col[6] = double(float(2.0 * (x * z + y * w)));
    e.col[7] = double(float(2.0 * (y * z - x * w)));
    e.col[8] = double(float(1.0 - 2.0 * (x * x + y * y)));
    for (int a = 0; a < 3; a++) e.radius[a] = in.sigma * double(in.scale[3 * size_t(i) + a]);
}

// The frame's entries as the float32 values frameOf rounds to: in float where
// every one is certified to equal the double path's rounding
// (frame_rows.cuh), else in double.
__device__ __forceinline__ void frameRows(const CloudInput& in, uint32_t i, float col[9]) {
    const float* q4 = in.rot + 4 * size_t(i);
    if (frame::rowsInFloat(q4[0], q4[1], q4[2], q4[3], col)) return;
    Ellipsoid full;
    frameOf(in, i, full);
    for (int q = 0; q < 9; q++) col[q] = float(full.col[q]);
}

// Doubles ordered as unsigned integers: the sign bit flipped on positives,
// every bit on negatives.
__device__ __forceinline__ unsigned long long orderedKey(double v) {
    const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v));
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

double fromOrderedKey(unsigned long long k) {
    const unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    double v;
    std::memcpy(&v, &u, 8);
    return v;
}

__device__ __forceinline__ unsigned long long warpMin64(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ unsigned long long warpMax64(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// The float side of the bounds and the stamp. For each Gaussian the bounds
// pass keeps a float estimate of its reach along each world axis and what the
// float frame may have put them off by (x, y, z, slack); a reach is NaN where
// it cannot be trusted, and only then is V8's hypot evaluated in double (FP64
// runs at a small fraction of the float rate on this part: a double division
// costs about a hundred float operations). The exact frame waits for the
// stamp, and for the Gaussians that need one there (2M Gaussians: 71 us with
// the frames certified and kept here, 41 without).

// The radii float(sigma) * scale for the estimate (within 2^-23 of the
// double sigma * scale of cloudVolume.js:196-199), NaN where out of its
// range.
__device__ void radiiOf(const CloudInput& in, uint32_t i, float rf[3]) {
    for (int a = 0; a < 3; a++) rf[a] = bounds::radiusEstimate(in.sigmaF, in.scale[3 * size_t(i) + a]);
}

// Floats ordered as unsigned integers (as orderedKey for doubles).
__device__ __forceinline__ uint32_t orderedKey32(float v) {
    const uint32_t u = __float_as_uint(v);
    return (u >> 31) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float fromOrderedKey32(uint32_t k) {
    return __uint_as_float((k >> 31) ? (k & 0x7fffffffu) : ~k);
}

// The exact reach along axis a (cloudVolume.js:201-209).
__device__ __noinline__ double exactReach(const CloudInput& in, uint32_t i, int a) {
    float col[9];
    frameRows(in, i, col);
    double v[3];
    for (int k = 0; k < 3; k++) {
        const float c = a == 0 ? col[3 * k] : a == 1 ? col[3 * k + 1] : col[3 * k + 2];
        v[k] = double(c) * (in.sigma * double(in.scale[3 * size_t(i) + k]));
    }
    return hypotV8(v[0], v[1], v[2]);
}

// cloudVolume.js:219-234 (materialBounds), first pass: per axis the smallest
// float upper bound on position - reach (keys[3..5]) and the largest float
// lower bound on position + reach (keys[0..2]) over all Gaussians, from the
// reach estimates with directed roundings; a Gaussian without an estimate is
// passed by, which leaves the bounds wider, not wrong. Fills `reach`. Reads
// 40 bytes a Gaussian and writes 16.
__global__ void __launch_bounds__(kCloudBlock) cloudBoundsKernel(CloudInput in, uint32_t* __restrict__ keys,
                                                                 float4* __restrict__ reach) {
    uint32_t lo[3] = {~0u, ~0u, ~0u}, hi[3] = {0, 0, 0};
    const bool quads = (reinterpret_cast<uintptr_t>(in.rot) & 15u) == 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < in.count; i += gridDim.x * blockDim.x) {
        const float* q4 = in.rot + 4 * size_t(i);
        const float4 q = quads ? *reinterpret_cast<const float4*>(q4) : make_float4(q4[0], q4[1], q4[2], q4[3]);
        float col[9], rf[3], hf[3];
        bounds::frameInFloat(q.x, q.y, q.z, q.w, col);
        radiiOf(in, i, rf);
        const float slack = bounds::reachSlack(q.x, q.y, q.z, q.w, rf);
        for (int a = 0; a < 3; a++) {
            const float p = in.pos[3 * size_t(i) + a];
            hf[a] = reachEstimate(col, rf, a);
            if (!isfinite(p) || !(slack <= 0x1p60f)) hf[a] = CUDART_NAN_F;
            if (isnan(hf[a])) continue;
            const float narrow = __fsub_rd(__fmul_rd(hf[a], float(1.0 - kReachSlack)), slack);  // <= reach
            lo[a] = min(lo[a], orderedKey32(__fsub_ru(p, narrow)));  // >= position - reach
            hi[a] = max(hi[a], orderedKey32(__fadd_rd(p, narrow)));  // <= position + reach
        }
        reach[i] = make_float4(hf[0], hf[1], hf[2], slack);
    }
    for (int a = 0; a < 3; a++) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = min(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = max(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
    }
    if ((threadIdx.x & 31) == 0) {
        // Six words that every warp adds to: only where it would change one.
        for (int a = 0; a < 3; a++) {
            if (lo[a] < __ldcg(keys + 3 + a)) atomicMin(keys + 3 + a, lo[a]);
            if (hi[a] > __ldcg(keys + a)) atomicMax(keys + a, hi[a]);
        }
    }
}

// Second pass: the exact extremes. Only a Gaussian whose position - reach can
// lie at or below the first pass's smallest upper bound can hold the minimum
// (every other one's exceeds it), and likewise for the maximum; those few get
// the exact reach and their exact bound into exact[0..5], and every Gaussian
// without an estimate does; a NaN among those raises *nan (Math.min and
// Math.max then give NaN). The test is in
// float, rounded outwards: position - reach >= RD(position - RU(RU(hf (1 +
// kReachSlack)) + slack)).
__global__ void cloudExtremesKernel(CloudInput in, const uint32_t* __restrict__ keys,
                                    const float4* __restrict__ reach, unsigned long long* __restrict__ exact,
                                    uint32_t* __restrict__ nan) {
    unsigned long long lo[3] = {~0ull, ~0ull, ~0ull}, hi[3] = {0, 0, 0};
    float bound[6];
    for (int q = 0; q < 6; q++) bound[q] = fromOrderedKey32(keys[q]);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < in.count; i += gridDim.x * blockDim.x) {
        const float4 r = reach[i];
        for (int a = 0; a < 3; a++) {
            const float p = in.pos[3 * size_t(i) + a];
            const float hf = a == 0 ? r.x : a == 1 ? r.y : r.z;
            bool low = true, high = true;
            if (!isnan(hf)) {
                const float wide = __fadd_ru(__fmul_ru(hf, float(1.0 + kReachSlack)), r.w);  // >= reach
                low = __fsub_rd(p, wide) <= bound[3 + a];
                high = __fadd_ru(p, wide) >= bound[a];
            }
            if (!(low || high)) continue;
            const double half = exactReach(in, i, a);
            if (isnan(double(p) - half) || isnan(double(p) + half)) atomicOr(nan, 1u);
            if (low) lo[a] = min(lo[a], orderedKey(double(p) - half));
            if (high) hi[a] = max(hi[a], orderedKey(double(p) + half));
        }
    }
    for (int a = 0; a < 3; a++) {
        lo[a] = warpMin64(lo[a]);
        hi[a] = warpMax64(hi[a]);
    }
    if ((threadIdx.x & 31) == 0) {
        for (int a = 0; a < 3; a++) {
            if (lo[a] != ~0ull) atomicMin(exact + a, lo[a]);
            if (hi[a] != 0) atomicMax(exact + 3 + a, hi[a]);
        }
    }
}

// cloudVolume.js:384-386 (cellOf) and :395-397 (offFace), on finite values.
__device__ __forceinline__ int64_t clampedCell(double v, double origin, double h, int64_t lo, int64_t hi) {
    const double f = floor((v - origin) / h);
    return static_cast<int64_t>(fmin(fmax(f, double(lo)), double(hi)));
}

// The float test of Gaussian i's box (bounds::floatTestInFloat), from the
// cloud's scales.
__device__ bool floatTestInFloat(const CloudInput& in, uint32_t i, const GridView& g, const Box& b, const double c[3],
                                 const float cf[3], const float col[9], FloatTest& f) {
    const float scale[3] = {in.scale[3 * size_t(i)], in.scale[3 * size_t(i) + 1], in.scale[3 * size_t(i) + 2]};
    return bounds::floatTestInFloat(g, b, c, cf, col, in.sigma, in.sigmaF, scale, f);
}

// The stamped cells, a bit each: 64 cells of a 4 x 4 x 4 brick to a word (bit
// x + 4 y + 16 z), bricks in x, y, z order. A Gaussian's box is a few cells
// wide, so one or two words (1.95 on average for boxes of two cells a side)
// hold the state of all of its cells, where bytes took a gather a cell.
struct Bricks {
    unsigned long long* bits;
    uint32_t nx, ny;  // bricks along x and y
    __device__ __forceinline__ unsigned long long* at(uint32_t bx, uint32_t by, uint32_t bz) const {
        return bits + (size_t(bz) * ny + by) * nx + bx;
    }
    __device__ __forceinline__ void set(uint32_t x, uint32_t y, uint32_t z) const {
        atomicOr(at(x >> 2, y >> 2, z >> 2), 1ull << ((x & 3) + 4 * (y & 3) + 16 * (z & 3)));
    }
};

// A box of cells, all of them in the grid: from lo to hi, hi included.
struct CellBox {
    uint32_t lo[3], hi[3];
    __device__ __forceinline__ uint32_t extent(int a) const { return hi[a] - lo[a] + 1; }
    // the box's cells in brick (bx, by, bz), which it meets
    __device__ __forceinline__ unsigned long long in(uint32_t bx, uint32_t by, uint32_t bz) const {
        const uint32_t x0 = max(lo[0], 4 * bx) & 3, x1 = min(hi[0] - 4 * bx, 3u);
        const uint32_t y0 = max(lo[1], 4 * by) & 3, y1 = min(hi[1] - 4 * by, 3u);
        const uint32_t z0 = max(lo[2], 4 * bz) & 3, z1 = min(hi[2] - 4 * bz, 3u);
        const uint32_t row = (0xfu << x0) & (0xfu >> (3 - x1));
        const uint32_t slice = row * ((0x1111u << 4 * y0) & (0xffffu >> 4 * (3 - y1)));
        return slice * ((0x0001000100010001ull << 16 * z0) & (~0ull >> 16 * (3 - z1)));
    }
    // Whether it meets at most two bricks along every axis.
    __device__ __forceinline__ bool small() const {
        return (hi[0] >> 2) - (lo[0] >> 2) < 2 && (hi[1] >> 2) - (lo[1] >> 2) < 2 && (hi[2] >> 2) - (lo[2] >> 2) < 2;
    }
    // A small box's empty cells: bit x + 4 y + 16 z of word dx + 2 dy + 4 dz
    // for a cell of the brick that lies (dx, dy, dz) after the box's first.
    // All of the words are read at once: one after another their round trips
    // were most of the stamp.
    __device__ __forceinline__ void empty(const Bricks& bricks, unsigned long long (&m)[8]) const {
        uint32_t row[2], col[2];       // x and y: the bits of a row, a row's bit in a slice
        unsigned long long slice[2];
        bool two[3];
        for (int a = 0; a < 3; a++) two[a] = (hi[a] >> 2) != (lo[a] >> 2);
        for (uint32_t d = 0; d < 2; d++) {
            const uint32_t x0 = d ? 0 : lo[0] & 3, x1 = d || !two[0] ? hi[0] & 3 : 3;
            const uint32_t y0 = d ? 0 : lo[1] & 3, y1 = d || !two[1] ? hi[1] & 3 : 3;
            const uint32_t z0 = d ? 0 : lo[2] & 3, z1 = d || !two[2] ? hi[2] & 3 : 3;
            row[d] = (0xfu << x0) & (0xfu >> (3 - x1));
            col[d] = (0x1111u << 4 * y0) & (0xffffu >> 4 * (3 - y1));
            slice[d] = (0x0001000100010001ull << 16 * z0) & (~0ull >> 16 * (3 - z1));
        }
        const unsigned long long* first = bricks.at(lo[0] >> 2, lo[1] >> 2, lo[2] >> 2);
        const size_t plane = size_t(bricks.nx) * bricks.ny;
#pragma unroll
        for (uint32_t q = 0; q < 8; q++) {
            const bool has = (!(q & 1) || two[0]) && (!(q & 2) || two[1]) && (!(q & 4) || two[2]);
            m[q] = has ? __ldcg(first + (q & 1) + (q & 2 ? bricks.nx : 0u) + (q & 4 ? plane : 0)) : ~0ull;
        }
#pragma unroll
        for (uint32_t q = 0; q < 8; q++) m[q] = slice[q >> 2] * (row[q & 1] * col[q >> 1 & 1]) & ~m[q];
    }
};

// A cell's sample, number s of nine, in its box's cells.
__device__ __forceinline__ int floatSampleOf(const FloatTest& f, float quick, float fi, float fj, float fk, int s) {
    const float ox = s == 8 ? 0.5f : float(s & 1), oy = s == 8 ? 0.5f : float((s >> 1) & 1);
    const float oz = s == 8 ? 0.5f : float((s >> 2) & 1);
    return quickSample(f, quick, fi + ox, fj + oy, fk + oz);
}

// Whether any sample of a cell is inside, in double. Unrolled: the samples'
// offsets repeat, and two thirds of their products with the frame with them
// (20,000 surfels of no thickness, boxes of 900 cells: 14.3 ms, as a loop 17.8).
__device__ __noinline__ bool exactCell(const CloudInput& in, uint32_t gaussian, const GridView& g, int64_t i, int64_t j,
                                       int64_t k) {
    Ellipsoid e;
    frameOf(in, gaussian, e);
    double c[3];
    for (int a = 0; a < 3; a++) c[a] = in.pos[3 * size_t(gaussian) + a];
#pragma unroll
    for (int s = 0; s < 9; s++)
        if (sampleInside(g, i, j, k, s, c, e)) return true;
    return false;
}

// Whether any sample of a cell from number s on is inside: s in double, and
// those after it that the float test cannot call.
__device__ __noinline__ bool exactFrom(const CloudInput& in, uint32_t gaussian, const GridView& g, const int64_t* lo,
                                       int64_t i, int64_t j, int64_t k, int s, const FloatTest& f, float quick) {
    Ellipsoid e;
    frameOf(in, gaussian, e);
    double c[3];
    for (int a = 0; a < 3; a++) c[a] = in.pos[3 * size_t(gaussian) + a];
    const float fi = float(int32_t(i - lo[0])), fj = float(int32_t(j - lo[1])), fk = float(int32_t(k - lo[2]));
    if (sampleInside(g, i, j, k, s, c, e)) return true;
    for (s++; s < 9; s++) {
        int inside = floatSampleOf(f, quick, fi, fj, fk, s);
        if (inside < 0) inside = sampleInside(g, i, j, k, s, c, e) ? 1 : 0;
        if (inside) return true;
    }
    return false;
}

// cloudVolume.js:170-173 for one cell of a box: any sample inside. What the
// float test cannot call (one sample in 10^5) is decided out of line: the
// double code would take the registers of half the warps.
//
// The float path converts nothing from double or 64-bit integers: on this
// part such conversions run on the FP64 pipe, and nine samples a cell made
// them the stamp's bottleneck. The cell's place in its box (under 2^20, so
// exact) is an int32 turned float once; the sample offsets are float
// constants.
__device__ __forceinline__ bool cellReached(const CloudInput& in, uint32_t gaussian, const GridView& g,
                                            const int64_t lo[3], int64_t i, int64_t j, int64_t k, const FloatTest* f,
                                            float quick) {
    if (!f) return exactCell(in, gaussian, g, i, j, k);
    const float fi = float(int32_t(i - lo[0])), fj = float(int32_t(j - lo[1])), fk = float(int32_t(k - lo[2]));
    int undecided = -1;
    bool reached = false;
#pragma unroll
    for (int s = 0; s < 9; s++) {
        const int inside = floatSampleOf(*f, quick, fi, fj, fk, s);
        if (inside == 0) continue;
        reached = inside > 0;
        if (inside < 0) undecided = s;
        break;
    }
    return undecided < 0 ? reached : exactFrom(in, gaussian, g, lo, i, j, k, undecided, *f, quick);
}


// Whether the float cells hold for a position on axis a (ranges that keep
// every term above a normal float's floor and below overflow).
__device__ __forceinline__ bool floatCellsHold(const GridView& g, float c, float reach) {
    return g.floatBound && g.invH > 0.0f && fabsf(c) <= 0x1p40f && reach <= 0x1p40f;
}

// As clampedCell: where hi < lo (a grid of one or two cells) it is hi.
__device__ __forceinline__ int64_t clampCell(int64_t v, int64_t lo, int64_t hi) { return min(max(v, lo), hi); }

// cloudVolume.js:384-386 for the centre: in float (false: not decided), or
// exact.
__device__ __forceinline__ bool floatCentre(const GridView& g, float c, int a, uint32_t& cell) {
    if (!floatCellsHold(g, c, 0.0f)) return false;
    const float co = c - g.originF[a];
    const float delta = bounds::cellDelta(g.originMag[a], c, co, 0.0f, g.invH);
    float at;
    if (!floatCellAt(co, 0.0f, 0.0f, g.invH, delta, at)) return false;
    cell = uint32_t(clampCell(int32_t(at), 0, int64_t(g.dims[a]) - 1));  // under 2^22, so an int32
    return true;
}

__device__ __forceinline__ uint32_t exactCentre(const GridView& g, float c, int a) {
    return uint32_t(clampedCell(double(c), g.origin[a], g.h, 0, int64_t(g.dims[a]) - 1));
}

// cloudVolume.js:147-160 along one axis: the cells from position - reach to
// position + reach, within one cell of the faces. With a reach estimate hf
// the exact reach lies in [hf (1 - kReachSlack) - slack, hf (1 + kReachSlack)
// + slack], also after those bounds are rounded to float (kReachSlack 2^-18
// against the estimate's 2^-21, slack twice what it must be), so each edge is
// the float cell of that interval; only an edge within delta of a cell
// boundary (or a Gaussian without an estimate) takes the exact reach and the
// double division.
__device__ __forceinline__ bool floatEdges(const GridView& g, int a, float c, const float4& reach, int32_t& lo,
                                           int32_t& hi) {
    const float hf = a == 0 ? reach.x : a == 1 ? reach.y : reach.z;
    const float narrow = hf * float(1.0 - kReachSlack) - reach.w, wide = hf * float(1.0 + kReachSlack) + reach.w;
    if (isnan(hf) || !floatCellsHold(g, c, wide)) return false;
    const float co = c - g.originF[a];
    const float delta = bounds::cellDelta(g.originMag[a], c, co, wide, g.invH);
    float l, u;
    const bool below = floatCellAt(co, -wide, -narrow, g.invH, delta, l);
    const bool above = floatCellAt(co, narrow, wide, g.invH, delta, u);
    if (!below || !above) return false;
    lo = int32_t(l);  // under 2^22; before the clamp to the faces
    hi = int32_t(u);
    return true;
}

__device__ __noinline__ void exactEdges(const CloudInput& in, uint32_t i, const GridView& g, int a, int64_t* edges) {
    const int64_t lo = 1, hi = int64_t(g.dims[a]) - 2;
    const double c = in.pos[3 * size_t(i) + a], half = exactReach(in, i, a);
    edges[0] = clampedCell(c - half, g.origin[a], g.h, lo, hi);
    edges[1] = clampedCell(c + half, g.origin[a], g.h, lo, hi);
}

__device__ __forceinline__ Box boxOf(const CloudInput& in, uint32_t i, const GridView& g,
                                     const float4* __restrict__ reach) {
    Box b;
    const float4 r = reach[i];
    for (int a = 0; a < 3; a++) {
        int32_t l, u;
        if (floatEdges(g, a, in.pos[3 * size_t(i) + a], r, l, u)) {
            b.lo[a] = clampCell(l, 1, int64_t(g.dims[a]) - 2);
            b.hi[a] = clampCell(u, 1, int64_t(g.dims[a]) - 2);
            continue;
        }
        int64_t edges[2];
        exactEdges(in, i, g, a, edges);
        b.lo[a] = edges[0];
        b.hi[a] = edges[1];
    }
    return b;
}

// The box where every edge is decided in float, of a grid with three cells
// or more on every axis.
__device__ __forceinline__ bool floatBox(const CloudInput& in, uint32_t i, const GridView& g,
                                         const float4* __restrict__ reach, CellBox& b) {
    bool ok = true;
    const float4 r = reach[i];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        int32_t l = 0, u = 0;
        ok = floatEdges(g, a, in.pos[3 * size_t(i) + a], r, l, u) && ok;
        const int32_t top = int32_t(min(g.dims[a] - 2, 1u << 30));
        b.lo[a] = uint32_t(max(1, min(l, top)));
        b.hi[a] = uint32_t(max(1, min(u, top)));
    }
    return ok;
}

__device__ __forceinline__ CellBox cellBox(const Box& b) {
    CellBox c;
    for (int a = 0; a < 3; a++) {
        c.lo[a] = uint32_t(b.lo[a]);
        c.hi[a] = uint32_t(b.hi[a]);
    }
    return c;
}

// Gaussians left for the pass that decides in double.
struct HardList {
    uint32_t* items;
    unsigned long long* count;
    __device__ __forceinline__ void add(uint32_t i) const { items[atomicAdd(count, 1ull)] = i; }
};

// One Gaussian's stamp as a walk over its box needs it, in shared memory.
struct StampEntry {
    FloatTest f;
    float quick;     // quickBound(f)
    uint32_t gaussian;
    uint32_t fast;   // the float test holds; else test in double
    CellBox box;
};

// The Gaussian's float test, from the frame formed again.
__device__ __forceinline__ bool testOf(const CloudInput& in, uint32_t i, const GridView& g, const Box& b,
                                       FloatTest& f) {
    float col[9], cf[3];
    double c[3];
    frameRows(in, i, col);
    for (int a = 0; a < 3; a++) {
        cf[a] = in.pos[3 * size_t(i) + a];
        c[a] = cf[a];
    }
    return floatTestInFloat(in, i, g, b, c, cf, col, f);
}

__device__ __forceinline__ void setUp(const CloudInput& in, uint32_t i, const GridView& g, const CellBox& box,
                                      StampEntry& e) {
    Box b;
    for (int a = 0; a < 3; a++) {
        b.lo[a] = box.lo[a];
        b.hi[a] = box.hi[a];
    }
    e.fast = testOf(in, i, g, b, e.f) ? 1u : 0u;
    e.quick = bounds::quickBound(e.f);
    e.gaussian = i;
    e.box = box;
}

__device__ __forceinline__ void markCell(const Bricks& bricks, const uint32_t at[3]) {
    unsigned long long* word = bricks.at(at[0] >> 2, at[1] >> 2, at[2] >> 2);
    const unsigned long long bit = 1ull << ((at[0] & 3) + 4 * (at[1] & 3) + 16 * (at[2] & 3));
    if ((__ldcg(word) & bit) == 0) atomicOr(word, bit);
}

constexpr uint32_t kStampBlock = 128;
constexpr uint32_t kStampBlocks = 7;  // an SM

// The place of the n-th set bit of a word that has more than n.
__device__ __forceinline__ uint32_t setBit(unsigned long long word, uint32_t n) {
    uint32_t w = uint32_t(word), at = 0;
    const uint32_t low = __popc(w);
    if (n >= low) {
        n -= low;
        w = uint32_t(word >> 32);
        at = 32;
    }
#pragma unroll
    for (uint32_t half = 16; half >= 1; half >>= 1) {
        const uint32_t here = __popc(w & ((1u << half) - 1u));
        if (n >= here) {
            n -= here;
            w >>= half;
            at += half;
        }
    }
    return at;
}

// cloudVolume.js:147-177 for boxes that meet at most two bricks on an axis;
// larger ones are listed for cloudStampBoxKernel. A block takes `rounds` times
// its threads of Gaussians and marks their centres. A Gaussian whose box then
// has no empty cell left is done (of 2M Gaussians on a surface of 418,000
// cells' centres 61 % at least); the others wait in shared memory until a
// block's worth of them can be set up together, since the set-up (the frame,
// the float test's bounds, some of them in double) costs more than finding
// that nothing is left to do. Then each warp walks the empty cells of its 32
// boxes as one list dealt to its lanes 32 at a time (a lane finds the Gaussian
// owning its cell by a binary search over the warp's running offsets).
// Marking is an OR: which lane tests a cell, and when, changes nothing; a cell
// that another marks meanwhile is tested for nothing.
//
// Its schedulers issue 0.56 of the time with the 26 warps an SM that its
// registers allow, waiting for the bricks' words (L2, at no two lanes' same
// place) the rest (2M Gaussians at 231 x 223 x 243 cells: 142 us, where setting
// every Gaussian up and walking bytes of all its cells took 405; with a
// brick's words read one after another 258). One wave of
// blocks: two of half as many rounds each take 20 us more, since the first
// rounds know the fewest marks.
//
// An edge or centre that float cannot decide (one of 250 Gaussians at 230 cells
// across) would hold its whole warp up for the exact reach and divisions, some
// four hundred double operations at 16 cycles a warp: such Gaussians are
// listed, and a second launch, HARD, takes
// them together.
template <bool HARD>
__global__ void __launch_bounds__(kStampBlock, HARD ? 4 : kStampBlocks) cloudStampKernel(const __grid_constant__ CloudInput in,
                                                                const __grid_constant__ GridView g,
                                                                const float4* __restrict__ reach, Bricks bricks,
                                                                uint32_t rounds, HardList hard,
                                                                uint32_t* __restrict__ big,
                                                                unsigned long long* __restrict__ bigCount) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ StampEntry entries[kStampBlock];
    __shared__ unsigned long long empties[8][kStampBlock];
    __shared__ uint32_t queue[2 * kStampBlock];
    __shared__ uint32_t queued;
    const uint32_t t = threadIdx.x, lane = t & 31, warpBase = t & ~31u;
    // Sets up a Gaussian a lane and walks the warp's empty cells.
    auto stamp = [&](bool active, uint32_t i, const CellBox& box) {
        uint32_t n = 0;
        if (active) {
            unsigned long long m[8];
            box.empty(bricks, m);
#pragma unroll
            for (uint32_t q = 0; q < 8; q++) {
                n += __popcll(m[q]);
                empties[q][t] = m[q];
            }
            if (n) setUp(in, i, g, box, entries[t]);
        }
        // The warp's running offsets: lane l's cells are [off, off + n).
        uint32_t incl = n;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(kAll, incl, d);
            if (lane >= uint32_t(d)) incl += v;
        }
        const uint32_t off = incl - n;
        const uint32_t total = __shfl_sync(kAll, incl, 31);
        __syncwarp();
        for (uint32_t base = 0; base < total; base += 32) {
            const uint32_t c = base + lane;
            // the last lane whose offset is at or below c (offsets never fall)
            uint32_t owner = 0;
#pragma unroll
            for (uint32_t step = 16; step >= 1; step >>= 1) {
                const uint32_t probe = __shfl_sync(kAll, off, owner + step);
                if (probe <= c) owner += step;
            }
            const uint32_t start = __shfl_sync(kAll, off, owner);
            if (c >= total) continue;
            const StampEntry& e = entries[warpBase + owner];
            // the cell: the (c - start)-th of the owner's empty ones
            uint32_t at = c - start, q = 0;
            unsigned long long m = empties[0][warpBase + owner];
            for (uint32_t here = __popcll(m); at >= here && q < 7; here = __popcll(m)) {
                at -= here;
                m = empties[++q][warpBase + owner];
            }
            const uint32_t bit = setBit(m, at);
            const uint32_t x = 4 * ((e.box.lo[0] >> 2) + (q & 1)) + (bit & 3);
            const uint32_t y = 4 * ((e.box.lo[1] >> 2) + (q >> 1 & 1)) + (bit >> 2 & 3);
            const uint32_t z = 4 * ((e.box.lo[2] >> 2) + (q >> 2)) + (bit >> 4);
            const int64_t lo[3] = {e.box.lo[0], e.box.lo[1], e.box.lo[2]};
            if (cellReached(in, e.gaussian, g, lo, x, y, z, e.fast ? &e.f : nullptr, e.quick)) bricks.set(x, y, z);
        }
        __syncwarp();  // the warp's entries have been read
    };
    if (HARD) {
        // Few, and the double chain of one axis is the time: a lane for each
        // axis, ten Gaussians a warp, the warps spread over the grid's blocks
        // first (2M Gaussians list about 8,000: 36 us with full warps, 23 so).
        constexpr uint32_t kTen = 10;
        const uint64_t listed = *hard.count;
        const uint32_t mine = lane / 3, axis = lane % 3;
        for (uint64_t base = ((t >> 5) * uint64_t(gridDim.x) + blockIdx.x) * kTen; base < listed;
             base += uint64_t(gridDim.x) * (kStampBlock / 32) * kTen) {
            uint32_t i = 0, centreAt = 0, l = 0, u = 0;
            if (mine < kTen && base + mine < listed) {
                i = hard.items[base + mine];
                const float c = in.pos[3 * size_t(i) + axis];
                if (!floatCentre(g, c, axis, centreAt)) centreAt = exactCentre(g, c, axis);
                int32_t lf, uf;
                int64_t edges[2];
                if (floatEdges(g, axis, c, reach[i], lf, uf)) {
                    edges[0] = clampCell(lf, 1, int64_t(g.dims[axis]) - 2);
                    edges[1] = clampCell(uf, 1, int64_t(g.dims[axis]) - 2);
                } else {
                    exactEdges(in, i, g, axis, edges);
                }
                l = uint32_t(edges[0]);
                u = uint32_t(edges[1]);
            }
            // gathered to a lane a Gaussian
            CellBox b;
            uint32_t centre[3];
#pragma unroll
            for (uint32_t a = 0; a < 3; a++) {
                centre[a] = __shfl_sync(kAll, centreAt, 3 * lane + a);
                b.lo[a] = __shfl_sync(kAll, l, 3 * lane + a);
                b.hi[a] = __shfl_sync(kAll, u, 3 * lane + a);
            }
            i = __shfl_sync(kAll, i, 3 * lane);
            bool small = false;
            if (lane < kTen && base + lane < listed) {
                markCell(bricks, centre);
                small = b.small();
                if (!small) big[atomicAdd(bigCount, 1ull)] = i;
            }
            stamp(small, i, b);
        }
        return;
    }
    if (t == 0) queued = 0;
    __syncthreads();
    const uint64_t first = uint64_t(blockIdx.x) * rounds * kStampBlock;
    for (uint32_t round = 0; round < rounds; round++) {
        const uint64_t at = first + uint64_t(round) * kStampBlock + t;
        bool left = false;
        if (at < in.count) {
            // cloudVolume.js:161: the centre's cell, unconditionally
            uint32_t centre[3];
            bool known = true;
#pragma unroll
            for (int a = 0; a < 3; a++) known = floatCentre(g, in.pos[3 * size_t(at) + a], a, centre[a]) && known;
            if (known) markCell(bricks, centre);
            CellBox b;
            if (!floatBox(in, uint32_t(at), g, reach, b) || !known) {
                hard.add(uint32_t(at));
            } else if (!b.small()) {
                big[atomicAdd(bigCount, 1ull)] = uint32_t(at);
            } else {
                unsigned long long m[8], any = 0;
                b.empty(bricks, m);
#pragma unroll
                for (uint32_t q = 0; q < 8; q++) any |= m[q];
                left = any != 0;
            }
        }
        const uint32_t keep = __ballot_sync(kAll, left);
        uint32_t slot = 0;
        if (lane == 0 && keep) slot = atomicAdd(&queued, uint32_t(__popc(keep)));
        slot = __shfl_sync(kAll, slot, 0) + __popc(keep & ((1u << lane) - 1u));
        if (left) queue[slot] = uint32_t(at);  // under kStampBlock wait from the round before
        __syncthreads();
        const uint32_t waiting = queued;
        __syncthreads();  // every thread has read it before the next round adds to it
        // The queue's last block's worth (in the last round all there is).
        uint32_t end = waiting;
        while (end >= kStampBlock || (end > 0 && round + 1 == rounds)) {
            const uint32_t take = min(end, kStampBlock);
            uint32_t i = 0;
            CellBox b;
            if (t < take) {
                i = queue[end - take + t];
                floatBox(in, i, g, reach, b);  // decided before
            }
            stamp(t < take, i, b);
            end -= take;
        }
        if (end != waiting) {
            __syncthreads();  // the queue's end has been read
            if (t == 0) queued = end;
            __syncthreads();
        }
    }
}

// The listed larger boxes, several to a block: one thread sets each up, then
// the block's warps walk the bricks of all of them, a brick's 64 cells two to
// a lane, and mark a brick by one OR. A brick with no empty cell of the box
// costs one read. A box whose samples all go to double (no float test holds,
// as for a surfel a thousandth of its width thick) is walked cell by cell
// instead: double operations cost a warp the same however few of its lanes
// hold a cell, and a brick at a box's edge holds few. Four blocks an SM (64 registers) against two with the exact
// samples inline (110): 20,000 Gaussians of 1,300 cells' boxes, a whole
// voxelisation 1,125 us with a block a box and byte cells, 1,175 with bricks
// at two blocks, 908 at four.
constexpr uint32_t kBoxThreads = 256;
constexpr uint32_t kBoxBlocks = 4;  // an SM
constexpr uint32_t kBoxBatch = kBoxThreads / 32;

__global__ void __launch_bounds__(kBoxThreads, kBoxBlocks) cloudStampBoxKernel(const __grid_constant__ CloudInput in,
                                                                   const __grid_constant__ GridView g,
                                                                   const float4* __restrict__ reach, Bricks bricks,
                                                                   const uint32_t* __restrict__ big,
                                                                   const unsigned long long* __restrict__ bigCount) {
    __shared__ StampEntry entries[kBoxBatch];
    __shared__ unsigned long long ends[kBoxBatch];
    const uint64_t listed = *bigCount;
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // as many a block as spreads the list over the grid
    const uint64_t even = (listed + gridDim.x - 1) / gridDim.x;
    const uint32_t batch = even < 1 ? 1 : even > kBoxBatch ? kBoxBatch : uint32_t(even);
    for (uint64_t base = uint64_t(blockIdx.x) * batch; base < listed; base += uint64_t(gridDim.x) * batch) {
        const uint32_t held = listed - base < batch ? uint32_t(listed - base) : batch;
        __syncthreads();
        if (t < held) {
            const uint32_t i = big[base + t];
            const CellBox box = cellBox(boxOf(in, i, g, reach));
            setUp(in, i, g, box, entries[t]);
            unsigned long long all = 1;
            const bool fast = entries[t].fast != 0;
            for (int a = 0; a < 3; a++) all *= fast ? (box.hi[a] >> 2) - (box.lo[a] >> 2) + 1 : box.extent(a);
            if (!fast) all = (all + 31) / 32;
            ends[t] = all;
        }
        __syncthreads();
        unsigned long long total = 0;
        for (uint32_t q = 0; q < held; q++) total += ends[q];
        for (unsigned long long task = warp; task < total; task += kBoxThreads / 32) {
            uint32_t q = 0;
            unsigned long long r = task;
            while (r >= ends[q]) r -= ends[q++];
            const StampEntry& e = entries[q];
            const int64_t lo[3] = {e.box.lo[0], e.box.lo[1], e.box.lo[2]};
            if (!e.fast) {
                const unsigned long long cell = r * 32 + lane;
                const uint32_t ex = e.box.extent(0), ey = e.box.extent(1);
                const unsigned long long row = cell / ex, plane = row / ey;
                if (plane >= e.box.extent(2)) continue;
                const uint32_t x = e.box.lo[0] + uint32_t(cell - row * ex), z = e.box.lo[2] + uint32_t(plane);
                const uint32_t y = e.box.lo[1] + uint32_t(row - plane * ey);
                const uint32_t bit = (x & 3) + 4 * (y & 3) + 16 * (z & 3);
                if (__ldcg(bricks.at(x >> 2, y >> 2, z >> 2)) >> bit & 1) continue;
                if (cellReached(in, e.gaussian, g, lo, x, y, z, nullptr, 0.0f)) bricks.set(x, y, z);
                continue;
            }
            const uint32_t bx0 = e.box.lo[0] >> 2, by0 = e.box.lo[1] >> 2, bz0 = e.box.lo[2] >> 2;
            const uint32_t ex = (e.box.hi[0] >> 2) - bx0 + 1, ey = (e.box.hi[1] >> 2) - by0 + 1;
            uint32_t bx, by, bz;
            if (r >> 32) {
                const unsigned long long row = r / ex;
                bx = uint32_t(r - row * ex);
                bz = uint32_t(row / ey);
                by = uint32_t(row - (unsigned long long)bz * ey);
            } else {
                const uint32_t row = uint32_t(r) / ex;
                bx = uint32_t(r) - row * ex;
                bz = row / ey;
                by = row - bz * ey;
            }
            bx += bx0;
            by += by0;
            bz += bz0;
            unsigned long long* word = bricks.at(bx, by, bz);
            // One lane's look for all: the ballots below are the whole warp's, and
            // lanes that read the word apart, other warps marking it meanwhile,
            // could part here.
            unsigned long long empty = lane == 0 ? e.box.in(bx, by, bz) & ~__ldcg(word) : 0ull;
            empty = __shfl_sync(0xffffffffu, empty, 0);
            if (empty == 0) continue;
            unsigned long long mark = 0;
#pragma unroll
            for (uint32_t half = 0; half < 2; half++) {
                const uint32_t bit = lane + 32 * half;
                bool in_ = (empty >> bit & 1) != 0;
                if (in_)
                    in_ = cellReached(in, e.gaussian, g, lo, 4 * bx + (bit & 3), 4 * by + (bit >> 2 & 3),
                                      4 * bz + (bit >> 4), &e.f, e.quick);
                mark |= static_cast<unsigned long long>(__ballot_sync(0xffffffffu, in_)) << 32 * half;
            }
            if (lane == 0 && mark) atomicOr(word, mark);
        }
    }
}

// The stamp of a grid with fewer than three cells on an axis (a flat cloud, no
// padding), where "within one cell of the faces" leaves the grid: the index is
// the reference's cellIndex of the (possibly out-of-grid) coordinates, and like a
// typed array the grid ignores an index outside it.

// The cell that (x, y, z) index, false where none.
__device__ __forceinline__ bool looseCell(const GridView& g, int64_t x, int64_t y, int64_t z, uint32_t at[3]) {
    const int64_t cell = x + int64_t(g.dims[0]) * (y + int64_t(g.dims[1]) * z);
    if (cell < 0 || cell >= int64_t(g.cells)) return false;
    const uint32_t row = uint32_t(cell) / g.dims[0];
    at[2] = row / g.dims[1];
    at[1] = row - at[2] * g.dims[1];
    at[0] = uint32_t(cell) - row * g.dims[0];
    return true;
}

__device__ __forceinline__ bool isMarked(const Bricks& bricks, const uint32_t at[3]) {
    const uint32_t bit = (at[0] & 3) + 4 * (at[1] & 3) + 16 * (at[2] & 3);
    return __ldcg(bricks.at(at[0] >> 2, at[1] >> 2, at[2] >> 2)) >> bit & 1;
}

struct LooseEntry {
    FloatTest f;
    float quick;
    int64_t lo[3];
    uint32_t ex, ey, gaussian, fast;
};

// A thread a Gaussian: its centre, its box, and whether the box has a cell that
// is still empty; larger boxes are listed for the kernel below. Each warp then
// deals the cells of those that do to its lanes, 32 at a time, as
// cloudStampKernel does (2M Gaussians on 501 x 1 x 501 cells, a whole
// voxelisation: 75 ms with a block a Gaussian, 0.46 so).
constexpr int64_t kLooseCells = 64;  // of a box that a warp's lanes share
__global__ void __launch_bounds__(kStampBlock) cloudStampLooseKernel(const __grid_constant__ CloudInput in,
                                                                     const __grid_constant__ GridView g,
                                                                     const float4* __restrict__ reach, Bricks bricks,
                                                                     uint32_t* __restrict__ big,
                                                                     unsigned long long* __restrict__ bigCount) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ LooseEntry entries[kStampBlock];
    const uint32_t t = threadIdx.x, lane = t & 31, warpBase = t & ~31u;
    const uint64_t i = uint64_t(blockIdx.x) * kStampBlock + t;
    uint32_t n = 0;
    if (i < in.count) {
        uint32_t at[3];
        for (int a = 0; a < 3; a++) {
            const float c = in.pos[3 * size_t(i) + a];
            if (!floatCentre(g, c, a, at[a])) at[a] = exactCentre(g, c, a);
        }
        markCell(bricks, at);
        const Box b = boxOf(in, uint32_t(i), g, reach);
        const int64_t ex = b.extent(0), ey = b.extent(1), ez = b.extent(2);
        if (ex > kLooseCells || ey > kLooseCells || ez > kLooseCells || ex * ey * ez > kLooseCells) {
            big[atomicAdd(bigCount, 1ull)] = uint32_t(i);
        } else {
            bool empty = false;
            for (int64_t z = b.lo[2]; z <= b.hi[2]; z++)
                for (int64_t y = b.lo[1]; y <= b.hi[1]; y++)
                    for (int64_t x = b.lo[0]; x <= b.hi[0]; x++)
                        if (looseCell(g, x, y, z, at) && !isMarked(bricks, at)) empty = true;
            if (empty) {
                LooseEntry& e = entries[t];
                e.fast = testOf(in, uint32_t(i), g, b, e.f) ? 1u : 0u;
                e.quick = bounds::quickBound(e.f);
                for (int a = 0; a < 3; a++) e.lo[a] = b.lo[a];
                e.ex = uint32_t(ex);
                e.ey = uint32_t(ey);
                e.gaussian = uint32_t(i);
                n = uint32_t(ex * ey * ez);
            }
        }
    }
    uint32_t incl = n;  // the warp's running offsets: lane l's cells are [off, off + n)
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(kAll, incl, d);
        if (lane >= uint32_t(d)) incl += v;
    }
    const uint32_t off = incl - n, total = __shfl_sync(kAll, incl, 31);
    __syncwarp();
    for (uint32_t base = 0; base < total; base += 32) {
        const uint32_t c = base + lane;
        uint32_t owner = 0;  // the last lane whose offset is at or below c
#pragma unroll
        for (uint32_t step = 16; step >= 1; step >>= 1) {
            const uint32_t probe = __shfl_sync(kAll, off, owner + step);
            if (probe <= c) owner += step;
        }
        const uint32_t first = __shfl_sync(kAll, off, owner);
        if (c >= total) continue;
        const LooseEntry& e = entries[warpBase + owner];
        const uint32_t row = (c - first) / e.ex, plane = row / e.ey;
        const int64_t x = e.lo[0] + (c - first - row * e.ex), y = e.lo[1] + (row - plane * e.ey), z = e.lo[2] + plane;
        uint32_t at[3];
        if (!looseCell(g, x, y, z, at) || isMarked(bricks, at)) continue;
        if (cellReached(in, e.gaussian, g, e.lo, x, y, z, e.fast ? &e.f : nullptr, e.quick)) markCell(bricks, at);
    }
}

// The larger boxes, a block each.
__global__ void __launch_bounds__(kCloudBlock) cloudStampLooseBoxKernel(const __grid_constant__ CloudInput in,
                                                                        const __grid_constant__ GridView g,
                                                                        const float4* __restrict__ reach, Bricks bricks,
                                                                        const uint32_t* __restrict__ big,
                                                                        const unsigned long long* __restrict__ bigCount) {
    __shared__ LooseEntry e;
    __shared__ Box b;
    const uint64_t listed = *bigCount;
    for (uint64_t n = blockIdx.x; n < listed; n += gridDim.x) {
        __syncthreads();  // the box before is done
        if (threadIdx.x == 0) {
            e.gaussian = big[n];
            b = boxOf(in, e.gaussian, g, reach);
            e.fast = testOf(in, e.gaussian, g, b, e.f) ? 1u : 0u;
            e.quick = bounds::quickBound(e.f);
        }
        __syncthreads();
        const int64_t ex = b.extent(0), ey = b.extent(1), cells = b.cells();
        for (int64_t t = threadIdx.x; t < cells; t += kCloudBlock) {
            const int64_t x = b.lo[0] + t % ex, y = b.lo[1] + t / ex % ey, z = b.lo[2] + t / (ex * ey);
            uint32_t at[3];
            if (!looseCell(g, x, y, z, at) || isMarked(bricks, at)) continue;
            if (cellReached(in, e.gaussian, g, b.lo, x, y, z, e.fast ? &e.f : nullptr, e.quick)) markCell(bricks, at);
        }
    }
}

struct Dims {
    uint32_t nx, ny, nz, cells;
};


// The root of a's tree. Labels only decrease along a path, so the walk ends;
// each step points a at its grandparent (path halving). A plain store is
// enough: the value written is an ancestor, and a link only ever lands on a
// root, which this never writes.
__device__ uint32_t findRoot(uint32_t* L, uint32_t a, uint32_t* err) {
    for (uint32_t step = 0; step < kFindLimit; step++) {
        const uint32_t p = __ldcg(L + a);
        if (p == a) return a;
        const uint32_t gp = __ldcg(L + p);
        if (gp != p) __stcg(L + a, gp);
        a = gp;
        if (step % kPollEvery == kPollEvery - 1 && *reinterpret_cast<volatile uint32_t*>(err)) return a;
    }
    atomicOr(err, 1u);
    return a;
}

// Joins the trees of a and b: the larger root is linked under the smaller
// with atomicMin; if it had been linked meanwhile, continue from its new
// parent. Every retry lowers a label, so it ends.
__device__ void unite(uint32_t* L, uint32_t a, uint32_t b, uint32_t* err) {
    for (uint32_t step = 0; step < kUniteLimit; step++) {
        a = findRoot(L, a, err);
        b = findRoot(L, b, err);
        if (a == b || *reinterpret_cast<volatile uint32_t*>(err)) return;
        if (a > b) {
            const uint32_t t = a;
            a = b;
            b = t;
        }
        const uint32_t old = atomicMin(L + b, a);
        if (old == b) return;
        b = old;
    }
    atomicOr(err, 1u);
}

// The labels seeded with x runs: a block takes kCloudBlock consecutive
// cells (a chunk starts at a multiple of kCloudBlock), and an empty cell
// whose -x neighbour is empty, in the same row and the same chunk, takes the
// label of its run's first cell (by ballot within a warp, then the last run
// start of the warps before it); every other cell labels itself. This joins
// the x edges inside a chunk without atomics.
__global__ void labelRunsKernel(const uint8_t* __restrict__ occ, uint32_t* __restrict__ L, Dims d) {
    __shared__ int lastStart[kCloudBlock / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t base = blockIdx.x * kCloudBlock; base < d.cells; base += gridDim.x * kCloudBlock) {
        const uint32_t idx = base + threadIdx.x;
        const bool empty = idx < d.cells && occ[idx] == 0;
        const bool linked = empty && threadIdx.x > 0 && occ[idx - 1] == 0 && idx % d.nx != 0;
        const uint32_t starts = __ballot_sync(0xffffffffu, !linked);
        if (lane == 31) lastStart[warp] = starts ? int(warp * 32 + 31 - __clz(starts)) : -1;
        __syncthreads();
        const uint32_t mine = starts & (0xffffffffu >> (31 - lane));
        int start = mine ? int(warp * 32 + 31 - __clz(mine)) : -1;
        for (int w = int(warp) - 1; start < 0 && w >= 0; w--) start = lastStart[w];
        // thread 0 is never linked, so every thread finds a start
        if (idx < d.cells) L[idx] = base + uint32_t(start);
        __syncthreads();
    }
}

// The remaining face-adjacent pairs of empty cells joined
// (cloudVolume.js:88-89, 359-364): an x edge across a chunk boundary; a y
// (z) edge unless the two cells' -x neighbours are both empty, in which case
// it is implied by edges already joined (cell ~ its -x neighbour ~ that
// one's -y (-z) neighbour ~ the cell's -y (-z) neighbour), so each stretch
// of overlapping runs is joined once, at its first cell.
__global__ void labelMergeKernel(const uint8_t* __restrict__ occ, uint32_t* L, Dims d, uint32_t* err) {
    const uint32_t plane = d.nx * d.ny;
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < d.cells; idx += gridDim.x * blockDim.x) {
        if (occ[idx] != 0) continue;
        const uint32_t i = idx % d.nx, j = (idx / d.nx) % d.ny, k = idx / plane;
        const bool left = i > 0 && occ[idx - 1] == 0;
        if (left && idx % kCloudBlock == 0) unite(L, idx, idx - 1, err);
        if (j > 0 && occ[idx - d.nx] == 0 && !(left && occ[idx - 1 - d.nx] == 0)) unite(L, idx, idx - d.nx, err);
        if (k > 0 && occ[idx - plane] == 0 && !(left && occ[idx - 1 - plane] == 0)) unite(L, idx, idx - plane, err);
    }
}

// The roots of the empty cells on the grid's faces marked reached (the
// flood's seeds, cloudVolume.js:344-352). After the merge the trees are
// fixed: the walks here only shorten paths, never change a root.
__global__ void markFaceRootsKernel(const uint8_t* __restrict__ occ, uint32_t* L, uint8_t* __restrict__ reached, Dims d,
                                    uint32_t* err) {
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < d.cells; idx += gridDim.x * blockDim.x) {
        if (occ[idx] != 0) continue;
        const uint32_t i = idx % d.nx, j = (idx / d.nx) % d.ny, k = idx / (d.nx * d.ny);
        if (i == 0 || j == 0 || k == 0 || i == d.nx - 1 || j == d.ny - 1 || k == d.nz - 1)
            reached[findRoot(L, idx, err)] = 1;
    }
}

__device__ __forceinline__ unsigned long long blockSum(unsigned long long v) {
    __shared__ unsigned long long part[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    unsigned long long total = 0;
    if (threadIdx.x == 0)
        for (uint32_t w = 0; w < (blockDim.x + 31) / 32; w++) total += part[w];
    return total;
}

// cloudVolume.js:367-374: every empty cell whose tree the flood did not
// reach becomes material; *filled counts them. The root is walked to, not
// read from the cell's label: a concurrent path-halving store may leave a
// label at an ancestor short of the root.
__global__ void fillEnclosedKernel(uint8_t* __restrict__ occ, uint32_t* L, const uint8_t* __restrict__ reached,
                                   uint32_t cells, unsigned long long* __restrict__ filled, uint32_t* err) {
    unsigned long long mine = 0;
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < cells; idx += gridDim.x * blockDim.x) {
        if (occ[idx] == 0 && !reached[findRoot(L, idx, err)]) {
            occ[idx] = 1;
            mine++;
        }
    }
    const unsigned long long total = blockSum(mine);
    if (threadIdx.x == 0 && total) atomicAdd(filled, total);
}

// Small device words of one run.
// ---------------------------------------------------------------- flood --
// The same set fillEnclosed's flood reaches (cloudVolume.js:321-375): the
// empty cells joined to an empty face cell by a path of face-adjacent empty
// cells. The grid's empty cells are packed 32 to a word along x (rows of
// nw words; bits past nx are clear, so never entered), the face cells seed
// `reached`, and sweeps spread it: along x within each row (an occluded
// fill, words carried into their neighbours, up then down), along y and z
// 32 columns at a time (a word takes its neighbour's reached bits where it
// is empty, then fills along x within itself). Every step only adds empty
// cells adjacent to reached ones, and a round of the three sweeps that adds
// nothing leaves a set closed under adjacency: the flood's set exactly. The
// rounds are capped; past the cap the union-find below decides instead.

struct Words {
    uint32_t nw;    // words per row
    uint32_t rows;  // ny * nz
    uint32_t ny, nz;
};

// Seeds g spread through the set bits of p towards higher (Up) or lower
// (Down) bit positions: Kogge-Stone occluded fill.
__device__ __forceinline__ uint32_t fillUp(uint32_t g, uint32_t p) {
    g |= p & (g << 1);
    p &= p << 1;
    g |= p & (g << 2);
    p &= p << 2;
    g |= p & (g << 4);
    p &= p << 4;
    g |= p & (g << 8);
    p &= p << 8;
    return g | (p & (g << 16));
}

__device__ __forceinline__ uint32_t fillDown(uint32_t g, uint32_t p) {
    g |= p & (g >> 1);
    p &= p >> 1;
    g |= p & (g >> 2);
    p &= p >> 2;
    g |= p & (g >> 4);
    p &= p >> 4;
    g |= p & (g >> 8);
    p &= p >> 8;
    return g | (p & (g >> 16));
}

// The valid bits of word `word` of a row (cells past nx are clear).
__device__ __forceinline__ uint32_t validBits(const Dims& d, uint32_t word) {
    const uint32_t count = min(32u, d.nx - word * 32);
    return count == 32 ? 0xffffffffu : (1u << count) - 1u;
}

// The stamp's bricks as words along x: a word is four cells each of eight
// bricks.
__global__ void brickWordsKernel(Bricks bricks, Dims d, Words w, uint32_t* __restrict__ bits) {
    const uint32_t total = w.rows * w.nw;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t row = t / w.nw, word = t - row * w.nw, z = row / w.ny, y = row - z * w.ny;
        const unsigned long long* brick = bricks.at(8 * word, y >> 2, z >> 2);
        const uint32_t shift = 4 * (y & 3) + 16 * (z & 3);
        uint32_t m = 0;
#pragma unroll
        for (uint32_t q = 0; q < 8; q++)
            if (8 * word + q < bricks.nx) m |= uint32_t(brick[q] >> shift & 0xf) << 4 * q;
        bits[t] = m;
    }
}

// A thread per word: bit b of word w of a row set where cell 32 w + b is.
__global__ void packCellsKernel(const uint8_t* __restrict__ occ, Dims d, Words w, uint32_t* __restrict__ bits) {
    const uint32_t total = w.rows * w.nw;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t row = t / w.nw, word = t - row * w.nw;
        const uint32_t first = word * 32, count = min(32u, d.nx - first);
        const uint8_t* cells = occ + size_t(row) * d.nx + first;
        uint32_t m = 0;
        for (uint32_t b = 0; b < count; b++) m |= uint32_t(cells[b] != 0) << b;
        bits[t] = m;
    }
}

// voxelize.js:402-435 (neighbourhoodPass) on packed words, a thread per
// word: a clear cell with a set face neighbour becomes set (dilate), a set
// cell with a clear one becomes clear (erode); outside the grid counts as
// clear. The x neighbours are the word shifted by one, the edge bits taken
// from the neighbouring words of the row.
template <bool DILATE>
__global__ void neighbourhoodWordsKernel(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, Dims d, Words w) {
    const uint32_t total = w.rows * w.nw, plane = w.nw * d.ny;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t row = t / w.nw, word = t - row * w.nw;
        const uint32_t j = row % d.ny, k = row / d.ny;
        const uint32_t c = src[t];
        const uint32_t left = word > 0 ? src[t - 1] : 0u, right = word + 1 < w.nw ? src[t + 1] : 0u;
        const uint32_t n[6] = {(c << 1) | (left >> 31), (c >> 1) | (right << 31), j > 0 ? src[t - w.nw] : 0u,
                               j + 1 < d.ny ? src[t + w.nw] : 0u, k > 0 ? src[t - plane] : 0u,
                               k + 1 < d.nz ? src[t + plane] : 0u};
        uint32_t out = c;
        for (int q = 0; q < 6; q++) out = DILATE ? (out | n[q]) : (out & n[q]);
        dst[t] = out & validBits(d, word);
    }
}

// A thread per word: the empty cells of the sealed grid, and as reached
// those on a face of the grid (the flood's seeds, cloudVolume.js:344-352).
__global__ void seedFloodKernel(const uint32_t* __restrict__ cur, Dims d, Words w, uint32_t* __restrict__ empty,
                                uint32_t* __restrict__ reached) {
    const uint32_t total = w.rows * w.nw;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t row = t / w.nw, word = t - row * w.nw;
        const uint32_t j = row % d.ny, k = row / d.ny;
        const uint32_t e = ~cur[t] & validBits(d, word);
        uint32_t face = (j == 0 || k == 0 || j == d.ny - 1 || k == d.nz - 1) ? 0xffffffffu : 0u;
        if (word == 0) face |= 1u;
        if (word == w.nw - 1) face |= 1u << ((d.nx - 1) % 32);
        empty[t] = e;
        reached[t] = e & face;
    }
}

// Along x: a thread per row, up then down, the edge bit carried between
// neighbouring words.
__global__ void sweepXKernel(Words w, const uint32_t* __restrict__ empty, uint32_t* __restrict__ reached,
                             uint32_t* __restrict__ changed) {
    bool grew = false;
    for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < w.rows; row += gridDim.x * blockDim.x) {
        uint32_t* r = reached + size_t(row) * w.nw;
        const uint32_t* e = empty + size_t(row) * w.nw;
        uint32_t carry = 0;
        for (uint32_t q = 0; q < w.nw; q++) {
            const uint32_t was = r[q], p = e[q];
            const uint32_t g = fillUp(was | (carry & p & 1u), p);
            carry = g >> 31;
            if (g != was) {
                r[q] = g;
                grew = true;
            }
        }
        carry = 0;
        for (uint32_t q = w.nw; q-- > 0;) {
            const uint32_t was = r[q], p = e[q];
            const uint32_t g = fillDown(was | ((carry << 31) & p), p);
            carry = g & 1u;
            if (g != was) {
                r[q] = g;
                grew = true;
            }
        }
    }
    if (__any_sync(0xffffffffu, grew) && (threadIdx.x & 31) == 0) atomicOr(changed, 1u);
}

// Along y (a line per word column of an xz plane: stride nw, lines nz) or
// z (a line per word column of an xy row: stride nw ny, lines ny), a warp per
// line. Along a line a word takes its predecessor's reached bits where it
// is empty, x -> r | (e & x): maps of that form compose associatively,
// (a2, b2) after (a1, b1) = (a2 | (b2 & a1), b2 & b1), so each lane folds its
// segment of the line into one map, a warp scan gives every lane the
// reached bits entering its segment, and a second walk applies them, each
// word also filled along x within itself. Up the line, then down.
__device__ void sweepLineWay(bool up, uint32_t lane, uint32_t length, uint32_t seg, size_t base, uint32_t stride,
                             const uint32_t* __restrict__ empty, uint32_t* __restrict__ reached, bool& grew) {
    constexpr unsigned kAll = 0xffffffffu;
    // lane l holds steps [l seg, (l + 1) seg), walked upwards or downwards;
    // the lanes come in lane order up, in reverse lane order down
    const uint32_t s0 = min(lane * seg, length), s1 = min(s0 + seg, length);
    auto at = [&](uint32_t s) { return base + size_t(s) * stride; };
    uint32_t a = 0, b = ~0u;
    if (up) {
        for (uint32_t s = s0; s < s1; s++) {
            const uint32_t e = empty[at(s)];
            a = reached[at(s)] | (e & a);
            b &= e;
        }
    } else {
        for (uint32_t s = s1; s-- > s0;) {
            const uint32_t e = empty[at(s)];
            a = reached[at(s)] | (e & a);
            b &= e;
        }
    }
    // inclusive scan in walk order (lane order up, reverse lane order down)
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t pa = up ? __shfl_up_sync(kAll, a, d) : __shfl_down_sync(kAll, a, d);
        const uint32_t pb = up ? __shfl_up_sync(kAll, b, d) : __shfl_down_sync(kAll, b, d);
        if (up ? lane >= d : lane + d < 32) {
            a |= b & pa;
            b &= pb;
        }
    }
    const uint32_t before = up ? __shfl_up_sync(kAll, a, 1) : __shfl_down_sync(kAll, a, 1);
    uint32_t carry = (up ? lane > 0 : lane < 31) ? before : 0u;
    auto apply = [&](uint32_t s) {
        const uint32_t was = reached[at(s)], e = empty[at(s)];
        const uint32_t g = fillDown(fillUp(was | (e & carry), e), e);
        carry = g;
        if (g != was) {
            reached[at(s)] = g;
            grew = true;
        }
    };
    if (up) {
        for (uint32_t s = s0; s < s1; s++) apply(s);
    } else {
        for (uint32_t s = s1; s-- > s0;) apply(s);
    }
}

__global__ void sweepLineKernel(Words w, uint32_t lines, uint32_t length, uint32_t stride, uint32_t lineStride,
                                const uint32_t* __restrict__ empty, uint32_t* __restrict__ reached,
                                uint32_t* __restrict__ changed) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t seg = (length + 31) / 32;
    bool grew = false;
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < lines * w.nw; t += warps) {
        const uint32_t line = t / w.nw, word = t - line * w.nw;
        const size_t base = size_t(line) * lineStride + word;
        sweepLineWay(true, lane, length, seg, base, stride, empty, reached, grew);
        __syncwarp();
        sweepLineWay(false, lane, length, seg, base, stride, empty, reached, grew);
        __syncwarp();
    }
    if (__any_sync(0xffffffffu, grew) && lane == 0) atomicOr(changed, 1u);
}

// cloudVolume.js:367-374 on the words: every empty cell not reached becomes
// material; *filled counts them. A thread per word.
__global__ void encloseWordsKernel(uint32_t* __restrict__ cur, Words w, const uint32_t* __restrict__ empty,
                                   const uint32_t* __restrict__ reached, unsigned long long* __restrict__ filled) {
    unsigned long long mine = 0;
    const uint32_t total = w.rows * w.nw;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t enclosed = empty[t] & ~reached[t];
        if (!enclosed) continue;
        mine += __popc(enclosed);
        cur[t] |= enclosed;
    }
    const unsigned long long sum = blockSum(mine);
    if (threadIdx.x == 0 && sum) atomicAdd(filled, sum);
}

// The cells of a | b as bytes (0 or 1) into occ, a thread per 16 cells of
// the byte grid (one 16-byte store where occ is 16-byte aligned, bytes
// otherwise); *occupied counts them when given.
__global__ void unpackCellsKernel(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, Dims d, Words w,
                                  uint8_t* __restrict__ occ, unsigned long long* __restrict__ occupied) {
    unsigned long long mine = 0;
    const uint32_t chunks = (d.cells + 15) / 16;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < chunks; q += gridDim.x * blockDim.x) {
        const uint32_t first = q * 16, count = min(16u, d.cells - first);
        uint32_t row = first / d.nx, i = first - row * d.nx;
        uint32_t at = ~0u, m = 0;
        uint32_t packed[4] = {0, 0, 0, 0};
#pragma unroll
        for (uint32_t c = 0; c < 16; c++) {
            if (c < count) {
                const uint32_t word = row * w.nw + (i >> 5);
                if (word != at) {
                    at = word;
                    m = a[word] | (b ? b[word] : 0u);
                }
                const uint32_t bit = (m >> (i & 31)) & 1u;
                packed[c >> 2] |= bit << (8 * (c & 3));
                mine += bit;
                if (++i == d.nx) {
                    i = 0;
                    row++;
                }
            }
        }
        if (count == 16 && (reinterpret_cast<uintptr_t>(occ) & 15u) == 0) {
            *reinterpret_cast<uint4*>(occ + first) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        } else {
            for (uint32_t c = 0; c < count; c++) occ[first + c] = uint8_t((packed[c >> 2] >> (8 * (c & 3))) & 1u);
        }
    }
    if (occupied) {
        const unsigned long long sum = blockSum(mine);
        if (threadIdx.x == 0 && sum) atomicAdd(occupied, sum);
    }
}

struct CloudScalars {
    uint32_t keys[6];             // the bounds' first pass, float keys: largest, then smallest
    unsigned long long exact[6];  // the exact extremes: smallest, then largest
    unsigned long long filled;
    unsigned long long occupied;
    unsigned long long bigCount;
    unsigned long long hardCount;
    uint32_t nan;
    uint32_t err;
    uint32_t changed[2];  // whether a flood round added cells, two rounds at a time
};

// Scratch comes from a stream-ordered memory pool of this library's own, one
// per device, that keeps what a call frees for the next call instead of
// unmapping it: repeated voxelisations do not remap hundreds of megabytes.
// The pool holds the largest scratch any call needed until the process exits.
int scratchPool(int device, cudaMemPool_t* out) {
    static std::mutex lock;
    static cudaMemPool_t pools[64] = {};
    if (device < 0 || device >= 64) return fail(VSIM_ERR_INVALID, "device ordinal out of range");
    std::lock_guard<std::mutex> hold(lock);
    if (!pools[device]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        CK(cudaMemPoolCreate(&pools[device], &props), "memory pool");
        uint64_t keep = ~0ull;
        CK(cudaMemPoolSetAttribute(pools[device], cudaMemPoolAttrReleaseThreshold, &keep), "memory pool");
    }
    *out = pools[device];
    return VSIM_OK;
}

// A pool allocation freed, in stream order, when it goes out of scope.
struct DeviceBuffer {
    void* p = nullptr;
    cudaStream_t stream = nullptr;
    ~DeviceBuffer() {
        if (p) cudaFreeAsync(p, stream);
    }
};

#define POOL_ALLOC(buffer, bytes, pool, st, what)                                         \
    do {                                                                                   \
        (buffer).stream = (st);                                                            \
        CK(cudaMallocFromPoolAsync(&(buffer).p, (bytes), (pool), (st)), what);             \
    } while (0)

uint32_t streamGrid(uint64_t items, int sms) {
    const uint64_t want = (items + kCloudBlock - 1) / kCloudBlock;
    return uint32_t(std::max<uint64_t>(1, std::min<uint64_t>(want, uint64_t(sms) * 8)));
}

int voxelizeCloud(vsim_cloud_volume* v, const CloudInput& in, const vsim_cloud_options& o) {
    cudaStream_t st = v->stream;
    int sms = 1;
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, v->device), "device attributes");
    cudaMemPool_t pool;
    if (int rc = scratchPool(v->device, &pool)) return rc;

    // 1. bounds
    DeviceBuffer scalarsBuf;
    POOL_ALLOC(scalarsBuf, sizeof(CloudScalars), pool, st, "cloud scratch");
    auto* sc = static_cast<CloudScalars*>(scalarsBuf.p);
    CK(cudaMemsetAsync(sc, 0, sizeof(CloudScalars), st), "cloud scratch");
    // of none the largest is 0, the smallest all ones
    CK(cudaMemsetAsync(sc->keys + 3, 0xff, sizeof(uint32_t) * 3 + sizeof(unsigned long long) * 3, st), "cloud scratch");
    DeviceBuffer reachBuf;
    POOL_ALLOC(reachBuf, size_t(in.count) * sizeof(float4), pool, st, "cloud scratch");
    auto* reach = static_cast<float4*>(reachBuf.p);
    cloudBoundsKernel<<<streamGrid(in.count, sms), kCloudBlock, 0, st>>>(in, sc->keys, reach);
    cloudExtremesKernel<<<streamGrid(in.count, sms), kCloudBlock, 0, st>>>(in, sc->keys, reach, sc->exact,
                                                                              &sc->nan);
    CK(cudaGetLastError(), "cloud bounds");
    CloudScalars got{};
    CK(cudaMemcpyAsync(&got, sc, sizeof got, cudaMemcpyDeviceToHost, st), "cloud bounds");
    CK(cudaStreamSynchronize(st), "cloud bounds");

    // cloudVolume.js:113-115, then 2. gridForBounds (voxelize.js:40-67)
    double lo[3], hi[3], extent[3];
    bool nan = got.nan != 0;
    for (int a = 0; a < 3; a++) {
        lo[a] = fromOrderedKey(got.exact[a]);
        hi[a] = fromOrderedKey(got.exact[3 + a]);
        extent[a] = hi[a] - lo[a];
        nan |= std::isnan(extent[a]);
    }
    if (nan || !(std::max(extent[0], std::max(extent[1], extent[2])) > 0))
        return fail(VSIM_ERR_INVALID, "voxelizeCloud: a cloud with no extent has no volume");
    const double h = o.element_size;
    if (!(h > 0 && std::isfinite(h)))
        return fail(VSIM_ERR_RANGE, "gridForBounds: elementSize must be a positive length in metres");
    double cells = 1;
    for (int a = 0; a < 3; a++) {
        const double n = std::max(1.0, std::ceil(extent[a] / h - 1e-6)) + 2.0 * o.padding;
        if (!(n < 4294967296.0)) return fail(VSIM_ERR_RANGE, "voxelizeCloud: the grid is too large");
        v->dims[a] = uint32_t(n);
        v->origin[a] = lo[a] - h * o.padding;
        cells *= n;
    }
    if (!(cells < 4294967296.0)) return fail(VSIM_ERR_RANGE, "voxelizeCloud: the grid has 2^32 cells or more");
    v->h = h;
    v->cells = uint64_t(cells);
    const uint32_t n = uint32_t(v->cells);
    const Dims d{v->dims[0], v->dims[1], v->dims[2], n};
    GridView g{};
    for (int a = 0; a < 3; a++) {
        g.dims[a] = v->dims[a];
        g.origin[a] = v->origin[a];
    }
    g.h = h;
    // float(1 / h) for the float cell estimate, which wants every quotient
    // it forms a normal float (quotients from 2^-60 / 2^40 up)
    const float invH = float(1.0 / h);
    g.invH = invH >= 0x1p-40f && invH <= 0x1p40f ? invH : 0.0f;
    g.hF = float(h);
    g.floatBound = h >= 0x1p-30 && h <= 0x1p30;
    for (int a = 0; a < 3; a++) {
        g.originF[a] = float(g.origin[a]);
        g.originMag[a] = std::max(std::fabs(g.originF[a]), 0x1p-100f);
        g.floatBound = g.floatBound && std::fabs(g.origin[a]) <= 0x1p40;
    }
    g.cells = n;

    CK(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&v->occupancy), n, pool, st), "cloud occupancy");

    // 3. stamp
    const Words W{(d.nx + 31) / 32, d.ny * d.nz, d.ny, d.nz};
    const size_t words = size_t(W.rows) * W.nw;
    const uint32_t wordGrid = streamGrid(words, sms);
    DeviceBuffer listsBuf, bricksBuf, wordsBuf;
    // a Gaussian is listed as hard at most once, and as large at most once
    POOL_ALLOC(listsBuf, size_t(in.count) * 2 * 4, pool, st, "cloud scratch");
    const HardList hard{static_cast<uint32_t*>(listsBuf.p), &sc->hardCount};
    uint32_t* big = hard.items + in.count;
    const size_t brickBytes = size_t((d.nx + 3) / 4) * ((d.ny + 3) / 4) * ((d.nz + 3) / 4) * 8;
    POOL_ALLOC(bricksBuf, brickBytes, pool, st, "cloud scratch");
    const Bricks bricks{static_cast<unsigned long long*>(bricksBuf.p), (d.nx + 3) / 4, (d.ny + 3) / 4};
    CK(cudaMemsetAsync(bricksBuf.p, 0, brickBytes, st), "cloud stamp");
    if (d.nx < 3 || d.ny < 3 || d.nz < 3) {
        cloudStampLooseKernel<<<uint32_t((uint64_t(in.count) + kStampBlock - 1) / kStampBlock), kStampBlock, 0, st>>>(
            in, g, reach, bricks, big, &sc->bigCount);
        cloudStampLooseBoxKernel<<<uint32_t(sms) * 4, kCloudBlock, 0, st>>>(in, g, reach, bricks, big, &sc->bigCount);
    } else {
        // As many rounds as make the blocks one wave.
        const uint64_t wave = uint64_t(sms) * kStampBlocks * kStampBlock;
        const uint32_t rounds = uint32_t((in.count + wave - 1) / wave);
        const uint64_t each = uint64_t(rounds) * kStampBlock;
        cloudStampKernel<false><<<uint32_t((in.count + each - 1) / each), kStampBlock, 0, st>>>(
            in, g, reach, bricks, rounds, hard, big, &sc->bigCount);
        // The last two on as many blocks as fit at their registers: they loop.
        cloudStampKernel<true><<<uint32_t(sms) * 4, kStampBlock, 0, st>>>(in, g, reach, bricks, 0, hard, big,
                                                                           &sc->bigCount);
        cloudStampBoxKernel<<<uint32_t(sms) * kBoxBlocks, kBoxThreads, 0, st>>>(in, g, reach, bricks, big, &sc->bigCount);
    }
    POOL_ALLOC(wordsBuf, words * (o.fill ? 5 : 1) * sizeof(uint32_t), pool, st, "cloud scratch");
    uint32_t* stampW = static_cast<uint32_t*>(wordsBuf.p);
    brickWordsKernel<<<wordGrid, kCloudBlock, 0, st>>>(bricks, d, W, stampW);
    CK(cudaGetLastError(), "cloud stamp");

    // 4. seal and fill
    const uint32_t grid = streamGrid(n, sms);
    if (o.fill) {
        // The seal and fill on the cells packed 32 to a word along x: `seal`
        // dilations of the stamp, the flood, the enclosed cells
        // set, `seal` erosions, the stamp put back as the words are written
        // out as bytes once.
        uint32_t* cur = stampW + words;
        uint32_t* other = cur + words;
        uint32_t* emptyW = other + words;
        uint32_t* reachedW = emptyW + words;
        const uint32_t* src = stampW;
        for (uint32_t p = 0; p < o.seal; p++) {
            neighbourhoodWordsKernel<true><<<wordGrid, kCloudBlock, 0, st>>>(src, cur, d, W);
            src = cur;
            std::swap(cur, other);
        }
        if (src != stampW) std::swap(cur, other);  // cur: the sealed grid
        else CK(cudaMemcpyAsync(cur, stampW, words * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st), "cloud fill");
        // The flood by sweeps, to a round that adds nothing; past the cap of
        // rounds the union-find decides.
        seedFloodKernel<<<wordGrid, kCloudBlock, 0, st>>>(cur, d, W, emptyW, reachedW);
        // a warp per line, four to a block
        auto lineBlocks = [](uint64_t lines) { return uint32_t(std::max<uint64_t>(1, (lines + 3) / 4)); };
        // Two rounds a look at the device: a grid seldom floods in one, and the
        // look costs as much as half a round.
        bool converged = false;
        const uint32_t rounds = floodRounds.load();
        for (uint32_t round = 0; round < rounds && !converged; round += 2) {
            const uint32_t now = std::min(2u, rounds - round);
            CK(cudaMemsetAsync(sc->changed, 0, sizeof sc->changed, st), "cloud flood");
            for (uint32_t r = 0; r < now; r++) {
                sweepXKernel<<<uint32_t((W.rows + 127) / 128), 128, 0, st>>>(W, emptyW, reachedW, sc->changed + r);
                sweepLineKernel<<<lineBlocks(uint64_t(d.nz) * W.nw), 128, 0, st>>>(
                    W, d.nz, d.ny, W.nw, W.nw * d.ny, emptyW, reachedW, sc->changed + r);
                sweepLineKernel<<<lineBlocks(uint64_t(d.ny) * W.nw), 128, 0, st>>>(
                    W, d.ny, d.nz, W.nw * d.ny, W.nw, emptyW, reachedW, sc->changed + r);
            }
            CK(cudaGetLastError(), "cloud flood");
            uint32_t changed[2] = {1, 1};
            CK(cudaMemcpyAsync(changed, sc->changed, now * sizeof(uint32_t), cudaMemcpyDeviceToHost, st),
               "cloud flood");
            CK(cudaStreamSynchronize(st), "cloud flood");
            for (uint32_t r = 0; r < now; r++) converged |= changed[r] == 0;
        }
        if (converged) {
            encloseWordsKernel<<<wordGrid, kCloudBlock, 0, st>>>(cur, W, emptyW, reachedW, &sc->filled);
        } else {
            // the sealed grid as bytes, filled by the union-find, packed back
            DeviceBuffer work;
            const size_t sealedAt = (size_t(n) * 4 + 15) / 16 * 16;
            POOL_ALLOC(work, sealedAt + size_t(n) * 2 + 64, pool, st, "cloud fill scratch");
            auto* labels = static_cast<uint32_t*>(work.p);
            uint8_t* sealed = static_cast<uint8_t*>(work.p) + sealedAt;
            uint8_t* reached = sealed + n;
            unpackCellsKernel<<<streamGrid((n + 15) / 16, sms), kCloudBlock, 0, st>>>(cur, nullptr, d, W, sealed,
                                                                                       nullptr);
            CK(cudaMemsetAsync(reached, 0, n, st), "cloud fill");
            labelRunsKernel<<<grid, kCloudBlock, 0, st>>>(sealed, labels, d);
            labelMergeKernel<<<grid, kCloudBlock, 0, st>>>(sealed, labels, d, &sc->err);
            markFaceRootsKernel<<<grid, kCloudBlock, 0, st>>>(sealed, labels, reached, d, &sc->err);
            fillEnclosedKernel<<<grid, kCloudBlock, 0, st>>>(sealed, labels, reached, n, &sc->filled, &sc->err);
            packCellsKernel<<<wordGrid, kCloudBlock, 0, st>>>(sealed, d, W, cur);
            CK(cudaStreamSynchronize(st), "cloud fill");  // before `work` is freed
        }
        for (uint32_t p = 0; p < o.seal; p++) {
            neighbourhoodWordsKernel<false><<<wordGrid, kCloudBlock, 0, st>>>(cur, other, d, W);
            std::swap(cur, other);
        }
        unpackCellsKernel<<<streamGrid((n + 15) / 16, sms), kCloudBlock, 0, st>>>(cur, stampW, d, W, v->occupancy,
                                                                                   &sc->occupied);
        CK(cudaGetLastError(), "cloud fill");
        CK(cudaMemcpyAsync(&got, sc, sizeof got, cudaMemcpyDeviceToHost, st), "cloud fill");
        CK(cudaStreamSynchronize(st), "cloud fill");  // before the words are freed
    } else {
        unpackCellsKernel<<<streamGrid((n + 15) / 16, sms), kCloudBlock, 0, st>>>(stampW, nullptr, d, W, v->occupancy,
                                                                                   &sc->occupied);
        CK(cudaGetLastError(), "cloud stamp");
        CK(cudaMemcpyAsync(&got, sc, sizeof got, cudaMemcpyDeviceToHost, st), "cloud stamp");
        CK(cudaStreamSynchronize(st), "cloud stamp");
    }
    if (got.err) return fail(VSIM_ERR_TIMEOUT, "voxelizeCloud: the fill's union-find reached its iteration cap");
    v->filled = got.filled;
    v->occupied = got.occupied;
    return VSIM_OK;
}

int checkOptions(const vsim_cloud_options* o, uint64_t count) {
    if (!o) return fail(VSIM_ERR_INVALID, "options is NULL");
    if (count == 0) return fail(VSIM_ERR_INVALID, "voxelizeCloud: a cloud with no Gaussians has no volume");
    if (count > 0xffffffffull) return fail(VSIM_ERR_RANGE, "voxelizeCloud: at most 2^32 - 1 Gaussians");
    return VSIM_OK;
}

int newVolume(vsim_cloud_volume** out, vsim_cloud_volume** made) {
    if (!out) return fail(VSIM_ERR_INVALID, "out is NULL");
    *out = nullptr;
    auto* v = new (std::nothrow) vsim_cloud_volume();
    if (!v) return fail(VSIM_ERR_NOMEM, "host allocation failed");
    CK(cudaGetDevice(&v->device), "current device");
    const cudaError_t e = cudaStreamCreateWithFlags(&v->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        delete v;
        return cudaFail(e, "stream");
    }
    *made = v;
    return VSIM_OK;
}

void destroyVolume(vsim_cloud_volume* v) {
    if (!v) return;
    if (v->occupancy) cudaFreeAsync(v->occupancy, v->stream);
    if (v->stream) cudaStreamDestroy(v->stream);
    delete v;
}

}  // namespace
}  // namespace vsim

using namespace vsim;

extern "C" {

int vsim_voxelize_cloud_device(const float* d_positions, const float* d_rotations, const float* d_scales,
                               uint64_t count, const vsim_cloud_options* options, void* stream,
                               vsim_cloud_volume** out) {
    clearError();
    if (int rc = checkOptions(options, count)) return rc;
    if (!d_positions || !d_rotations || !d_scales) return fail(VSIM_ERR_INVALID, "NULL cloud array");
    vsim_cloud_volume* v = nullptr;
    if (int rc = newVolume(out, &v)) return rc;
    // the caller's work on the inputs finishes first
    cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
    int rc = e == cudaSuccess ? VSIM_OK : cudaFail(e, "caller stream");
    if (!rc) rc = voxelizeCloud(v, CloudInput{d_positions, d_rotations, d_scales, uint32_t(count), options->sigma, float(options->sigma)},
                                *options);
    if (rc) {
        cudaStreamSynchronize(v->stream);
        destroyVolume(v);
        return rc;
    }
    *out = v;
    return VSIM_OK;
}

namespace {

// Host inputs copied into pool memory on the volume's stream, then the device path.
int voxelizeHostCloud(vsim_cloud_volume* v, const float* positions, const float* rotations, const float* scales,
                      size_t n, const vsim_cloud_options& o) {
    cudaMemPool_t pool;
    if (int rc = scratchPool(v->device, &pool)) return rc;
    DeviceBuffer inputs;
    POOL_ALLOC(inputs, n * 40, pool, v->stream, "cloud inputs");
    auto* dPos = static_cast<float*>(inputs.p);
    float* dRot = dPos + 3 * n;
    float* dScale = dRot + 4 * n;
    CK(cudaMemcpyAsync(dPos, positions, n * 12, cudaMemcpyHostToDevice, v->stream), "cloud inputs");
    CK(cudaMemcpyAsync(dRot, rotations, n * 16, cudaMemcpyHostToDevice, v->stream), "cloud inputs");
    CK(cudaMemcpyAsync(dScale, scales, n * 12, cudaMemcpyHostToDevice, v->stream), "cloud inputs");
    return voxelizeCloud(v, CloudInput{dPos, dRot, dScale, uint32_t(n), o.sigma, float(o.sigma)}, o);
}

}  // namespace

int vsim_voxelize_cloud(const float* positions, const float* rotations, const float* scales, uint64_t count,
                        const vsim_cloud_options* options, vsim_cloud_volume** out) {
    clearError();
    if (int rc = checkOptions(options, count)) return rc;
    if (!positions || !rotations || !scales) return fail(VSIM_ERR_INVALID, "NULL cloud array");
    vsim_cloud_volume* v = nullptr;
    if (int rc = newVolume(out, &v)) return rc;
    const int rc = voxelizeHostCloud(v, positions, rotations, scales, size_t(count), *options);
    if (rc) {
        cudaStreamSynchronize(v->stream);
        destroyVolume(v);
        return rc;
    }
    *out = v;
    return VSIM_OK;
}

int vsim_cloud_volume_grid(const vsim_cloud_volume* volume, vsim_cloud_grid* out) {
    clearError();
    if (!volume || !out) return fail(VSIM_ERR_INVALID, "NULL argument");
    for (int a = 0; a < 3; a++) {
        out->dims[a] = volume->dims[a];
        out->origin[a] = volume->origin[a];
    }
    out->h = volume->h;
    out->occupied = volume->occupied;
    out->filled = volume->filled;
    return VSIM_OK;
}

int vsim_cloud_volume_read(vsim_cloud_volume* volume, uint8_t* occupancy, size_t cells) {
    clearError();
    if (!volume || !occupancy) return fail(VSIM_ERR_INVALID, "NULL argument");
    if (cells < volume->cells) return fail(VSIM_ERR_CAPACITY, "occupancy buffer smaller than the grid");
    DeviceGuard guard(volume->device);
    CK(cudaMemcpyAsync(occupancy, volume->occupancy, volume->cells, cudaMemcpyDeviceToHost, volume->stream),
       "read occupancy");
    CK(cudaStreamSynchronize(volume->stream), "read occupancy");
    return VSIM_OK;
}

int vsim_cloud_volume_destroy(vsim_cloud_volume* volume) {
    clearError();
    if (!volume) return VSIM_OK;
    DeviceGuard guard(volume->device);
    destroyVolume(volume);
    return VSIM_OK;
}

uint32_t vsim_cloud_set_flood_rounds(uint32_t rounds) { return floodRounds.exchange(rounds); }

}  // extern "C"
