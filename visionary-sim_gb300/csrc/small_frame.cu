// A small scene's whole frame in one launch.
//
// A frame of a scene without contact is a chain of dependent passes: four row
// passes a sweep and the closing pass, ten substeps of them in a graph of
// launches, each waiting ~1.5 us for its turn and its nodes. Where every row
// pass is one group (at most 128 even and 128 odd cells), one block runs the
// frame with every node's state in shared memory: a pass is its two cells'
// arithmetic (1.3 us each, one warp a scheduler) and little else. The
// arithmetic is the passes' own (projectCellInRange, predictNode,
// finalizeNode). A 16x4x4 bar's ten substeps: 190 us as launches, 145 us here.
// More groups than one are left to the launches: a cluster of
// blocks handing nodes on through L2 was slower (a 31x9x10 bar's frame, four
// groups and the stretch limit: 1078 against 822 us), and one SM would take
// the groups one after another.
#include "row_pass.cuh"

namespace vsim {

namespace {

__global__ void __launch_bounds__(kRowBlock, 1) smallFrameKernel(SmallFrame f, const FrameParams* fp,
                                                                 const DevBody* __restrict__ bodies,
                                                                 const uint32_t* __restrict__ bodyActive,
                                                                 const uint32_t* __restrict__ active,
                                                                 const uint32_t* __restrict__ activeBody,
                                                                 const uint4* __restrict__ rows, DriveTables drive,
                                                                 float4* __restrict__ posOut, float4* __restrict__ prevOut,
                                                                 float4* __restrict__ velOut) {
    extern __shared__ float4 state[];
    float4* const pos = state;
    float4* const prev = pos + f.nodeCount;
    float4* const vel = prev + f.nodeCount;
    const uint32_t t = threadIdx.x;
    for (uint32_t n = t; n < f.nodeCount; n += kRowBlock) {
        pos[n] = posOut[n];
        prev[n] = prevOut[n];
        vel[n] = velOut[n];
    }
    __syncthreads();
    auto drives = [&](uint32_t n, float4 P) {
        const int32_t driven = f.driving ? drive.drivenOf[n] : -1;
        if (driven >= 0) applyDrive(fp, drive.offsets, drive.grabs, driven, n, P, pos, prev, vel);
    };
    for (uint32_t i = t; i < f.activeCount; i += kRowBlock) {
        if (!bodyActive[activeBody[i]]) continue;
        const uint32_t n = active[i];
        drives(n, predictNode(fp, n, pos, prev, vel));
    }
    __syncthreads();
    // The cells of a phase: pass phase / 2 % 4, even then odd.
    auto cellOf = [&](uint32_t phase) {
        const uint32_t q = phase / 2 % kRowPasses, group = f.rowStart[q];
        return group < f.rowStart[q + 1] ? rows[size_t(group) * kRowGroup + phase % 2 * kRowBlock + t]
                                         : make_uint4(0, 0, 0, 0);
    };
    const uint32_t phases = (f.iterations + (f.limited ? 3u : 0u)) * 2 * kRowPasses;
    for (uint32_t step = 0; step < f.steps; step++) {
        // The projection's sweeps, then the limit's own three.
        uint4 e = cellOf(0);
        uint32_t body = 0;
        CellConsts k = cellConsts(bodies);
        bool live = bodyActive[0] != 0;
#pragma unroll 1
        for (uint32_t phase = 0; phase < phases; phase++) {
            if ((e.y & ~kRowCell) != body) {
                body = e.y & ~kRowCell;
                k = cellConsts(bodies + body);
                live = bodyActive[body] != 0;
            }
            const uint4 cell = make_uint4(e.x, body, e.z & ((1u << kRowStrideBits) - 1), e.w);
            const bool project = phase < f.iterations * 2 * kRowPasses;
            const bool solve = (e.y & kRowCell) && live;
            if (phase + 1 < phases) e = cellOf(phase + 1);  // on its way while this one is solved
            if (solve && (project || k.maxStretch > 1.0f)) {
                uint32_t ids[8];
                cornerNodes(cell, ids);
                V p[8];
                float w[8];
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const float4 P = pos[ids[c]];
                    p[c] = xyz(P);
                    w[c] = P.w;
                }
                if (project && !projectCellInRange(p, [&](int c) { return sharedXyz(prev + ids[c]); }, w, k)) {
                    projectCellAgain(cell, bodies + body, pos, prev);
#pragma unroll
                    for (int c = 0; c < 8; c++) p[c] = xyz(pos[ids[c]]);
                }
                if (f.limited && k.maxStretch > 1.0f) limitStretch(p, w, k, f.lens);
#pragma unroll
                for (int c = 0; c < 8; c++) pos[ids[c]] = withW(p[c], w[c]);
            }
            __syncthreads();
        }
        const bool next = step + 1 < f.steps;
        for (uint32_t i = t; i < f.activeCount; i += kRowBlock) {
            const uint32_t body = activeBody[i];
            if (!bodyActive[body]) continue;
            const float friction = bodies[body].friction, damp = bodies[body].damp;
            if (next)
                finalizeNode<false, true>(fp, active[i], friction, damp, -1, pos, prev, vel, nullptr, nullptr, nullptr,
                                          drives);
            else
                finalizeNode<false, false>(fp, active[i], friction, damp, -1, pos, prev, vel, nullptr, nullptr, nullptr,
                                           drives);
        }
        __syncthreads();
    }
    for (uint32_t n = t; n < f.nodeCount; n += kRowBlock) {
        posOut[n] = pos[n];
        prevOut[n] = prev[n];
        velOut[n] = vel[n];
    }
}

}  // namespace

cudaError_t launchSmallFrame(cudaStream_t st, const DeviceState& s, const SmallFrame& f) {
    const size_t bytes = 3 * size_t(f.nodeCount) * sizeof(float4);
    if (cudaError_t e = cudaFuncSetAttribute(smallFrameKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             int(3 * kSmallNodes * sizeof(float4))))
        return e;
    const DriveTables drive{s.drivenOf, s.drivenOffset, s.grabs};
    smallFrameKernel<<<1, kRowBlock, bytes, st>>>(f, s.fp, s.bodies, s.bodyActive, s.active, s.activeBody, s.rows, drive,
                                                  s.pos, s.prev, s.vel);
    return cudaGetLastError();
}

}  // namespace vsim
