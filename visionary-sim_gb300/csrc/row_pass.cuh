// A group of a row pass (kRowBlock): its even cells, then its odd ones, by one
// block. Shared by the row pass (step_kernels.cu) and the kernel that runs a
// small scene's whole frame (small_frame.cu).
#pragma once

#include "step_device.cuh"

namespace vsim {

__device__ __forceinline__ void copyAsync16(float4* dst, const float4* src) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// A record's x, y and z in shared memory, read anew at every call (the
// compiler would keep it in registers from its first use to its last).
__device__ __forceinline__ V sharedXyz(const float4* record) {
    float x, y, z, w;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(x), "=f"(y), "=f"(z), "=f"(w)
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(record))));
    return mk(x, y, z);
}

// What a block keeps of its group: the odd cells' positions, by corner, and
// the even and the odd cells' previous positions.
struct RowShared {
    float4 stage[8][kRowBlock];
    float4 before[2][8][kRowBlock];
};

// The group's cells projected (with `project`) and their stretch limited (with
// `limit`, where their body limits it), by the kRowBlock threads of a block.
// ready() is called once the tables are read and before any node is, solved()
// between the last arithmetic and the odd cells' stores.
//
// The odd cells' sixteen node records are copied to shared memory (cp.async)
// while the even cells are solved; each even cell then puts the faces that an
// odd cell holds into that cell's copy, and stores the others. So every node
// is loaded about once and stored once for the two colours.
template <class Ready, class Solved>
__device__ __forceinline__ void rowGroup(const uint4* group, const DevBody* bodies, const uint32_t* bodyActive,
                                         float4* pos, const float4* prevState, const StretchLengths& lens, bool project,
                                         bool limit, RowShared& shared, Ready&& ready, Solved&& solved) {
    auto& stage = shared.stage;
    auto& before = shared.before;
    const uint32_t t = threadIdx.x;
    const uint4 even = group[t], odd = group[kRowBlock + t];
    auto takesPart = [&](uint4 e, float maxStretch) {
        return (e.y & kRowCell) && bodyActive[e.y & ~kRowCell] && (project || maxStretch > 1.0f);
    };
    const uint32_t oddBody = odd.y & ~kRowCell;
    uint32_t body = even.y & ~kRowCell;  // an empty slot names body 0
    CellConsts k = cellConsts(bodies + body);
    bool solve = takesPart(even, k.maxStretch);
    const bool solveOdd = takesPart(odd, bodies[oddBody].maxStretch);
    constexpr uint32_t kStride = (1u << kRowStrideBits) - 1;
    const uint32_t nearOdd = even.z >> kRowStrideBits & 0xffu, farOdd = even.z >> (kRowStrideBits + 8) & 0xffu;
    uint4 cell = make_uint4(even.x, body, even.z & kStride, even.w);
    uint32_t ids[8];
    cornerNodes(cell, ids);
    ready();
    V p[8];
    float w[8];
    if (solve) {
#pragma unroll
        for (int c = 0; c < 8; c++) {
            copyAsync16(&before[0][c][t], prevState + ids[c]);
            const float4 P = pos[ids[c]];
            p[c] = xyz(P);
            w[c] = P.w;
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (solveOdd) {
        uint32_t at[8];
        cornerNodes(make_uint4(odd.x, 0, odd.z & kStride, odd.w), at);
#pragma unroll
        for (int c = 0; c < 8; c++) {
            copyAsync16(&stage[c][t], pos + at[c]);
            copyAsync16(&before[1][c][t], prevState + at[c]);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // the even cells' copies have landed
    // One copy of the projection's code for both cells: two would not stay in
    // the instruction cache.
#pragma unroll 1
    for (uint32_t second = 0; second < 2; second++) {
        if (second) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();  // every copy has landed
            if (solve) {
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const uint32_t holder = c & 1 ? farOdd : nearOdd;
                    const float4 P = withW(p[c], w[c]);
                    // the odd cell's face on the other side of the plane
                    if (holder != kNoRowCell)
                        stage[c ^ 1][holder] = P;
                    else
                        pos[ids[c]] = P;
                }
            }
            __syncthreads();
            solve = solveOdd;
            cell.x = odd.x;
            // The even cell's body and strides serve but at a few cells: the
            // next body's first ones, a group's unpaired ones.
            if (solve && (oddBody != body || !(even.y & kRowCell))) {
                body = oddBody;
                k = cellConsts(bodies + body);
                const uint4 again = group[kRowBlock + t];
                cell = make_uint4(again.x, body, again.z, again.w);
            }
            cornerNodes(cell, ids);
            if (solve) {
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const float4 P = stage[c][t];
                    p[c] = xyz(P);
                    w[c] = P.w;
                }
            }
        }
        if (!solve) continue;
        // The previous positions stay in shared memory, read where they are
        // used: 24 registers fewer, which is a block more an SM.
        auto prev = [&](int c) { return sharedXyz(&before[second][c][t]); };
        if (project && !projectCellInRange(p, prev, w, k)) {
            if (second) {
#pragma unroll
                for (int c = 0; c < 8; c++) pos[ids[c]] = stage[c][t];
            }
            projectCellAgain(cell, bodies + body, pos, prevState);
#pragma unroll
            for (int c = 0; c < 8; c++) p[c] = xyz(pos[ids[c]]);
        }
        if (limit && k.maxStretch > 1.0f) limitStretch(p, w, k, lens);
    }
    solved();
    if (!solve) return;
#pragma unroll
    for (int c = 0; c < 8; c++) pos[ids[c]] = withW(p[c], w[c]);
}

}  // namespace vsim
