// The substep kernels of the solver: prediction, the kinematic drive, the
// 8-colour stable Neo-Hookean projection, body contact and the closing pass.
//
// Node state lives in HBM as three float4 arrays in the reference's dense
// node order (pos, prev, vel; state.wgsl:16-19). pos.w carries the node's
// inverse mass as the solver sees it (the reference's separate nodeInvMass
// buffer, particles.js:206-215), so one 16-byte load brings a node's
// position and weight together; every kernel that writes pos keeps w.
#include "row_pass.cuh"

namespace vsim {

void kuhnTable(float out[54]) {
    for (int t = 0; t < 6; t++)
        for (int col = 0; col < 3; col++)
            for (int row = 0; row < 3; row++) out[t * 9 + col * 3 + row] = float(kKuhn.v[t][col][row]);
}


// ------------------------------------------------------------- kernels --

// predict.wgsl:19-36 over the active nodes; with DRIVE, a driven node then
// takes the drive law (the reference's next pass in the substep).
template <bool DRIVE>
__global__ void predictKernel(const FrameParams* __restrict__ fp, Work work, const uint32_t* __restrict__ active,
                              const uint32_t* __restrict__ activeBody, const uint32_t* __restrict__ bodyActive,
                              DriveTables drive, float4* __restrict__ pos, float4* __restrict__ prev,
                              float4* __restrict__ vel) {
    struct Pre {
        uint32_t n, live;
        int32_t driven;
    };
    auto pre = [&](uint32_t i) {
        const uint32_t n = active[i];
        return Pre{n, bodyActive[activeBody[i]], DRIVE ? drive.drivenOf[n] : -1};
    };
    forEachItemAfterWait(work, pre, [&](uint32_t i, Pre q) {
        if (!q.live) return;
        const float4 P = predictNode(fp, q.n, pos, prev, vel);
        if (DRIVE && q.driven >= 0) applyDrive(fp, drive.offsets, drive.grabs, q.driven, q.n, P, pos, prev, vel);
    });
}

// Marks (or, with row < 0, clears) the driven nodes' rows in drivenOf.
__global__ void markDrivenKernel(const uint32_t* __restrict__ driven, uint32_t n, int32_t* __restrict__ drivenOf,
                                 int clear) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) drivenOf[driven[i]] = clear ? -1 : int32_t(i);
}

// project.wgsl:35-184: one colour pass, one thread per occupied cell.
// `cells` holds (global node of corner 0, body, node stride along y, along z)
// per cell of this colour, so the corner loads wait on one load only.
template <bool LIMIT_ONLY>
__global__ void __launch_bounds__(512) elasticKernel(const uint4* __restrict__ cells, Work work,
                                                     const DevBody* __restrict__ bodies,
                                                     const uint32_t* __restrict__ bodyActive, float4* __restrict__ pos,
                                                     const float4* __restrict__ prevState, StretchLengths lens) {
    struct Pre {
        uint4 entry;
        uint32_t live;
        CellConsts k;
    };
    auto pre = [&](uint32_t slot) {
        const uint4 entry = cells[slot];
        return Pre{entry, bodyActive[entry.y], cellConsts(bodies + entry.y)};
    };
    forEachItemAfterWait(work, pre, [&](uint32_t, const Pre& q) {
        if (!q.live) return;
        if (LIMIT_ONLY && !(q.k.maxStretch > 1.0f)) return;
        solveCellAt<LIMIT_ONLY>(q.entry, bodies + q.entry.y, q.k, pos, prevState, lens);
    });
}

// The colour pass with each cell split over the four lanes of a quad
// (solveCellQuad): four times the threads of elasticKernel, each running
// the spine of the cell's chain and a quarter of its per-corner work. Dense
// passes only (the cell list, not a chunk table); every lane loads the
// cell, lane q stores corners q and q + 4.
__global__ void __launch_bounds__(128) elasticQuadKernel(const uint4* __restrict__ cells, uint32_t count,
                                                         const DevBody* __restrict__ bodies,
                                                         const uint32_t* __restrict__ bodyActive,
                                                         float4* __restrict__ pos,
                                                         const float4* __restrict__ prevState, StretchLengths lens) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t slot = t >> 2, q = t & 3;
    const uint32_t quad = 0xfu << (threadIdx.x & 28u);
    const bool has = slot < count;
    uint4 entry = make_uint4(0, 0, 0, 0);
    uint32_t live = 0;
    CellConsts k{};
    if (has) {
        entry = cells[slot];
        live = bodyActive[entry.y];
        k = cellConsts(bodies + entry.y);
    }
    pdlWait();
    pdlLaunchNext();
    if (!has || !live) return;  // the whole quad: its lanes share the cell
    uint32_t ids[8];
    cornerNodes(entry, ids);
    V p[8], prev[8];
    float w[8];
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const float4 P = pos[ids[c]];
        p[c] = xyz(P);
        w[c] = P.w;
    }
#pragma unroll
    for (int c = 0; c < 8; c++) prev[c] = xyz(prevState[ids[c]]);
    solveCellQuad(p, prev, w, k, lens, q, quad);
#pragma unroll
    for (int c = 0; c < 8; c++)
        if ((c & 3) == int(q)) pos[ids[c]] = withW(p[c], w[c]);
}

// project.wgsl:35-184, two colours a launch: a block per group of runs (see
// kRowBlock), a thread per even cell, then a thread per odd cell (rowGroup). A
// substep has four dependent launches where it had eight. No two blocks share
// a node: the update is in place.
//
// What bounds it: at a pass under a wave of blocks, the chain of one launch
// (~1 us), the loads (~0.6 us) and two cells' arithmetic (1.3 us each, see
// projectTetInRange); past that, FP32 issue and the latency that three blocks
// an SM leave uncovered. Microseconds a colour, eight single passes with the
// IEEE operators -> here: a 16x4x4 bar 3.43 -> 2.18, a 64^3 blob 4.84 -> 2.82,
// 256 boxes (1.3M cells) 18.4 -> 13.7, a 161x150x157 blob and sheet 20.7 ->
// 18.0.
//
// WORK: the projection of scenes in which no body limits its stretch, the
// projection with the limit, or a limit-only sweep. (The limit's code in the
// common pass costs it registers: 256 boxes 13.7 us a colour without, 15.0
// with.) EARLY (many waves) lets the next kernel launch at once, so that its blocks
// fill the SMs this pass's last wave leaves idle, and holds the registers to
// three blocks an SM (batch and large blob with two blocks: 15.6 and 20.4 us;
// with four, which spill: 15.5 and 19.9). Otherwise a block that becomes
// resident beside one in mid-flight holds it up by ~1,500 cycles (3.6 against
// 2.8 us a colour on the 64^3 blob), more than the launch it hides: the next
// kernel may launch once the arithmetic is done.
template <RowWork WORK, bool EARLY>
__global__ void __launch_bounds__(kRowBlock, EARLY ? 3 : 2) elasticRowKernel(const uint4* __restrict__ groups,
                                                                             const DevBody* __restrict__ bodies,
                                                                             const uint32_t* __restrict__ bodyActive,
                                                                             float4* __restrict__ pos,
                                                                             const float4* __restrict__ prevState,
                                                                             StretchLengths lens) {
    __shared__ RowShared shared;
    rowGroup(
        groups + size_t(blockIdx.x) * kRowGroup, bodies, bodyActive, pos, prevState, lens, WORK != RowWork::kLimit,
        WORK != RowWork::kProject, shared,
        [] {
            pdlWait();
            if (EARLY) pdlLaunchNext();
        },
        [] {
            if (!EARLY) pdlLaunchNext();
        });
}

// The row pass over the groups a chunked frame's table lists, blocks taking
// them in turn: a frame of a few sessions is a chain of short launches, and
// this halves the elastic ones. Ten sessions of 5,000 to 40,000 cells: 8.4 us
// for two colours, 6.5 each one by one; a one-frame request of a 5,364-cell
// session 0.46 ms against 0.55.
template <RowWork WORK>
__global__ void __launch_bounds__(kRowBlock, kRowChunksPerSm) elasticRowChunksKernel(
    const uint4* __restrict__ groups, Work work, const DevBody* __restrict__ bodies,
    const uint32_t* __restrict__ bodyActive, float4* __restrict__ pos, const float4* __restrict__ prevState,
    StretchLengths lens) {
    __shared__ RowShared shared;
    const uint2 d = work.table[work.span];
    bool waited = false;
    auto ready = [&] {
        if (waited) return;
        waited = true;
        pdlWait();
        pdlLaunchNext();
    };
    for (uint32_t c = blockIdx.x; c < d.y; c += gridDim.x) {
        if (c != blockIdx.x) __syncthreads();  // the group before is out of shared memory
        rowGroup(groups + size_t(work.table[kSpans + d.x + c].x) * kRowGroup, bodies, bodyActive, pos, prevState, lens,
                 WORK != RowWork::kLimit, WORK != RowWork::kProject, shared, ready, [] {});
    }
    ready();  // a block without a group still follows the kernel before
}

// The colour pass for passes much larger than the GPU: each thread solves
// cells in turn (grid-stride) and copies the next cell's eight positions and
// eight previous positions into its slots of shared memory (cp.async) while
// it solves the current one, so the gathers' latency hides behind the
// arithmetic instead of stalling the warp. Cells of one colour share no
// node, so reading ahead is safe. Same arithmetic as elasticKernel.

__global__ void __launch_bounds__(kStreamBlock, kStreamBlocksPerSm) elasticStreamKernel(const uint4* __restrict__ cells, uint32_t count,
                                                                    const DevBody* __restrict__ bodies,
                                                                    const uint32_t* __restrict__ bodyActive,
                                                                    float4* __restrict__ pos,
                                                                    const float4* __restrict__ prevState,
                                                                    StretchLengths lens) {
    __shared__ float4 stage[16][kStreamBlock];  // [corner] pos, [8 + corner] prev
    const uint32_t t = threadIdx.x;
    const uint32_t stride = gridDim.x * blockDim.x;
    uint32_t slot = blockIdx.x * blockDim.x + t;
    uint4 entry = slot < count ? cells[slot] : make_uint4(0, 0, 0, 0);  // frame constants: before the wait
    pdlWait();
    pdlLaunchNext();
    if (slot >= count) return;
    // Copies cell `e`'s nodes into the stage; `after` (zero, computed from the
    // values just read out of the stage) orders the copies after those reads.
    auto fetch = [&](uint4 e, uint32_t after) {
        const uint32_t nx = e.z, nxy = e.w, n0 = e.x + after;
        const uint32_t ids[8] = {n0,       n0 + 1,       n0 + nx,       n0 + nx + 1,
                                 n0 + nxy, n0 + nxy + 1, n0 + nxy + nx, n0 + nxy + nx + 1};
#pragma unroll
        for (int c = 0; c < 8; c++) {
            copyAsync16(&stage[c][t], pos + ids[c]);
            copyAsync16(&stage[8 + c][t], prevState + ids[c]);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(entry, 0);
    while (true) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        V p[8], prev[8];
        float w[8];
        uint32_t bits = 0;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const float4 P = stage[c][t];
            const float4 Q = stage[8 + c][t];
            p[c] = xyz(P);
            w[c] = P.w;
            prev[c] = xyz(Q);
            // One word of each 16-byte read is enough: a read's registers
            // are written together.
            bits ^= __float_as_uint(P.w) ^ __float_as_uint(Q.x);
        }
        uint32_t zero;
        asm volatile("and.b32 %0, %1, 0;" : "=r"(zero) : "r"(bits));
        const uint4 cur = entry;
        const uint32_t next = slot + stride;
        if (next < count) {
            entry = cells[next];
            fetch(entry, zero);
        }
        if (bodyActive[cur.y]) {
            solveCell<false>(cur, bodies + cur.y, p, prev, w, cellConsts(bodies + cur.y), pos, prevState, lens);
        }
        if (next >= count) break;
        slot = next;
    }
}

// finalize.wgsl:44-74 over the active nodes; the velocity factor
// exp(-damping dt) is the body's, evaluated once on the host.
//
// With CONTACT the pass first does what settle.wgsl:20-36 does for a node
// with a surface record -- apply its averaged contact correction, empty its
// bucket -- so no separate pass runs between contact and the closing pass.
// With PREDICT it continues straight into the next substep's
// predict.wgsl:19-36 from the position and velocity it has just computed,
// which are the values that pass would read back; with DRIVE as well a
// driven node then takes the drive law, that substep's first constraint.
template <bool CONTACT, bool PREDICT, bool DRIVE>
__global__ void finalizeKernel(const FrameParams* __restrict__ fp, Work work, const uint32_t* __restrict__ active,
                               const uint32_t* __restrict__ activeBody, const DevBody* __restrict__ bodies,
                               float4* __restrict__ pos, float4* __restrict__ prevState, float4* __restrict__ vel,
                               const int32_t* __restrict__ nodeRecord, const float4* __restrict__ delta,
                               const uint32_t* __restrict__ key, uint32_t* __restrict__ count,
                               uint32_t* __restrict__ cursor, const uint32_t* __restrict__ bodyActive,
                               DriveTables drive, const __grid_constant__ Crowds crowds) {
    struct Pre {
        uint32_t n, live;
        int32_t record, driven;
        float friction, damp;
    };
    auto pre = [&](uint32_t i) {
        const uint32_t body = activeBody[i];
        const uint32_t n = active[i];
        return Pre{n, bodyActive[body], CONTACT ? nodeRecord[n] : -1, DRIVE ? drive.drivenOf[n] : -1,
                   bodies[body].friction, bodies[body].damp};
    };
    forEachItemAfterWait(work, pre, [&](uint32_t, const Pre& q) {
        if (!q.live) return;
        finalizeNode<CONTACT, PREDICT>(fp, q.n, q.friction, q.damp, q.record, pos, prevState, vel, delta, key, count,
                                       [&](uint32_t n, float4 P) {
                                           if (DRIVE && q.driven >= 0)
                                               applyDrive(fp, drive.offsets, drive.grabs, q.driven, n, P, pos,
                                                          prevState, vel);
                                       });
    });
    // After the wait (inside the loop above): the gather has read it.
    const uint32_t thread = blockIdx.x * blockDim.x + threadIdx.x;
    if (CONTACT && thread == 0) *cursor = 0;
    if (CONTACT && crowds.bucket) {
        constexpr uint32_t kParts = kBucketSlots / 4;
        const uint32_t parts = *crowds.gathered * kParts;
        for (uint32_t i = thread; i < parts; i += gridDim.x * blockDim.x) {
            const uint32_t at = crowds.used[i / kParts];
            const uint4 idle = make_uint4(kIdle, kIdle, kIdle, kIdle);
            reinterpret_cast<uint4*>(crowds.lowest)[size_t(at) * kParts + i % kParts] = idle;
            reinterpret_cast<uint4*>(crowds.ordered)[size_t(at) * kParts + i % kParts] = idle;
            if (i % kParts == 0) crowds.bucket[at] = kIdle;
        }
    }
}

// ------------------------------------------------------------- contact --
//
// The reference bins every surface record into a fixed 32-slot bucket with
// an atomic, then canonicalises each bucket by an insertion sort
// (bin.wgsl, sort.wgsl). Here the grid is a counting sort: per-bucket
// counts with the arrival rank of each record, one contiguous segment
// allocated per occupied bucket, a scatter, and an ascending sort of each
// segment's first 32 entries -- the same visible set, in the same order, with
// work proportional to the surface rather than to the grid.

__global__ void binKernel(const FrameParams* __restrict__ fp, Work work, const uint4* __restrict__ surf,
                          const DevBody* __restrict__ bodies, const uint32_t* __restrict__ bodyActive,
                          const float4* __restrict__ pos, uint32_t* __restrict__ key, uint32_t* __restrict__ rank,
                          uint32_t* __restrict__ count) {
    struct Pre {
        uint4 rec;
        uint32_t live;
    };
    auto pre = [&](uint32_t r) {
        const uint4 rec = surf[r];
        return Pre{rec, bodyActive[rec.y]};
    };
    forEachItemAfterWait(work, pre, [&](uint32_t r, const Pre& q) {
        const uint4 rec = q.rec;
        if (!q.live) {
            key[r] = kIdle;
            rank[r] = kIdle;
            return;
        }
        binRecord(r, rec, bodies, pos, key, rank, count);
    });
}

// Each bucket's first-arriving record reserves the bucket's segment; one
// atomic per block on the shared cursor.
__global__ void allocKernel(const FrameParams* __restrict__ fp, Work work, const uint32_t* __restrict__ key,
                            const uint32_t* __restrict__ rank, const uint32_t* __restrict__ count,
                            uint32_t* __restrict__ start, uint32_t* __restrict__ cursor) {
    pdlWait();
    pdlLaunchNext();
    __shared__ uint32_t warpSum[32];
    __shared__ uint32_t blockBase;
    forEachItemUniform(work, [&](bool has, uint32_t r) {
        const bool first = has && rank[r] == 0;
        const uint32_t b = first ? key[r] : 0;
        const uint32_t need = first ? count[b] : 0;
        // Block-wide exclusive prefix of `need`.
        const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        uint32_t incl = need;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= uint32_t(d)) incl += v;
        }
        if (lane == 31) warpSum[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const uint32_t nw = blockDim.x >> 5;
            uint32_t v = lane < nw ? warpSum[lane] : 0;
            uint32_t scan = v;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, scan, d);
                if (lane >= uint32_t(d)) scan += u;
            }
            if (lane < nw) warpSum[lane] = scan - v;
            if (lane == nw - 1) blockBase = scan > 0 ? atomicAdd(cursor, scan) : 0;
        }
        __syncthreads();
        if (first) start[b] = blockBase + warpSum[warp] + (incl - need);
        __syncthreads();  // warpSum and blockBase are rewritten by the next chunk
    });
}

__global__ void scatterKernel(const FrameParams* __restrict__ fp, Work work, const uint32_t* __restrict__ key,
                              const uint32_t* __restrict__ rank, const uint32_t* __restrict__ start,
                              uint32_t* __restrict__ entries) {
    pdlWait();
    pdlLaunchNext();
    forEachItem(work, [&](uint32_t r) {
        if (key[r] == kIdle) return;
        entries[start[key[r]] + rank[r]] = r;
    });
}

// sort.wgsl:14-53: the bucket's visible entries -- its kBucketSlots lowest
// record indices -- in ascending order at the front of its segment, the
// rest after them; every entry's record, position, motion over the substep
// (position - its substep start, as collide.wgsl:100-101 subtracts them)
// with its body's friction, record index and bucket copied out in that
// order, so the gather reads each neighbour bucket's visible entries as one
// contiguous run and both a record's own data and a candidate's one load
// deep.
//
// Each record finds its own place, how many of the bucket's records have a
// lower index, and copies itself there, all records at once.
__global__ void canonKernel(const FrameParams* __restrict__ fp, Work work, const uint32_t* __restrict__ key,
                            const uint32_t* __restrict__ rank, const uint32_t* __restrict__ start,
                            const uint32_t* __restrict__ count, const uint32_t* __restrict__ entries,
                            const uint4* __restrict__ surf, const float4* __restrict__ pos,
                            const float4* __restrict__ prevState, const DevBody* __restrict__ bodies,
                            uint4* __restrict__ sMeta, float4* __restrict__ sPos, float4* __restrict__ sMoved,
                            uint32_t* __restrict__ sRec, uint32_t* __restrict__ sKey) {
    pdlWait();
    pdlLaunchNext();
    const ContactArrays arrays{bodies, surf, key, rank, start, count, nullptr, nullptr, nullptr, nullptr, nullptr,
                               nullptr};
    const SortedEntries out{sMeta, sPos, sMoved, sRec, sKey};
    forEachItem(work, [&](uint32_t r) {
        if (key[r] == kIdle) return;
        canonRecord<true>(r, arrays, entries, out, pos, prevState);
    });
}

// collide.wgsl:16-125, reading each neighbour bucket's visible entries as
// the contiguous run canonKernel laid out. With EMIT, every counted hit
// (r, other) is also appended to `pairs` (capacity-checked), for the
// pair-set checks.
//
// Records are taken in bucket order (the counting sort's output as canonKernel
// copied it, `*cursor` long), so neighbouring records read the same runs.
// Two mappings
// of records to threads, chosen per launch from the number of records:
//
// - few records (below `warpModeBelow`): one warp per record. The record's
//   candidates -- the visible entries of its 27 neighbour buckets,
//   concatenated in the reference's order (buckets dz, dy, dx; entries in
//   bucket order) -- are dealt to the lanes 32 at a time: lane q < 27 sizes
//   neighbour bucket q, a warp scan turns the sizes into offsets, and each
//   lane finds its candidate's run as the last one starting at or before it
//   (a ballot of the runs starting in the round, the run carried over from
//   the round before). The record's chain of
//   dependent candidate loads is spread over 32 lanes, which is what a
//   launch too small to fill the GPU needs;
// - many records: one thread per record, scanning the runs itself, which
//   costs fewer instructions per record once the GPU is full anyway.
//
// Either way each record's hits are added to its sum one at a time in
// candidate order, so both give the sequential result.

template <bool EMIT>
__global__ void __launch_bounds__(kCollideBlock, 5) collideKernel(
    const FrameParams* __restrict__ fp, uint32_t items, uint32_t warpModeBelow, const uint32_t* __restrict__ cursor,
    const DevBody* __restrict__ bodies, const uint32_t* __restrict__ start, const uint32_t* __restrict__ count,
    const uint4* __restrict__ sMeta, const float4* __restrict__ sPos, const float4* __restrict__ sMoved,
    const uint32_t* __restrict__ sRec, const uint32_t* __restrict__ sKey, float4* __restrict__ delta,
    uint32_t* __restrict__ pairs, uint32_t capacity, unsigned long long* __restrict__ pairCount) {
    pdlWait();
    pdlLaunchNext();
    const uint32_t total = min(items, *cursor);
    const uint32_t selfContact = fp->selfContact;
    const uint32_t thread = blockIdx.x * blockDim.x + threadIdx.x;
    const ContactArrays arrays{bodies, nullptr, nullptr, nullptr, start, count, sMeta, sPos, sMoved, sRec, sKey, delta};
    auto emit = [&](uint32_t r, uint32_t at) {
        const unsigned long long slot = atomicAdd(pairCount, 1ull);
        if (slot < capacity) {
            pairs[2 * slot] = r;
            pairs[2 * slot + 1] = sRec[at];
        }
    };
    if (total >= warpModeBelow) {
        for (uint32_t i = thread; i < total; i += gridDim.x * blockDim.x)
            collideThread<EMIT>(i, arrays, selfContact, emit);
        return;
    }
    // Per warp: the neighbour bucket (lane) whose run starts at each
    // candidate position of the current round.
    __shared__ uint32_t runAt[kCollideBlock / 32][32];
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t i = thread >> 5; i < total; i += warps)
        collideWarp<EMIT>(i, arrays, selfContact, runAt[threadIdx.x >> 5], emit);
}

// ------------------------------------------- contact in two launches --
//
// The chain above takes five dependent launches, of which segments, scatter
// and order only lay the buckets out. A bucket rarely holds more than a few
// records (edge h, about one surface node each at rest), so here bin stores a
// record straight into its bucket: the first kSlots arrivals in the bucket's
// own slots, later ones in a list threaded through the records. The gather
// reads the buckets around a record as bin left them and orders each one's
// few entries itself, as sort.wgsl:14-53 would: ascending, the 32 lowest.
// Two launches against five: the 64^3 blob's frame (49k records) 569 -> 465
// us, a six-body pile's (8.9k) 322 -> 285 us, a 161x150x157 scene's (352k) 9.10
// -> 8.66 ms.
//
// Nothing is reset but the counts (by the closing pass): slots past a
// bucket's count and the list past its overflow are never read.
//
// A bucket that more than 32 records reach (bodies dragged past the tank's
// faces share its outermost buckets, a scene that has gone NaN its first one)
// is a crowd: later arrivals leave the list alone and put themselves among the
// crowd's 32 lowest, found in a hash table by their bucket. Each of its words
// takes the lower of itself and what comes and passes the other on to the next
// (atomicMin), which leaves the lowest in ascending order whatever the order of
// arrival; a record above the last of them, as nearly all of thousands are,
// looks once and leaves. So a crowd of n costs about n looks, and the gather
// reads at most 64 of it. The closing pass empties the crowds of the substep.
//
// The bodies share one grid of at most kSlotBuckets buckets, so a record's
// bucket and which faces of the grid it lies on fit one word.

// Where bucket b's crowd is looked for first.
__device__ __forceinline__ uint32_t crowdAt(uint32_t b, const Crowds& crowds) {
    return (b * 0x9e3779b1u >> 7) & crowds.mask;
}

// Record r among the 32 lowest of bucket b's crowd. The table has more places
// than there can be crowds, so the search ends.
__device__ __noinline__ void joinCrowd(uint32_t r, uint32_t b, const Crowds& crowds) {
    uint32_t at = crowdAt(b, crowds);
    for (uint32_t probe = 0; probe <= crowds.mask; probe++, at = (at + 1) & crowds.mask) {
        uint32_t holder = __ldcg(crowds.bucket + at);
        if (holder == kIdle) {
            holder = atomicCAS(crowds.bucket + at, kIdle, b);
            if (holder == kIdle) {
                crowds.used[atomicAdd(crowds.count, 1u)] = at;
                holder = b;
            }
        }
        if (holder == b) break;
    }
    uint32_t* lowest = crowds.lowest + size_t(at) * kBucketSlots;
    // The words only fall: one below the record now stays below it.
    if (__ldcg(lowest + kBucketSlots - 1) < r) return;
    for (uint32_t i = 0; i < kBucketSlots && r != kIdle; i++)
        if (__ldcg(lowest + i) > r) r = max(atomicMin(lowest + i, r), r);
}

__global__ void binSlotsKernel(Work work, const uint4* __restrict__ surf, const DevBody* __restrict__ bodies,
                               const uint32_t* __restrict__ bodyActive, const float4* __restrict__ pos,
                               uint32_t* __restrict__ key, uint32_t* __restrict__ place, uint32_t* __restrict__ count,
                               uint32_t* __restrict__ slots, uint32_t* __restrict__ over, uint32_t* __restrict__ next,
                               float4* __restrict__ recPos, const __grid_constant__ Crowds crowds) {
    struct Pre {
        uint4 rec;
        uint32_t live;
    };
    auto pre = [&](uint32_t r) {
        const uint4 rec = surf[r];
        return Pre{rec, bodyActive[rec.y]};
    };
    forEachItemAfterWait(work, pre, [&](uint32_t r, const Pre& q) {
        if (!q.live) {
            key[r] = kIdle;
            place[r] = kIdle;
            return;
        }
        const float4 P = pos[q.rec.x];
        const DevBody* grid = bodies + q.rec.y;
        int coord[3];
        const uint32_t b = bucketOf(grid, xyz(P), coord);
        const uint32_t rank = atomicAdd(&count[b], 1u);
        uint32_t faces = 0;
#pragma unroll
        for (int a = 0; a < 3; a++)
            faces |= (coord[a] == 0 ? 1u : 0u) << (2 * a) | (coord[a] + 1 == int(grid->gridDims[a]) ? 2u : 0u) << (2 * a);
        key[r] = b;
        place[r] = b | faces * kSlotBuckets;
        recPos[r] = P;
        if (rank < kSlots)
            slots[kSlots * size_t(b) + rank] = r;
        else if (rank < kBucketSlots)
            next[r] = atomicExch(&over[b], r);
        else
            joinCrowd(r, b, crowds);
    });
}

constexpr uint32_t kSlotsBlock = 128;   // threads of a gather block
constexpr uint32_t kGatherLanes = 9;    // lanes a record: one per row of three buckets along x
constexpr uint32_t kGatherRecords = 3;  // records a warp
constexpr uint32_t kGatherList = 96;    // candidates of a record its lanes go through together
static_assert(kGatherRecords * kGatherList == 9 * kBucketSlots, "a warp's lists hold what nine buckets show");

// collide.wgsl:16-125 for record r by a whole warp (every lane calls it with the
// same r): a record with more candidates than its own list holds, or next to a
// crowd. Lane q < 27 lays the early records of neighbour bucket q into `list`
// (the warp's three lists together; `owner` names the bucket of each), and the
// warp merges each crowd's lowest with them, unless another has left them in
// order. The lanes look at the candidates as they come, 32 at a time; only those
// in reach are then put in order, each ranked against its bucket's others, and
// corrected for. Where the 27 buckets show more than the list holds they are
// gone through nine by nine. Returns the corrections' sum and the number of
// hits, added in candidate order.
//
// Instructions and the walk along a bucket's list bound it (3,100 a record when
// every candidate was put in order, 2,000 here, as the longer chain's warp takes
// on buckets ordered before). Contact of a frame of ten substeps, microseconds,
// longer chain by a warp a record and here: 64^3 blob (51k records) squeezed to
// 0.45, 0.3 and 0.12: 708, 1273, 3350 and 751, 1525, 4821; past a tank's corner
// 3877 and 2912 (24k records 2238 and 2252), gone NaN 7722 and 3803.
__device__ __forceinline__ float4 collideFull(uint32_t r, uint32_t selfContact, uint32_t rowStride, uint32_t planeStride,
                                              const uint4* surf, const DevBody* bodies, const uint32_t* place,
                                              const uint32_t* count, const uint4* slots, const uint32_t* over,
                                              const uint32_t* next, const float4* recPos, const float4* prevState,
                                              const Crowds& crowds, uint32_t* list, uint8_t* owner) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t home = place[r], faces = home / kSlotBuckets;
    const uint32_t dx = lane % 3, dy = lane / 3 % 3, dz = lane / 9;  // offsets + 1
    const uint32_t outside = (dx == 0 ? 1u : dx == 2 ? 2u : 0u) | (dy == 0 ? 4u : dy == 2 ? 8u : 0u) |
                             (dz == 0 ? 16u : dz == 2 ? 32u : 0u);
    const uint32_t b = (home & (kSlotBuckets - 1)) + (dx - 1) + (dy - 1) * rowStride + (dz - 1) * planeStride;
    const uint32_t n = lane < 27 && !(faces & outside) ? count[b] : 0;
    const uint32_t held = min(n, kBucketSlots);
    uint32_t end = held;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(kAll, end, d);
        if (lane >= d) end += v;
    }
    const uint32_t total = __shfl_sync(kAll, end, 31);
    const uint32_t each = total <= 9 * kBucketSlots ? 27 : 9;  // buckets at a time
    uint32_t crowd = 0;                                        // the bucket's, where it has one
    if (n > kBucketSlots) {
        crowd = crowdAt(b, crowds);
        for (uint32_t probe = 0; probe < crowds.mask && crowds.bucket[crowd] != b; probe++)
            crowd = (crowd + 1) & crowds.mask;
    }
    Contactor c;
    c.me = surf[r];
    c.node = c.me.x;
    c.radius = __uint_as_float(c.me.w);
    const float4 P = recPos[r];
    c.pi = xyz(P);
    c.wi = P.w;
    V sum = mk(0.0f, 0.0f, 0.0f);
    float hits = 0.0f;
#pragma unroll 1
    for (uint32_t first = 0; first < 27; first += each) {
        const uint32_t before = first ? __shfl_sync(kAll, end, first - 1) : 0u;
        const uint32_t candidates = __shfl_sync(kAll, end, first + each - 1) - before;
        const bool mine = lane >= first && lane < first + each && held > 0;
        const uint32_t at = end - held - before;  // of the lane's bucket in the list
        __syncwarp();                             // the list's readers are done with it
        // The crowds that some warp has ordered before (a word of theirs is idle
        // or final, so a whole row speaks for itself).
        uint32_t unordered = 0;
        uint32_t some = __ballot_sync(kAll, mine && n > kBucketSlots);
        const uint32_t* ordered = crowds.ordered + lane;
        uint32_t ahead = kIdle;
        if (some) ahead = __ldcg(ordered + size_t(__shfl_sync(kAll, crowd, __ffs(some) - 1)) * kBucketSlots);
        while (some) {
            const uint32_t q = __ffs(some) - 1, row = ahead;
            some &= some - 1;
            if (some) ahead = __ldcg(ordered + size_t(__shfl_sync(kAll, crowd, __ffs(some) - 1)) * kBucketSlots);
            const uint32_t base = __shfl_sync(kAll, at, q);
            if (__any_sync(kAll, row == kIdle)) {
                unordered |= 1u << q;
            } else {
                list[base + lane] = row;
                owner[base + lane] = uint8_t(q);
            }
        }
        if (mine && (n <= kBucketSlots || (unordered >> lane & 1))) {
            const uint4 s = slots[b];
            list[at] = s.x;
            if (held > 1) list[at + 1] = s.y;
            if (held > 2) list[at + 2] = s.z;
            if (held > 3) list[at + 3] = s.w;
            uint32_t e = held > kSlots ? over[b] : 0;
            for (uint32_t i = kSlots; i < held; i++) {
                list[at + i] = e;
                if (i + 1 < held) e = next[e];
            }
            for (uint32_t i = 0; i < held; i++) owner[at + i] = uint8_t(lane);
        }
        __syncwarp();
        // The others: the lowest of their early records, put in order, and of the
        // rest, which ascend. The lower of the one from below and the other from
        // above are the lowest of both, falling and rising once: five exchanges
        // order them.
        for (; unordered; unordered &= unordered - 1) {
            const uint32_t q = __ffs(unordered) - 1, base = __shfl_sync(kAll, at, q);
            const size_t row = size_t(__shfl_sync(kAll, crowd, q)) * kBucketSlots + lane;
            uint32_t e = list[base + lane];
            const uint32_t late = crowds.lowest[row];
            auto exchange = [&](uint32_t distance, bool up) {
                const uint32_t other = __shfl_xor_sync(kAll, e, distance);
                e = up == ((lane & distance) == 0) ? min(e, other) : max(e, other);
            };
#pragma unroll
            for (uint32_t size = 2; size <= 32; size *= 2)
#pragma unroll
                for (uint32_t distance = size / 2; distance > 0; distance /= 2)
                    exchange(distance, (lane & size) == 0 || size == 32);
            e = min(late, __shfl_sync(kAll, e, 31 - lane));
#pragma unroll
            for (uint32_t distance = 16; distance > 0; distance /= 2) exchange(distance, true);
            list[base + lane] = e;
            __stcg(crowds.ordered + row, e);
        }
        __syncwarp();
        // The records in reach, moved to the list's front as they are found.
        uint32_t found = 0;
        for (uint32_t from = 0; from < candidates; from += 32) {
            bool hit = false;
            uint32_t e = 0, of = 0;
            if (from + lane < candidates) {
                e = list[from + lane];
                of = owner[from + lane];
                float dist2;
                hit = contactHit(c, surf[e], recPos[e], selfContact, dist2);
            }
            const uint32_t bits = __ballot_sync(kAll, hit);
            if (hit) {
                const uint32_t to = found + __popc(bits & ((1u << lane) - 1u));
                list[to] = e;
                owner[to] = uint8_t(of);
            }
            found += __popc(bits);
        }
        __syncwarp();
        // As many whole buckets' at a time as 32 lanes hold, one a lane.
        for (uint32_t from = 0; from < found;) {
            uint32_t here = min(32u, found - from);
            uint32_t e = lane < here ? list[from + lane] : 0;
            const uint32_t of = lane < here ? owner[from + lane] : 0xffu;
            const uint32_t left = __shfl_up_sync(kAll, of, 1);
            // bit l: a bucket's start at lane l
            uint32_t starts = __ballot_sync(kAll, lane < here && (lane == 0 || of != left));
            if (from + here < found && owner[from + here] == __shfl_sync(kAll, of, 31)) {
                here = 31 - __clz(starts);  // the last goes on
                starts &= (1u << here) - 1u;
            }
            const uint32_t upTo = starts & (0xffffffffu >> (31 - lane)), above = starts & ~(0xffffffffu >> (31 - lane));
            const uint32_t run = 31 - __clz(upTo | 1u);  // where the lane's bucket starts, and how many it has
            const uint32_t holds = lane < here ? (above ? __ffs(above) - 1 : here) - run : 0;
            const uint32_t most = __reduce_max_sync(kAll, holds);
            if (most > 1) {
                uint32_t rank = 0;
                for (uint32_t j = 0; j < most; j++) {
                    const uint32_t other = __shfl_sync(kAll, e, run + j);
                    rank += j < holds && other < e ? 1u : 0u;
                }
                if (lane < here) list[from + run + rank] = e;
                __syncwarp();
                if (lane < here) e = list[from + lane];
            }
            V correction = mk(0.0f, 0.0f, 0.0f);
            if (lane < here) {
                const uint4 them = surf[e];
                const float4 Q = recPos[e];
                const V d = c.pi - xyz(Q);
                c.movedI = c.pi - xyz(prevState[c.node]);
                c.frictionI = bodies[c.me.y].friction;
                const V moved = xyz(Q) - xyz(prevState[them.x]);
                correction = contactCorrection(c, them, Q, withW(moved, bodies[them.y].friction), dot(d, d));
            }
            for (uint32_t at = 0; at < here; at++) {
                const V add = mk(__shfl_sync(kAll, correction.x, at), __shfl_sync(kAll, correction.y, at),
                                 __shfl_sync(kAll, correction.z, at));
                sum = sum + add;
                hits = hits + 1.0f;
            }
            from += here;
        }
    }
    return withW(sum, hits);
}

// collide.wgsl:16-125 for every live record. Nine lanes share a record, three
// records a warp: a lane sizes and orders the three buckets of its row
// (dy, dz), the entries go into one list in the reference's candidate order
// (dz, dy, dx, then ascending), and the lanes take the list eighteen at a
// time; hits are added in list order. Against a warp a record this is 190
// warp instructions a record instead of 430, and everything a candidate
// needs but its record index is one load deep: bin left each record's
// position by record. Bound by the latency of its four dependent loads (own
// record, buckets, candidates, a hit's motion) at half issue: 128 threads
// and 64 registers, eight blocks an SM, measured best (the 64^3 blob's frame
// 465 us; with ten blocks, which spill, 484).
//
// A record with more than kGatherList candidates, or next to a crowd, is gone
// through by its whole warp after that (collideFull).
__global__ void __launch_bounds__(kSlotsBlock, 8) collideSlotsKernel(
    const FrameParams* __restrict__ fp, uint32_t records, uint32_t rowStride, uint32_t planeStride,
    const uint4* __restrict__ surf, const DevBody* __restrict__ bodies, const uint32_t* __restrict__ place,
    const uint32_t* __restrict__ count, const uint4* __restrict__ slots, const uint32_t* __restrict__ over,
    const uint32_t* __restrict__ next, const float4* __restrict__ recPos, const float4* __restrict__ prevState,
    const __grid_constant__ Crowds crowds, float4* __restrict__ delta) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr uint32_t kGroup = (1u << kGatherLanes) - 1u;
    __shared__ uint32_t lists[kSlotsBlock / 32][kGatherRecords][kGatherList];
    __shared__ uint8_t owners[kSlotsBlock / 32][kGatherRecords * kGatherList];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t group = lane / kGatherLanes, q = lane - group * kGatherLanes;
    const uint32_t r = (blockIdx.x * (kSlotsBlock / 32) + warp) * kGatherRecords + group;
    const bool valid = group < kGatherRecords && r < records;
    Contactor c;
    c.me = valid ? surf[r] : make_uint4(0, 0, 0, 0);
    c.node = c.me.x;
    c.radius = __uint_as_float(c.me.w);
    const uint32_t selfContact = fp->selfContact;
    pdlWait();
    const uint32_t home = valid ? place[r] : kIdle;
    const bool live = home != kIdle;
    const float4 P = live ? recPos[r] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    c.pi = xyz(P);
    c.wi = P.w;
    // Whether row `row` (dy + 3 dz, offsets + 1) of the record's buckets is in
    // the grid, and its middle bucket; whether its bucket d (dx + 1) is.
    auto rowOf = [&](uint32_t row, uint32_t& middle) {
        const uint32_t dy = row % 3, dz = row / 3, faces = home / kSlotBuckets;
        middle = (home & (kSlotBuckets - 1)) + (dy - 1) * rowStride + (dz - 1) * planeStride;
        return !((dy == 0 && faces & 4u) || (dy == 2 && faces & 8u) || (dz == 0 && faces & 16u) ||
                 (dz == 2 && faces & 32u));
    };
    auto inRow = [&](uint32_t d) { return !((d == 0 && home & kSlotBuckets) || (d == 2 && home & (2 * kSlotBuckets))); };
    uint32_t held[3] = {0, 0, 0}, middle = 0;
    uint4 entry[3] = {};
    if (live && rowOf(q, middle)) {
#pragma unroll
        for (uint32_t d = 0; d < 3; d++) {
            if (!inRow(d)) continue;
            held[d] = count[middle + d - 1];
            entry[d] = slots[middle + d - 1];  // read with the count: past it, left over and unused
        }
    }
    // Where the lane's entries go in the record's list.
    const uint32_t mine = held[0] + held[1] + held[2];
    uint32_t end = mine;
#pragma unroll
    for (uint32_t d = 1; d < kGatherLanes; d <<= 1) {
        const uint32_t v = __shfl_up_sync(kAll, end, d);
        if (q >= d) end += v;
    }
    const uint32_t groupAt = group * kGatherLanes;
    const uint32_t total = __shfl_sync(kAll, end, min(groupAt + kGatherLanes - 1, 31u));
    const uint32_t crowded = __ballot_sync(kAll, max(held[0], max(held[1], held[2])) > kBucketSlots);
    const bool listed = live && total <= kGatherList && (crowded >> groupAt & kGroup) == 0;
    uint32_t* list = lists[warp][min(group, kGatherRecords - 1)];
    if (listed) {
        uint32_t at = end - mine;
#pragma unroll
        for (uint32_t d = 0; d < 3; d++) {
            const uint32_t n = held[d];
            // The slots' records in ascending order, left-overs last.
            uint32_t e0 = n > 0 ? entry[d].x : kIdle, e1 = n > 1 ? entry[d].y : kIdle;
            uint32_t e2 = n > 2 ? entry[d].z : kIdle, e3 = n > 3 ? entry[d].w : kIdle;
            auto ascend = [](uint32_t& a, uint32_t& b) {
                const uint32_t low = min(a, b);
                b = max(a, b);
                a = low;
            };
            ascend(e0, e1);
            ascend(e2, e3);
            ascend(e0, e2);
            ascend(e1, e3);
            ascend(e1, e2);
            if (n > 0) list[at] = e0;
            if (n > 1) list[at + 1] = e1;
            if (n > 2) list[at + 2] = e2;
            if (n > 3) list[at + 3] = e3;
            uint32_t more = 0;
            for (uint32_t i = kSlots; i < n; i++) {  // the few past the slots, by insertion
                more = i == kSlots ? over[middle + d - 1] : next[more];
                uint32_t to = at + i;
                while (to > at && list[to - 1] > more) {
                    list[to] = list[to - 1];
                    to--;
                }
                list[to] = more;
            }
            at += n;
        }
    }
    __syncwarp();
    V sum = mk(0.0f, 0.0f, 0.0f);
    float hits = 0.0f;
    // The correction of a hit.
    auto correct = [&](uint4 them, float4 Q, float dist2) {
        c.movedI = c.pi - xyz(prevState[c.node]);
        c.frictionI = bodies[c.me.y].friction;
        const V moved = xyz(Q) - xyz(prevState[them.x]);
        return contactCorrection(c, them, Q, withW(moved, bodies[them.y].friction), dist2);
    };
    const uint32_t longest = __reduce_max_sync(kAll, listed ? total : 0u);
    for (uint32_t round = 0; round < longest; round += 2 * kGatherLanes) {
        // Two candidates a lane, nine apart, their records loaded together.
        uint4 them[2];
        float4 Q[2];
        bool has[2];
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            const uint32_t j = round + h * kGatherLanes + q;
            has[h] = listed && j < total;
            if (has[h]) {
                const uint32_t other = list[j];
                them[h] = surf[other];
                Q[h] = recPos[other];
            }
        }
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            float dist2 = 0.0f;
            const bool hit = has[h] && contactHit(c, them[h], Q[h], selfContact, dist2);
            uint32_t bits = __ballot_sync(kAll, hit);
            if (bits == 0) continue;
            V correction = mk(0.0f, 0.0f, 0.0f);
            if (hit) correction = correct(them[h], Q[h], dist2);
            bits = group < kGatherRecords ? bits >> groupAt & kGroup : 0u;
            while (__any_sync(kAll, bits != 0)) {
                const uint32_t from = bits ? groupAt + __ffs(bits) - 1 : lane;
                const V add = mk(__shfl_sync(kAll, correction.x, from), __shfl_sync(kAll, correction.y, from),
                                 __shfl_sync(kAll, correction.z, from));
                if (!bits) continue;
                sum = sum + add;
                hits = hits + 1.0f;
                bits &= bits - 1;
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *crowds.gathered = *crowds.count;
        *crowds.count = 0;
    }
    if (listed && q == 0) delta[r] = withW(sum, hits);
    for (uint32_t full = __ballot_sync(kAll, live && !listed && q == 0); full; full &= full - 1) {
        const uint32_t at = __shfl_sync(kAll, r, __ffs(full) - 1);
        const float4 d = collideFull(at, selfContact, rowStride, planeStride, surf, bodies, place, count, slots, over,
                                     next, recPos, prevState, crowds, reinterpret_cast<uint32_t*>(&lists[warp]), owners[warp]);
        if (lane == 0) delta[at] = d;
    }
    pdlLaunchNext();
}

// settle.wgsl:20-36 (gain 1, bodyContact.js:48), then empties the buckets
// this substep used and the segment cursor, restoring the empty grid.
__global__ void settleKernel(const FrameParams* __restrict__ fp, Work work, const uint4* __restrict__ surf,
                             const uint32_t* __restrict__ key, const float4* __restrict__ delta,
                             float4* __restrict__ pos, uint32_t* __restrict__ count, uint32_t* __restrict__ cursor,
                             int apply) {
    pdlWait();
    pdlLaunchNext();
    if (blockIdx.x == 0 && threadIdx.x == 0) *cursor = 0;
    forEachItem(work, [&](uint32_t r) {
        if (apply) {
            const float4 d = delta[r];
            if (d.w > 0.0f) {
                const uint32_t node = surf[r].x;
                const float4 P = pos[node];
                const V step = xyz(d) * (1.0f / d.w);
                pos[node] = withW(xyz(P) + step, P.w);
            }
        }
        if (key[r] != kIdle) count[key[r]] = 0;
    });
}

// The gather's work on the current grid, for measurement: per live record,
// its 27 neighbour buckets' visible entries (min(count, kBucketSlots) each,
// what collideKernel reads), summed into out[1]; live records into out[0],
// occupied buckets (their first-arriving records) into out[2]. Runs between
// the gather and the pass that empties the grid.
__global__ void censusKernel(Work work, const uint4* __restrict__ surf, const DevBody* __restrict__ bodies,
                             const uint32_t* __restrict__ key, const uint32_t* __restrict__ rank,
                             const uint32_t* __restrict__ count, unsigned long long* __restrict__ out) {
    forEachItem(work, [&](uint32_t r) {
        const uint32_t b = key[r];
        if (b == kIdle) return;
        const DevBody* g = bodies + surf[r].y;
        const uint32_t linear = b - g->gridBase;
        const uint32_t z = divBy(linear, g->divXY);
        const uint32_t rest = linear - z * (g->gridDims[0] * g->gridDims[1]);
        const uint32_t y = divBy(rest, g->divX);
        const int c[3] = {int(rest - y * g->gridDims[0]), int(y), int(z)};
        unsigned long long seen = 0;
        for (int q = 0; q < 27; q++) {
            const int x = c[0] + q % 3 - 1, yy = c[1] + (q / 3) % 3 - 1, zz = c[2] + q / 9 - 1;
            if (x < 0 || yy < 0 || zz < 0 || x >= int(g->gridDims[0]) || yy >= int(g->gridDims[1]) ||
                zz >= int(g->gridDims[2]))
                continue;
            const uint32_t n = count[g->gridBase + uint32_t(x) + g->gridDims[0] * (uint32_t(yy) + g->gridDims[1] * uint32_t(zz))];
            seen += n < kBucketSlots ? n : kBucketSlots;
        }
        atomicAdd(&out[0], 1ull);
        atomicAdd(&out[1], seen);
        if (rank[r] == 0) atomicAdd(&out[2], 1ull);
    });
}

// ------------------------------------------------------- node utilities --

// pos.w := base[n] for a list of nodes (restoring a released hold).
__global__ void restoreWKernel(const uint32_t* __restrict__ nodes, uint32_t n, const float* __restrict__ base,
                               float4* __restrict__ pos) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) pos[nodes[i]].w = base[nodes[i]];
}

// pos.w := 0 for a list of nodes (a hard hold prescribes them).
__global__ void zeroWKernel(const uint32_t* __restrict__ nodes, uint32_t n, float4* __restrict__ pos) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) pos[nodes[i]].w = 0.0f;
}

// pos.w := base[n] for a node range (after a density change).
__global__ void refreshWKernel(uint32_t first, uint32_t n, const float* __restrict__ base, float4* __restrict__ pos) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) pos[first + i].w = base[first + i];
}

// pos.xyz := in.xyz keeping w (writing a state from the host).
__global__ void mergeXyzKernel(const float4* __restrict__ in, uint32_t n, float4* __restrict__ pos) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const float4 a = in[i];
        pos[i] = make_float4(a.x, a.y, a.z, pos[i].w);
    }
}

// out := (in.xyz, 0): a state read out (positions cross the ABI with w 0).
__global__ void dropWKernel(const float4* __restrict__ in, uint32_t n, float4* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const float4 a = in[i];
        out[i] = make_float4(a.x, a.y, a.z, 0.0f);
    }
}

// ------------------------------------------------------------ launchers --

namespace {
template <class... KArgs, class... Args>
cudaError_t launch(const LaunchCtx& ctx, void (*kernel)(KArgs...), uint32_t grid, uint32_t block, Args... args) {
    if (grid == 0) return cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = ctx.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx.pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

inline uint32_t blocks(uint32_t n, uint32_t b) { return (n + b - 1) / b; }
}  // namespace

Span denseSpan(uint32_t count, uint32_t block) { return Span{Work{nullptr, 0, count}, blocks(count, block), block}; }

// A colour pass of a small scene has too few cells to put a block of the
// configured size on every SM; smaller blocks spread it over all of them
// (at the headline body's 15,800 cells a pass, blocks of 32 measured faster
// in the frame than blocks of 64: 4.97 against 5.15 us a pass).
Span elasticSpan(uint32_t count, uint32_t block, uint32_t sms) {
    while (block > 32 && blocks(count, block) < 2 * sms) block /= 2;
    return denseSpan(count, block);
}

namespace {
DriveTables driveTables(const DeviceState& s) {
    return DriveTables{s.drivenOf, s.drivenOffset, s.grabs};
}
}  // namespace

cudaError_t launchPredict(const LaunchCtx& c, const DeviceState& s, const Span& n, bool drive) {
    auto go = [&](auto kernel) {
        return launch(c, kernel, n.grid, n.block, s.fp, n.work, s.active, s.activeBody,
                      (const uint32_t*)s.bodyActive, driveTables(s), s.pos, s.prev, s.vel);
    };
    return drive ? go(predictKernel<true>) : go(predictKernel<false>);
}

cudaError_t launchMarkDriven(cudaStream_t st, const uint32_t* driven, uint32_t n, int32_t* drivenOf, bool clear) {
    if (n == 0) return cudaSuccess;
    markDrivenKernel<<<blocks(n, 256), 256, 0, st>>>(driven, n, drivenOf, clear ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launchElastic(const LaunchCtx& c, const DeviceState& s, const uint4* cells, const Span& sp,
                          bool limitOnly, const StretchLengths& lens) {
    if (c.quadCells && !limitOnly && !sp.work.table && !streamsColourPass(sp.work.count, c.sms))
        return launch(c, elasticQuadKernel, blocks(4 * sp.work.count, 128), 128, cells, sp.work.count, s.bodies,
                      (const uint32_t*)s.bodyActive, s.pos, (const float4*)s.prev, lens);
    if (!limitOnly && !sp.work.table && streamsColourPass(sp.work.count, c.sms))
        return launch(c, elasticStreamKernel, std::min(blocks(sp.work.count, kStreamBlock), kStreamBlocksPerSm * c.sms),
                      kStreamBlock,
                      cells, sp.work.count, s.bodies, (const uint32_t*)s.bodyActive, s.pos, (const float4*)s.prev,
                      lens);
    if (limitOnly)
        return launch(c, elasticKernel<true>, sp.grid, sp.block, cells, sp.work, s.bodies,
                      (const uint32_t*)s.bodyActive, s.pos, (const float4*)s.prev, lens);
    return launch(c, elasticKernel<false>, sp.grid, sp.block, cells, sp.work, s.bodies,
                  (const uint32_t*)s.bodyActive, s.pos, (const float4*)s.prev, lens);
}

cudaError_t launchElasticRows(const LaunchCtx& c, const DeviceState& s, const uint4* groups, uint32_t count,
                              RowWork work, const StretchLengths& lens) {
    auto go = [&](auto kernel) {
        return launch(c, kernel, count, kRowBlock, groups, (const DevBody*)s.bodies, (const uint32_t*)s.bodyActive,
                      s.pos, (const float4*)s.prev, lens);
    };
    // One block an SM or fewer: a single wave, whose launch of the next kernel
    // waits for its arithmetic.
    const bool early = count > c.sms;
    switch (work) {
        case RowWork::kProject:
            return early ? go(elasticRowKernel<RowWork::kProject, true>) : go(elasticRowKernel<RowWork::kProject, false>);
        case RowWork::kBoth:
            return early ? go(elasticRowKernel<RowWork::kBoth, true>) : go(elasticRowKernel<RowWork::kBoth, false>);
        default:
            return early ? go(elasticRowKernel<RowWork::kLimit, true>) : go(elasticRowKernel<RowWork::kLimit, false>);
    }
}

cudaError_t launchElasticRowChunks(const LaunchCtx& c, const DeviceState& s, const Span& span, RowWork work,
                                   const StretchLengths& lens) {
    auto go = [&](auto kernel) {
        return launch(c, kernel, span.grid, span.block, (const uint4*)s.rows, span.work, (const DevBody*)s.bodies,
                      (const uint32_t*)s.bodyActive, s.pos, (const float4*)s.prev, lens);
    };
    return work == RowWork::kProject ? go(elasticRowChunksKernel<RowWork::kProject>)
           : work == RowWork::kBoth  ? go(elasticRowChunksKernel<RowWork::kBoth>)
                                     : go(elasticRowChunksKernel<RowWork::kLimit>);
}

cudaError_t launchFinalize(const LaunchCtx& c, const DeviceState& s, const Span& n, bool contact, bool predictNext,
                           bool drive) {
    auto go = [&](auto kernel) {
        return launch(c, kernel, n.grid, n.block, s.fp, n.work, s.active, s.activeBody, s.bodies, s.pos, s.prev,
                      s.vel, (const int32_t*)s.nodeRecord, (const float4*)s.delta, (const uint32_t*)s.key, s.count,
                      s.cursor, (const uint32_t*)s.bodyActive, driveTables(s), s.crowds);
    };
    if (predictNext && drive)
        return contact ? go(finalizeKernel<true, true, true>) : go(finalizeKernel<false, true, true>);
    if (contact) return predictNext ? go(finalizeKernel<true, true, false>) : go(finalizeKernel<true, false, false>);
    return predictNext ? go(finalizeKernel<false, true, false>) : go(finalizeKernel<false, false, false>);
}

// Solve mode leaves the corrections in `delta` for the closing pass, which
// applies them and empties the grid; Pairs mode lists the hits and empties
// the grid itself.
cudaError_t launchContact(const LaunchCtx& c, const DeviceState& s, const Span& r, uint32_t recordItems,
                          int mapping, ContactMode mode, uint32_t* pairs, uint32_t capacity,
                          unsigned long long* pairCount, cudaEvent_t* marks) {
    const uint32_t g = r.grid, b = r.block;
    const Work w = r.work;
    cudaError_t e;
    auto mark = [&](int i) { return marks ? cudaEventRecord(marks[i], c.stream) : cudaSuccess; };
    if ((e = mark(0))) return e;
    if ((e = launch(c, binKernel, g, b, s.fp, w, s.surf, (const DevBody*)s.bodies, (const uint32_t*)s.bodyActive,
                    (const float4*)s.pos, s.key, s.rank, s.count)))
        return e;
    if ((e = mark(1))) return e;
    if ((e = launch(c, allocKernel, g, b, s.fp, w, (const uint32_t*)s.key, (const uint32_t*)s.rank,
                    (const uint32_t*)s.count, s.start, s.cursor)))
        return e;
    if ((e = mark(2))) return e;
    if ((e = launch(c, scatterKernel, g, b, s.fp, w, (const uint32_t*)s.key, (const uint32_t*)s.rank,
                    (const uint32_t*)s.start, s.entries)))
        return e;
    if ((e = mark(3))) return e;
    if ((e = launch(c, canonKernel, g, b, s.fp, w, (const uint32_t*)s.key, (const uint32_t*)s.rank,
                    (const uint32_t*)s.start, (const uint32_t*)s.count, (const uint32_t*)s.entries, (const uint4*)s.surf,
                    (const float4*)s.pos, (const float4*)s.prev, (const DevBody*)s.bodies, s.sMeta, s.sPos,
                    s.sMoved, s.sRec, s.sKey)))
        return e;
    if ((e = mark(4))) return e;
    // The gather runs over the bucket-ordered entries (at most recordItems),
    // a warp each while fewer than 2048 per SM, else a thread each. Over one
    // body (a dense span) one resident wave of blocks (five an SM at its
    // launch bounds) loops over the records: on the headline body 32.8
    // against 34.8 us for a block per eight records. Over many isolated
    // bodies (a chunked span: settled sessions whose records' candidate
    // counts vary widely) the span says: up to a block per eight records
    // (64 an SM) keeps the SMs balanced on large frames -- the looping wave
    // cut the serving pool's saturation by 7 % -- and 16 an SM suits small
    // ones (a one-session tick 0.62 against 0.68 ms).
    const uint32_t cg = std::min(blocks(recordItems, 8), (r.work.table ? r.gatherPerSm : 5u) * c.sms);
    const uint32_t warpModeBelow = mapping == VSIM_GATHER_WARP     ? 0xffffffffu
                                   : mapping == VSIM_GATHER_THREAD ? 0u
                                                                   : 2048 * c.sms;
    auto collide = [&](auto kernel, uint32_t* out, uint32_t cap, unsigned long long* n) {
        return launch(c, kernel, cg, kCollideBlock, s.fp, recordItems, warpModeBelow, (const uint32_t*)s.cursor,
                      (const DevBody*)s.bodies, (const uint32_t*)s.start, (const uint32_t*)s.count,
                      (const uint4*)s.sMeta, (const float4*)s.sPos, (const float4*)s.sMoved,
                      (const uint32_t*)s.sRec, (const uint32_t*)s.sKey, s.delta, out, cap, n);
    };
    if (mode == ContactMode::Pairs) {
        if ((e = collide(collideKernel<true>, pairs, capacity, pairCount))) return e;
        if ((e = mark(5))) return e;
        return launch(c, settleKernel, g, b, s.fp, w, s.surf, (const uint32_t*)s.key, (const float4*)s.delta, s.pos,
                      s.count, s.cursor, 0);
    }
    if ((e = collide(collideKernel<false>, (uint32_t*)nullptr, 0u, (unsigned long long*)nullptr))) return e;
    return mark(5);
}

cudaError_t launchContactSlots(const LaunchCtx& c, const DeviceState& s, const Span& r, uint32_t rowStride,
                               uint32_t planeStride) {
    cudaError_t e;
    if ((e = launch(c, binSlotsKernel, r.grid, r.block, r.work, s.surf, (const DevBody*)s.bodies,
                    (const uint32_t*)s.bodyActive, (const float4*)s.pos, s.key, s.rank, s.count,
                    reinterpret_cast<uint32_t*>(s.slots), s.over, s.next, s.recPos, s.crowds)))
        return e;
    return launch(c, collideSlotsKernel, blocks(r.work.count, kGatherRecords * (kSlotsBlock / 32)), kSlotsBlock, s.fp,
                  r.work.count, rowStride, planeStride, s.surf, (const DevBody*)s.bodies, (const uint32_t*)s.rank,
                  (const uint32_t*)s.count, (const uint4*)s.slots, (const uint32_t*)s.over, (const uint32_t*)s.next,
                  (const float4*)s.recPos, (const float4*)s.prev, s.crowds, s.delta);
}

cudaError_t launchCensus(const LaunchCtx& c, const DeviceState& s, const Span& r, unsigned long long* out) {
    cudaError_t e_;
    if ((e_ = launch(c, censusKernel, r.grid, r.block, r.work, (const uint4*)s.surf, (const DevBody*)s.bodies,
                     (const uint32_t*)s.key, (const uint32_t*)s.rank, (const uint32_t*)s.count, out)))
        return e_;
    // empty the grid without applying the corrections
    return launch(c, settleKernel, r.grid, r.block, s.fp, r.work, s.surf, (const uint32_t*)s.key,
                  (const float4*)s.delta, s.pos, s.count, s.cursor, 0);
}

cudaError_t launchRestoreW(cudaStream_t st, const uint32_t* nodes, uint32_t n, const float* base, float4* pos) {
    if (n == 0) return cudaSuccess;
    restoreWKernel<<<blocks(n, 256), 256, 0, st>>>(nodes, n, base, pos);
    return cudaGetLastError();
}

cudaError_t launchZeroW(cudaStream_t st, const uint32_t* nodes, uint32_t n, float4* pos) {
    if (n == 0) return cudaSuccess;
    zeroWKernel<<<blocks(n, 256), 256, 0, st>>>(nodes, n, pos);
    return cudaGetLastError();
}

cudaError_t launchRefreshW(cudaStream_t st, uint32_t first, uint32_t n, const float* base, float4* pos) {
    if (n == 0) return cudaSuccess;
    refreshWKernel<<<blocks(n, 256), 256, 0, st>>>(first, n, base, pos);
    return cudaGetLastError();
}

cudaError_t launchDropW(cudaStream_t st, const float4* in, uint32_t n, float4* out) {
    if (n == 0) return cudaSuccess;
    dropWKernel<<<blocks(n, 256), 256, 0, st>>>(in, n, out);
    return cudaGetLastError();
}

cudaError_t launchMergeXyz(cudaStream_t st, const float4* in, uint32_t n, float4* pos) {
    if (n == 0) return cudaSuccess;
    mergeXyzKernel<<<blocks(n, 256), 256, 0, st>>>(in, n, pos);
    return cudaGetLastError();
}

}  // namespace vsim
