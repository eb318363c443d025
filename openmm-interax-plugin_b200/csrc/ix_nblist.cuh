// Device neighbor list of the fused pair pass: a deterministic cell sort of the particles into blocks of 32, block
// bounding boxes, and per i-block lists of "tiles" (one i-block x 32 candidate j particles within cutoff + skin of the
// i-block's box).  Each tile carries its pair masks: bit j of row i is set when the pair (i, j) can interact before
// the next rebuild (within cutoff + skin at build time, not excluded, j after i, some term gated on), and the
// transposed column masks; the pair kernel visits only those pairs and needs no per-step candidate test.
//
// Every kernel of the build reads the rebuild flag and returns at once when it is clear, so the whole pipeline is
// launched every step (and captured in a CUDA graph) without a host round trip.  The build is five kernels (six
// without periodic boundaries), each as much as can be done before the next grid-wide dependency, with the scans in
// the last block of the kernel that feeds them.  As a chain of fifteen kernels in the body of a conditional graph node
// a step without a rebuild paid 9.5 us for the node (28 us where its other branch held the position refresh), and a
// step with one waited 49 us for the body's first kernel and 115 us for the build (24,000 atoms); the five launches take
// 10 us when they return at once (4.4 us for 648 atoms, whose kernels let their successors in early) and 71 us when they
// build.
//
// The reference gets its list from OpenMM (NonbondedUtilities, called at platforms/common/src/
// CommonInteraxKernels.cpp:209) and, on the Reference platform, a voxel hash (ReferenceInteraxPairIxn.h:86-87).
// Any list containing every pair within the cutoff gives the same interacting set once the kernel applies the exact
// r < cutoff test, which it does.
#pragma once

#include "ix_common.cuh"

namespace ix {

constexpr float kPairSkin = IX_TUNE_PAIR_SKIN;   // nm; rebuild when a particle has moved by more than half of it

// Particle flags in the sorted parameter arrays.
constexpr int kFlagReal = 1 << 3;
constexpr int kFlagGateDisp = 1 << 4;    // alpha != 0
constexpr int kFlagGateExch = 1 << 5;    // exchange width != 0
constexpr int kFlagGateSr = 1 << 6;      // short-range width != 0
constexpr int kFlagGates = kFlagGateDisp | kFlagGateExch | kFlagGateSr;

// Frame shared by the build and evaluation kernels.
struct ListGeometry {
    int periodic;          // CutoffPeriodic
    int useCutoff;         // not NoCutoff
    Box box;
    BoxF boxf;
    float listCutoff;      // cutoff + skin (ignored without cutoff)
    int nc[3];             // cell grid
    float invCell[3];      // cells per unit of fractional coordinate (periodic) or per nm (non-periodic)
};

struct ListBuffers {
    int n, nb, np;
    // rebuild control: flag[0] rebuild, flag[1] tile overflow, flag[2..3] unused
    int* flag;
    // original-order input positions and the positions at the last build
    const double* pos;
    double* refPos;
    float* bboxMinMax;          // non-periodic bounding box of all particles (6 floats, as ordered ints)
    // cell sort
    int* cellKey;               // n
    int* cellCount;             // numCells
    int* cellStart;             // numCells + 1
    int* cellArrival;           // n: place among its cell's particles, in the order the atomics took them
    int* order;                 // n: particles in cell order (within a cell in order of arrival)
    unsigned* ticket;           // blocks done, of the kernels whose last block scans (wraps to 0)
    const int* cellRank;        // dense cell index -> rank along the Hilbert curve
    int numCells;
    // sorted particles
    int* sortedAtom;            // np: original index, -1 for padding
    int* slotOf;                // n
    double* shift;              // np x 3: build frame = position - shift
    double* spos;               // np x 3: current position in the build frame
    float4* sposf;              // np
    float4* bbox;               // nb x 2: center (xyz), half extent (xyz)
    // tiles
    int* blockAtoms;            // nb: candidate j particles of each i-block
    int* blockEntries;          // nb: candidate blocks of each i-block
    int4* entries;              // nb x entryCap: (block J, mask of its candidate particles, candidates before them)
    int entryCap;
    int markStride;             // a row of `entries` holds 4 x entryCap marks, one for each kMarkBlocks x markStride blocks
    int* blockTiles;            // nb + 1: exclusive scan of the tile counts, then the total
    int* tileJ;                 // tileCap x 32
    int* tileIBlock;            // tileCap
    int* bucketCount;           // kTileBuckets: tiles by their number of candidate pairs, while the masks are made
    int* bucketTiles;           // kTileBuckets x tileCap: the tiles of each bucket (a batch: all in one, in order)
    int* bucketEnd;             // 32: the end of each bucket, the fullest tiles' first, in the pair kernel's sequence of tasks
                                // (null: no buckets; a small system's kernel takes the tiles as they are)
    unsigned* bucketOffset;     // 32: where a bucket's tasks find their tiles: bucketTiles[bucketOffset + task]
    unsigned* tileMask;         // tileCap x 64: row masks (per i lane, bit = j slot), then column masks (per j lane)
    int* numTiles;              // tiles to evaluate (0 after an overflow)
    int* taskCounter;           // next tile of the pair kernel's dynamic schedule (zeroed before each launch)
    int tileCap;
    const int* flags;           // sorted particle flags (the term gates of each particle)
    // exclusions (original indices), CSR with sorted partners and their range
    const int* exclStart;
    const int* exclList;
    const int2* exclRange;
};

__device__ __forceinline__ bool rebuildRequested(const ListBuffers& L) { return *(volatile int*)L.flag != 0; }

// The pair kernel takes the tiles by decreasing number of candidate pairs, so that the last tiles its warps take are
// short: 32 pairs to a bucket up to 320, where the tiles of a liquid lie (64 to a bucket cost 0.9 us of 105 for 24,000
// atoms), then 64 and 128.  The mask kernel appends each tile to its bucket and its last block sums the counts up; the
// order within a bucket follows the atomics and varies from build to build, which changes no result: forces are summed in
// fixed point and energies go to each tile's own slot.
constexpr int kTileBuckets = 16;
__device__ __forceinline__ int tileBucket(unsigned pairs) {
    if (pairs < 320) return (int)(pairs >> 5);
    return pairs < 512 ? 5 + (int)(pairs >> 6) : min(9 + (int)(pairs >> 7), kTileBuckets - 1);
}

// Current positions in the build frame, and whether any particle moved more than half the skin since the last build,
// which sets the rebuild flag (then, and where it is set already, the build writes the positions itself).  Padding
// slots copy the last real particle's position, which keeps the blocks' boxes tight; they never interact.
__global__ void kRefreshPositions(ListBuffers L, float maxMove2) {
    dependentStart(L.nb <= kEarlyBlocks);
    if (rebuildRequested(L)) return;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    bool moved = false;
    if (s < L.np) {
        const int src = s < L.n ? s : L.n - 1;
        const int i = L.sortedAtom[src];
        const double p[3] = {L.pos[3 * i], L.pos[3 * i + 1], L.pos[3 * i + 2]};
        const double x = p[0] - L.shift[3 * src], y = p[1] - L.shift[3 * src + 1], z = p[2] - L.shift[3 * src + 2];
        L.spos[3 * s] = x;
        L.spos[3 * s + 1] = y;
        L.spos[3 * s + 2] = z;
        L.sposf[s] = make_float4((float)x, (float)y, (float)z, 0.0f);
        const double dx = p[0] - L.refPos[3 * i], dy = p[1] - L.refPos[3 * i + 1], dz = p[2] - L.refPos[3 * i + 2];
        moved = (float)(dx * dx + dy * dy + dz * dz) > maxMove2;
    }
    if (__any_sync(0xffffffffu, moved) && (threadIdx.x & 31) == 0) atomicOr(L.flag, 1);
}

// Float as an order-preserving int, so that min/max reductions can use integer atomics.
__device__ __forceinline__ int floatToOrdered(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float orderedToFloat(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// Whether this block is the last of the grid to get here (all threads call it); the others' writes are then visible.
__device__ __forceinline__ bool lastBlock(unsigned* ticket) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

// Exclusive prefix of one value per thread over a block of T threads; `total` receives the sum.
template <int T>
__device__ __forceinline__ int blockPrefix(int v, int& total) {
    __shared__ int warpSum[T / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) warpSum[warp] = incl;
    __syncthreads();
    int before = 0;
    total = 0;
    for (int w = 0; w < T / 32; w++) {
        before += w < warp ? warpSum[w] : 0;
        total += warpSum[w];
    }
    __syncthreads();
    return before + incl - v;
}

// Start values of the non-periodic bounding box.
__device__ __forceinline__ void resetBounds(const ListBuffers& L) {
    if (threadIdx.x < 6)
        reinterpret_cast<int*>(L.bboxMinMax)[threadIdx.x] =
            threadIdx.x < 3 ? floatToOrdered(INFINITY) : floatToOrdered(-INFINITY);
}

// Bounding box of all particles (non-periodic cell grids span it).
__global__ void kParticleBounds(ListBuffers L) {
    dependentStart(L.nb <= kEarlyBlocks);
    if (!rebuildRequested(L)) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    float v[6];
    for (int k = 0; k < 3; k++) {
        float x = i < L.n ? (float)L.pos[3 * i + k] : INFINITY;
        v[k] = warpMinF(x);
        float y = i < L.n ? (float)L.pos[3 * i + k] : -INFINITY;
        v[3 + k] = warpMaxF(y);
    }
    if ((threadIdx.x & 31) == 0) {
        int* mm = reinterpret_cast<int*>(L.bboxMinMax);
        for (int k = 0; k < 3; k++) {
            atomicMin(mm + k, floatToOrdered(v[k]));
            atomicMax(mm + 3 + k, floatToOrdered(v[3 + k]));
        }
    }
}

// Wrap a position into the reduced periodic cell (c, then b, then a), returning the shift (position - wrapped).
__device__ __forceinline__ void wrapIntoCell(const double p[3], const Box& box, double w[3], double s[3]) {
    w[0] = p[0];
    w[1] = p[1];
    w[2] = p[2];
    double k = floor(w[2] * box.inv[2]);
    w[0] -= k * box.c[0];
    w[1] -= k * box.c[1];
    w[2] -= k * box.c[2];
    k = floor(w[1] * box.inv[1]);
    w[0] -= k * box.b[0];
    w[1] -= k * box.b[1];
    k = floor(w[0] * box.inv[0]);
    w[0] -= k * box.a[0];
    for (int d = 0; d < 3; d++) s[d] = p[d] - w[d];
}

__device__ __forceinline__ int cellOf(const double w[3], const ListGeometry& G, const float* mm) {
    int c[3];
    if (G.periodic) {
        // fractional coordinates of the reduced cell
        double fz = w[2] * G.box.inv[2];
        double fy = (w[1] - fz * G.box.c[1]) * G.box.inv[1];
        double fx = (w[0] - fz * G.box.c[0] - fy * G.box.b[0]) * G.box.inv[0];
        double f[3] = {fx, fy, fz};
        for (int d = 0; d < 3; d++) c[d] = min(max((int)(f[d] * G.nc[d]), 0), G.nc[d] - 1);
    }
    else {
        for (int d = 0; d < 3; d++) {
            float lo = orderedToFloat(__float_as_int(mm[d])), hi = orderedToFloat(__float_as_int(mm[3 + d]));
            float ext = fmaxf(hi - lo, 1e-3f);
            c[d] = min(max((int)(((float)w[d] - lo) / ext * G.nc[d]), 0), G.nc[d] - 1);
        }
    }
    return (c[2] * G.nc[1] + c[1]) * G.nc[0] + c[0];
}

// Cell of each particle, with its place among the cell's particles in the order of the atomics.  The last block scans
// the counts into the cells' starts, and leaves the counts and the bounds as the next build needs them.
constexpr int kCellThreads = 512;
__global__ void __launch_bounds__(kCellThreads) kCellKeys(ListBuffers L, ListGeometry G) {
    dependentStart(L.nb <= kEarlyBlocks);
    if (!rebuildRequested(L)) return;
    const int t = threadIdx.x, i = blockIdx.x * kCellThreads + t;
    if (i < L.n) {
        double p[3] = {L.pos[3 * i], L.pos[3 * i + 1], L.pos[3 * i + 2]};
        double w[3], s[3];
        if (G.periodic) wrapIntoCell(p, G.box, w, s);
        else {
            for (int d = 0; d < 3; d++) w[d] = p[d];
        }
        const int key = L.cellRank[cellOf(w, G, L.bboxMinMax)];
        L.cellKey[i] = key;
        L.cellArrival[i] = atomicAdd(L.cellCount + key, 1);
    }
    if (!lastBlock(L.ticket)) return;
    // each thread a contiguous share of the cells, read four at a time (the arrays hold a multiple of four cells)
    const int per = ((L.numCells + kCellThreads - 1) / kCellThreads + 3) & ~3;
    const int begin = min(t * per, L.numCells), end = min(begin + per, L.numCells);
    int4* count = reinterpret_cast<int4*>(L.cellCount);
    int4* start = reinterpret_cast<int4*>(L.cellStart);
    int sum = 0;
    for (int c = begin; c < end; c += 4) {
        const int4 v = __ldcg(count + (c >> 2));
        sum += (v.x + v.y) + (v.z + v.w);
    }
    int total;
    int run = blockPrefix<kCellThreads>(sum, total);
    for (int c = begin; c < end; c += 4) {
        const int4 v = __ldcg(count + (c >> 2));
        count[c >> 2] = make_int4(0, 0, 0, 0);
        start[c >> 2] = make_int4(run, run + v.x, run + v.x + v.y, run + v.x + v.y + v.z);
        run += (v.x + v.y) + (v.z + v.w);
    }
    __syncthreads();
    if (t == 0) L.cellStart[L.numCells] = total;
    resetBounds(L);
}

__global__ void kScatterCells(ListBuffers L) {
    dependentStart(L.nb <= kEarlyBlocks);
    if (!rebuildRequested(L)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < L.n) L.order[L.cellStart[L.cellKey[i]] + L.cellArrival[i]] = i;
}

// Per-particle arrays in original order and in sorted order.
struct SortedParams {
    const float4 *p0o, *p1o, *p2o, *p3o;
    const int* flagso;
    float4 *p0, *p1, *p2, *p3;
    int* flags;
};

// Bounding box of a block from the positions of its lanes.
// The center's w is 1 when the block's tiles may place each j particle once, at its minimum image relative to the
// block center, instead of taking the minimum image of every pair: that holds in a rectangular periodic box when
// half of every box length exceeds the block's half extent plus the list cutoff plus the skin (room for the motion
// between rebuilds), since then no interacting pair can need a different image.
__device__ __forceinline__ void blockBounds(const ListBuffers& L, const ListGeometry& G, int block, int lane, float4 p) {
    float lo[3] = {warpMinF(p.x), warpMinF(p.y), warpMinF(p.z)};
    float hi[3] = {warpMaxF(p.x), warpMaxF(p.y), warpMaxF(p.z)};
    if (lane == 0) {
        const float half[3] = {0.5f * (hi[0] - lo[0]), 0.5f * (hi[1] - lo[1]), 0.5f * (hi[2] - lo[2])};
        float shift = 0.0f;
        if (G.periodic && !G.box.triclinic) {
            const float len[3] = {(float)G.box.a[0], (float)G.box.b[1], (float)G.box.c[2]};
            bool ok = true;
            for (int d = 0; d < 3; d++) ok = ok && (half[d] + G.listCutoff + kPairSkin < 0.4999f * len[d]);
            shift = ok ? 1.0f : 0.0f;
        }
        L.bbox[2 * block] = make_float4(0.5f * (lo[0] + hi[0]), 0.5f * (lo[1] + hi[1]), 0.5f * (lo[2] + hi[2]), shift);
        L.bbox[2 * block + 1] = make_float4(half[0], half[1], half[2], 0.0f);
    }
}

// Block bounds from the current positions (batches, whose order never changes).
__global__ void kBlockBounds(ListBuffers L, ListGeometry G) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp < L.nb) blockBounds(L, G, warp, lane, L.sposf[warp * 32 + lane]);
}

// The sorted particles, a warp per block of 32 slots: within each cell the particles by index, so that the order does
// not depend on the atomics (slot k of a cell takes the particle that k others of the cell precede: a cell holds about
// four), the image shift that places each in the build frame, its positions and parameters, and the block's box.
__global__ void __launch_bounds__(256) kSortBlocks(ListBuffers L, ListGeometry G, SortedParams P) {
    dependentStart(L.nb <= kEarlyBlocks);
    if (!rebuildRequested(L)) return;
    const int lane = threadIdx.x & 31;
    const int block = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (block >= L.nb) return;
    const int s = block * 32 + lane, lastLane = min(31, L.n - 1 - block * 32);
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    double x[3] = {0.0, 0.0, 0.0};
    int i = -1;
    if (s < L.n) {
        i = L.order[s];
        const int key = L.cellKey[i], b = L.cellStart[key], e = L.cellStart[key + 1];
        for (int a = b; a < e && e - b > 1; a++) {
            const int v = L.order[a];
            int before = 0;
            for (int c = b; c < e; c++) before += L.order[c] < v;
            if (before == s - b) {
                i = v;
                break;
            }
        }
        L.slotOf[i] = s;
        const double p[3] = {L.pos[3 * i], L.pos[3 * i + 1], L.pos[3 * i + 2]};
        double w[3], sh[3] = {0, 0, 0};
        if (G.periodic) wrapIntoCell(p, G.box, w, sh);
        for (int d = 0; d < 3; d++) {
            L.shift[3 * s + d] = sh[d];
            L.refPos[3 * i + d] = p[d];
            x[d] = p[d] - sh[d];
        }
    }
    L.sortedAtom[s] = i;
    for (int d = 0; d < 3; d++) {
        const double last = __shfl_sync(0xffffffffu, x[d], lastLane);
        if (i < 0) {
            x[d] = last;
            L.shift[3 * s + d] = 0.0;
        }
        L.spos[3 * s + d] = x[d];
    }
    const float4 f = make_float4((float)x[0], (float)x[1], (float)x[2], 0.0f);
    L.sposf[s] = f;
    P.p0[s] = i >= 0 ? P.p0o[i] : zero;
    P.p1[s] = i >= 0 ? P.p1o[i] : zero;
    P.p2[s] = i >= 0 ? P.p2o[i] : zero;
    P.p3[s] = i >= 0 ? P.p3o[i] : zero;
    P.flags[s] = i >= 0 ? P.flagso[i] : 0;
    blockBounds(L, G, block, lane, f);
}

// Squared distance between the boxes of two blocks (rectangular minimum image when periodic); 0 if they overlap.
// Triclinic boxes are not pruned (every block is a candidate); the pair kernel's exact test decides.
__device__ __forceinline__ float boxBoxDist2(float4 ci, float4 ei, float4 cj, float4 ej, const ListGeometry& G) {
    float dx = cj.x - ci.x, dy = cj.y - ci.y, dz = cj.z - ci.z;
    if (G.periodic) {
        if (G.box.triclinic) return 0.0f;
        dx -= G.boxf.a[0] * rintf(dx * G.boxf.inv[0]);
        dy -= G.boxf.b[1] * rintf(dy * G.boxf.inv[1]);
        dz -= G.boxf.c[2] * rintf(dz * G.boxf.inv[2]);
    }
    dx = fmaxf(fabsf(dx) - ei.x - ej.x, 0.0f);
    dy = fmaxf(fabsf(dy) - ei.y - ej.y, 0.0f);
    dz = fmaxf(fabsf(dz) - ei.z - ej.z, 0.0f);
    return dx * dx + dy * dy + dz * dz;
}

__device__ __forceinline__ float pointBoxDist2(float4 p, float4 ci, float4 ei, const ListGeometry& G) {
    return boxBoxDist2(ci, ei, p, make_float4(0, 0, 0, 0), G);
}

// Whether every block pairs with every block after it: without a cutoff, and in a triclinic box, where nothing is pruned.
__device__ __forceinline__ bool everyBlockListed(const ListGeometry& G) {
    return !G.useCutoff || (G.periodic && G.box.triclinic);
}

__device__ __forceinline__ bool isExcluded(const ListBuffers& L, int oi, int oj) {
    int2 range = L.exclRange[oi];
    if (oj < range.x || oj > range.y) return false;
    int lo = L.exclStart[oi], hi = L.exclStart[oi + 1] - 1;
    while (lo <= hi) {
        int mid = (lo + hi) >> 1;
        int v = L.exclList[mid];
        if (v == oj) return true;
        if (v < oj) lo = mid + 1;
        else hi = mid - 1;
    }
    return false;
}

constexpr int kListThreads = 256;
constexpr int kListWarps = kListThreads / 32;
constexpr int kMarkBlocks = 32;        // what a warp of kListBlocks tests at a time

// The candidates of each i-block: the particles of the blocks J >= I whose box is within the list cutoff of block I's box
// and whose own position is within it too, in the order (J, slot).  One thread block per i-block: the blocks are
// examined 256 at a time, each thread testing one block's box; the candidate blocks are compacted in block order and
// the warps take them round robin for the particle tests (neighbors along the curve are neighbors in space, so
// contiguous shares would be uneven: 37 us for 24,000 atoms).  The entries hold what the mask kernel needs to find the
// candidates of a tile; a second pass over the same candidates to write the tiles had taken 15.6 us.  A block with more
// candidate blocks than its row holds keeps marks there instead: the number of its candidates before every kMarkBlocks *
// markStride blocks from its own on, from which the mask kernel searches again.  Where every block is listed
// (everyBlockListed) there is nothing to search.  The last block
// scans the tile counts.  On overflow no tile is scheduled (nothing is written beyond the buffers); the host grows
// them and evaluates again.
__global__ void __launch_bounds__(kListThreads) kListBlocks(ListBuffers L, ListGeometry G) {
    dependentStart(L.nb <= kEarlyBlocks);
    if (!rebuildRequested(L)) return;
    __shared__ int candJ[kListThreads], prefix[kListThreads];
    __shared__ unsigned keep[kListThreads];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float cut2 = G.listCutoff * G.listCutoff;
    for (int I = blockIdx.x; I < L.nb; I += gridDim.x) {
        if (everyBlockListed(G)) {
            if (tid == 0) L.blockAtoms[I] = L.n - 32 * I;
            continue;
        }
        const float4 ci = L.bbox[2 * I], ei = L.bbox[2 * I + 1];
        int atoms = 0, entries = 0;
        // the entries, or, of a block that has more than its row holds, in a second pass the row's marks
        for (int pass = 0; pass < 2; pass++) {
            atoms = entries = 0;
            for (int Jc = I; Jc < L.nb; Jc += kListThreads) {
                // the candidate blocks of this chunk, in block order
                const int J = Jc + tid;
                const bool cand = J < L.nb && boxBoxDist2(ci, ei, L.bbox[2 * J], L.bbox[2 * J + 1], G) < cut2;
                int total;
                const int at = blockPrefix<kListThreads>(cand, total);
                if (cand) candJ[at] = J;
                __syncthreads();
                // the particle tests of the candidate blocks, four blocks' loads in flight
                for (int k0 = warp; k0 < total; k0 += 4 * kListWarps) {
                    float4 p[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) p[u] = L.sposf[32 * candJ[min(k0 + u * kListWarps, total - 1)] + lane];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int k = k0 + u * kListWarps;
                        const bool in = k < total && 32 * candJ[min(k, total - 1)] + lane < L.n &&
                                        pointBoxDist2(p[u], ci, ei, G) < cut2;
                        const unsigned m = __ballot_sync(0xffffffffu, in);
                        if (lane == 0 && k < total) keep[k] = m;
                    }
                }
                __syncthreads();
                // entries (in the upper bits) and candidates of the chunk before each candidate block
                const unsigned m = tid < total ? keep[tid] : 0u;
                int sum;
                const int before = blockPrefix<kListThreads>(__popc(m) + (m ? 1 << 16 : 0), sum);
                if (pass == 0) {
                    const int e = entries + (before >> 16);
                    if (m && e < L.entryCap)
                        L.entries[(size_t)I * L.entryCap + e] = make_int4(candJ[tid], (int)m, atoms + (before & 0xffff), 0);
                }
                else {
                    prefix[tid] = before & 0xffff;
                    __syncthreads();
                    // each warp the 32 blocks it tested first: `at` is their first place among the candidate blocks
                    const int group = (J - I) / kMarkBlocks;
                    if (lane == 0 && J < L.nb && group % L.markStride == 0)
                        reinterpret_cast<int*>(L.entries + (size_t)I * L.entryCap)[group / L.markStride] =
                            atoms + (at < total ? prefix[at] : sum & 0xffff);
                }
                entries += sum >> 16;
                atoms += sum & 0xffff;
                __syncthreads();   // the shared arrays are refilled by the next chunk
            }
            if (entries <= L.entryCap) break;
        }
        if (tid == 0) {
            L.blockAtoms[I] = atoms;
            L.blockEntries[I] = entries;
        }
    }
    if (!lastBlock(L.ticket)) return;
    auto tiles = [&](int c) { return (__ldcg(L.blockAtoms + c) + 31) / 32; };
    const int per = (L.nb + kListThreads - 1) / kListThreads;
    const int begin = min(tid * per, L.nb), end = min(begin + per, L.nb);
    int sum = 0;
    for (int c = begin; c < end; c++) sum += tiles(c);
    int total;
    int run = blockPrefix<kListThreads>(sum, total);
    for (int c = begin; c < end; c++) {
        L.blockTiles[c] = run;
        run += tiles(c);
    }
    if (tid < kTileBuckets) L.bucketCount[tid] = 0;
    if (tid == 0) {
        L.blockTiles[L.nb] = total;
        *L.numTiles = total > L.tileCap ? 0 : total;
        if (total > L.tileCap) atomicOr(L.flag + 1, 1);
    }
}

// The last of the n ascending marks that is at most `value` (the first always is), by a warp.
__device__ __forceinline__ int lastMark(const int* marks, int n, int value, int lane) {
    int lo = 0;
    while (n > 1) {
        const int step = (n + 31) / 32;
        const unsigned below = __ballot_sync(0xffffffffu, lane * step < n && marks[lo + lane * step] <= value);
        const int k = 31 - __clz(below);             // lane 0 always holds
        lo += k * step;
        n = min(step, n - k * step);
    }
    return lo;
}

// The i-block of tile t: the last whose first tile is at or before t and that has tiles (its first tile differs from the
// next block's, and the last of equals is taken).
__device__ __forceinline__ int tileBlock(const ListBuffers& L, int t, int lane) {
    return lastMark(L.blockTiles, L.nb + 1, t, lane);
}

// The candidates first .. first + 31 of i-block I to slots[0..31] (-1 after the last), by one warp: where every block is
// listed, block I + first / 32 as it is; else from the entries, or, where they did not fit, by the search again from the
// last mark before them.  Without the marks each tile searched from block I on, which is cubic in the number of blocks:
// an evaluation with a rebuild of 96,000 atoms took 169 ms in a triclinic box (whose blocks are all listed) and takes
// 10.8, and 15.2 ms with a cutoff of 2.6 nm, of 24,000 atoms 3.2 and 4.0 ms; they take 6.2, 0.83 and 1.7 ms (with rows
// of 384 entries, and so from the marks, 6.6 and 1.84 ms for the long cutoff).
__device__ __forceinline__ void tileCandidates(const ListBuffers& L, const ListGeometry& G, int I, int first, int lane,
                                               int* slots) {
    if (everyBlockListed(G)) {
        const int J = I + first / 32, j = 32 * J + lane;
        // (without a cutoff a distance beyond the range of a float leaves the block out)
        const bool near = boxBoxDist2(L.bbox[2 * I], L.bbox[2 * I + 1], L.bbox[2 * J], L.bbox[2 * J + 1], G) < INFINITY;
        slots[lane] = near && j < L.n ? j : -1;
        __syncwarp();
        return;
    }
    const unsigned lt = laneMaskLt();
    slots[lane] = -1;
    __syncwarp();
    auto take = [&](int J, unsigned m, int at) {      // `at`: the place of the mask's first candidate in the tile
        const int q = at + __popc(m & lt);
        if (((m >> lane) & 1u) && q >= 0 && q < 32) slots[q] = 32 * J + lane;
    };
    const int n = L.blockEntries[I];
    const int4* E = L.entries + (size_t)I * L.entryCap;
    if (n <= L.entryCap) {
        for (int e0 = 0; e0 < n; e0 += 32) {
            const int4 v = e0 + lane < n ? E[e0 + lane] : make_int4(0, 0, INT_MAX, 0);
            const bool after = v.z >= first + 32, mine = !after && v.z + __popc((unsigned)v.y) > first;
            for (unsigned b = __ballot_sync(0xffffffffu, mine); b; b &= b - 1) {
                const int k = __ffs(b) - 1;
                take(__shfl_sync(0xffffffffu, v.x, k), (unsigned)__shfl_sync(0xffffffffu, v.y, k),
                     __shfl_sync(0xffffffffu, v.z, k) - first);
            }
            if (__any_sync(0xffffffffu, after)) break;
        }
    }
    else {
        const float4 ci = L.bbox[2 * I], ei = L.bbox[2 * I + 1];
        const float cut2 = G.listCutoff * G.listCutoff;
        const int* marks = reinterpret_cast<const int*>(E);
        const int between = kMarkBlocks * L.markStride;
        const int k = lastMark(marks, (L.nb - I + between - 1) / between, first, lane);
        int before = marks[k];
        for (int Jc = I + k * between; Jc < L.nb && before < first + 32; Jc += 32) {
            const int J = Jc + lane;
            const bool near = J < L.nb && boxBoxDist2(ci, ei, L.bbox[2 * J], L.bbox[2 * J + 1], G) < cut2;
            for (unsigned todo = __ballot_sync(0xffffffffu, near); todo && before < first + 32;) {
                // four blocks' loads in flight
                int K[4];
                float4 p[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    K[u] = todo ? Jc + __ffs(todo) - 1 : L.nb;
                    todo &= todo - 1;
                    p[u] = L.sposf[32 * min(K[u], L.nb - 1) + lane];
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const unsigned m = __ballot_sync(0xffffffffu, 32 * K[u] + lane < L.n && pointBoxDist2(p[u], ci, ei, G) < cut2);
                    take(K[u], m, before - first);
                    before += __popc(m);
                }
            }
        }
    }
    __syncwarp();
}

// The 32 x 32 bit matrix whose row r is lane r's word, transposed (lane c receives bit r = bit c of lane r's word):
// the off-diagonal blocks of 16, 8, 4, 2 and 1 exchanged between lane pairs.
__device__ __forceinline__ unsigned transposeBits(unsigned x, int lane) {
    const unsigned masks[5] = {0x0000ffffu, 0x00ff00ffu, 0x0f0f0f0fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const int s = 16 >> k;
        const unsigned m = masks[k];
        const unsigned y = __shfl_xor_sync(0xffffffffu, x, s);
        x = (lane & s) ? ((x & ~m) | ((y & ~m) >> s)) : ((x & m) | ((y & m) << s));
    }
    return x;
}

// The tiles, one warp per tile over the whole list (the tiles of an i-block vary in number, so a per-i-block
// distribution would wait on the largest): its i-block and candidate j particles, and its pair masks; lane = the tile's
// j lane, the i particles from shared memory.
// A pair's bit is set when j's slot follows i's (each pair once), both are real particles gated on for a common term,
// the pair is not excluded and its build-time distance (minimum image) is within the list cutoff: then no pair outside
// the masks can come within the cutoff before the displacement check requests the next build.  The tests that do not
// depend on the distance are masks formed once per tile; where the i-block allows it (rectangular box, block small
// against the box), j is placed at its image nearest the block's center once, as in the pair kernel, instead of a
// minimum image per pair.  Exclusions are looked up only for the pairs whose i lies in j's exclusion range.  Row
// masks: lane = i slot, bit k = the tile's j lane k; column masks: the transpose.  The last block lays out the pair
// kernel's sequence of tasks.
__global__ void __launch_bounds__(kListThreads) kTileMasks(ListBuffers L, ListGeometry G) {
    dependentStart(false);
    if (!rebuildRequested(L)) return;
    __shared__ float4 ipos[kListWarps][32];   // xyz and the original index (as its bits)
    __shared__ int slots[kListWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the margin covers the float rounding of the build-time distance
    const float cut2 = G.useCutoff ? G.listCutoff * G.listCutoff * (1.0f + 1e-5f) : INFINITY;
    const int numTiles = *L.numTiles;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < numTiles; t += warps) {
        const int I = tileBlock(L, t, lane);
        tileCandidates(L, G, I, 32 * (t - L.blockTiles[I]), lane, slots[warp]);
        const int sj = slots[warp][lane];
        L.tileJ[32LL * t + lane] = sj;
        if (lane == 0) L.tileIBlock[t] = I;
        const int si = I * 32 + lane;
        const int oi = L.sortedAtom[si];
        const int fi = L.flags[si];
        float4 p = L.sposf[si];
        p.w = __int_as_float(oi);
        __syncwarp();
        ipos[warp][lane] = p;
        __syncwarp();
        const unsigned iReal = __ballot_sync(0xffffffffu, oi >= 0);
        const unsigned gateD = __ballot_sync(0xffffffffu, (fi & kFlagGateDisp) != 0);
        const unsigned gateE = __ballot_sync(0xffffffffu, (fi & kFlagGateExch) != 0);
        const unsigned gateS = __ballot_sync(0xffffffffu, (fi & kFlagGateSr) != 0);
        int oj = -1, fj = 0;
        float4 pj = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        int2 jr = make_int2(1, 0);
        if (sj >= 0) {
            oj = L.sortedAtom[sj];
            fj = L.flags[sj];
            pj = L.sposf[sj];
            if (oj >= 0) jr = L.exclRange[oj];
        }
        unsigned column = 0;
        if (oj >= 0) {
            column = iReal & (((fj & kFlagGateDisp) ? gateD : 0u) | ((fj & kFlagGateExch) ? gateE : 0u) |
                              ((fj & kFlagGateSr) ? gateS : 0u));
            const int d = sj - I * 32;   // the i slots of the block below j's
            column &= d >= 32 ? 0xffffffffu : (d <= 0 ? 0u : (1u << d) - 1u);
        }
        // the pairs within the list cutoff, and those whose i lies in j's exclusion range, which are looked up
        unsigned in = 0, suspect = 0;
        const unsigned span = jr.x <= jr.y ? (unsigned)(jr.y - jr.x) : 0u;
        const int low = jr.x <= jr.y ? jr.x : INT_MIN;          // no index is that low
        const float4 c = L.bbox[2 * I];
        if (G.periodic && c.w == 0.0f && G.useCutoff) {
#pragma unroll 4
            for (int i = 0; i < 32; i++) {
                const float4 q = ipos[warp][i];
                float dx = pj.x - q.x, dy = pj.y - q.y, dz = pj.z - q.z;
                minimumImageF(dx, dy, dz, G.boxf);
                if (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < cut2) in |= 1u << i;
                if ((unsigned)(__float_as_int(q.w) - low) <= span) suspect |= 1u << i;
            }
        }
        else {
            if (G.periodic) {
                pj.x -= G.boxf.a[0] * rintf((pj.x - c.x) * G.boxf.inv[0]);
                pj.y -= G.boxf.b[1] * rintf((pj.y - c.y) * G.boxf.inv[1]);
                pj.z -= G.boxf.c[2] * rintf((pj.z - c.z) * G.boxf.inv[2]);
            }
#pragma unroll
            for (int i = 0; i < 32; i++) {
                const float4 q = ipos[warp][i];
                const float dx = pj.x - q.x, dy = pj.y - q.y, dz = pj.z - q.z;
                if (fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < cut2) in |= 1u << i;
                if ((unsigned)(__float_as_int(q.w) - low) <= span) suspect |= 1u << i;
            }
        }
        if (G.useCutoff) column &= in;
        for (suspect &= column; suspect; suspect &= suspect - 1) {
            const int i = __ffs(suspect) - 1;
            if (isExcluded(L, oj, __float_as_int(ipos[warp][i].w))) column &= ~(1u << i);
        }
        const unsigned row = transposeBits(column, lane);
        L.tileMask[64LL * t + lane] = row;
        L.tileMask[64LL * t + 32 + lane] = column;
        const unsigned pairs = __reduce_add_sync(0xffffffffu, (unsigned)__popc(column));
        if (lane == 0 && L.bucketEnd) {
            const int b = tileBucket(pairs);
            L.bucketTiles[(size_t)b * L.tileCap + atomicAdd(L.bucketCount + b, 1)] = t;
        }
    }
    if (!L.bucketEnd || !lastBlock(L.ticket) || warp != 0) return;
    const int b = kTileBuckets - 1 - lane;
    const int count = b >= 0 ? __ldcg(L.bucketCount + b) : 0;
    int end = count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += v;
    }
    L.bucketEnd[lane] = end;
    if (b >= 0) L.bucketOffset[lane] = (unsigned)b * (unsigned)L.tileCap - (unsigned)(end - count);
}

}  // namespace ix
