// Axilrod-Teller-Muto three-body kernels (the reference's five-kernel pipeline is
// platforms/common/src/kernels/interaxThreeBody.cc:11-655 with host code CommonInteraxKernels.cpp:386-646; the FP64
// definition is openmmapi/include/internal/InteraxThreeBodyTerms.h:51-146 and
// platforms/reference/src/ReferenceInteraxThreeBodyIxn.cpp:84-135).
//
//   kSiteCentroids       site positions (unweighted centroids, double) and the site rebuild check
//   kSiteNeighbors       (rebuild only) per site A the sites B > A of other molecules within cutoff + skin
//   kTriplesFast         one warp per site A with a short list: the neighbors within the cutoff are staged in shared
//                        memory with their double-precision minimum-image displacements from A (rounded to float);
//                        four lanes take one neighbor C and share the others B among them, so that each triple is
//                        seen once from B and once from C and each visit adds only the force on its own C, in
//                        registers (no stores per triple, no gather, no atomics)
//   kTriplesWide         the same for sites with longer lists, 8 warps per site (chunked beyond kAtmMaxStaged within
//                        the cutoff, so any length); a site whose list overflowed its capacity scans the sites
//                        instead, so an overflow never drops a triple
//   kSpreadSiteForces    the site forces, shared equally among each site's particles, into the particle forces
#pragma once

#include "ix_common.cuh"

namespace ix {

constexpr float kSiteSkin = IX_TUNE_SITE_SKIN;

struct AtmConfig {
    int numSites;
    int periodic;
    Box box;
    BoxF boxf;
    float cutoff2;
    float listCutoff2;
    float scale;                 // scale factor
    float lambda;                // alchemical parameter (1 without alchemical sites)
    int useTangToennies;
    float twoBeta;               // 2 x damping scale
    float invCentroidRadius;     // 0 = no centroid damping
    float maxMove2;
    int zeroSlots, zeroOffset;   // energy slots the centroid kernel clears (those of a wide kernel that may not run)
    int imageBC;                 // the displacement of C from B can need a minimum image of its own
};

// Whether two neighbors of a site can be nearest to each other through another image than the site's: not in a
// rectangular box whose edges exceed three cutoffs, where such an image is farther than the cutoff.
inline int tripleNeedsImages(const AtmConfig& C, double cutoff) {
    return C.periodic && (C.box.triclinic || !(C.box.a[0] > 3.001 * cutoff && C.box.b[1] > 3.001 * cutoff &&
                                               C.box.c[2] > 3.001 * cutoff));
}

// Cell grid of the site-list search in a rectangular periodic box whose edges hold at least three cells as wide as
// the list cutoff: every site within the list cutoff of a site lies in its cell or the 26 around it.
struct SiteCells {
    int nc[3];                   // cells per axis; nc[0] = 0: no grid (the chunk scan is used)
    float cellsPerNm[3];
    int* cellStart;              // numCells + 1
    int* cellSites;              // the sites by cell, each cell's in increasing order
    int* siteCell;               // numSites
    float4* wrapped;             // numSites: each site's position wrapped into the box (float), w its molecule (int
                                 // bits), written by the cell sort for the list search
    unsigned* order;             // numSites: the x coordinate as a 32-bit fraction of the box, at the last build
};

// The owner of a triple is the site that comes first; site `b` comes after site `a` (both within the list cutoff of
// each other).  By index, the lists of the sites next to the periodic boundary hold all their neighbors where the
// others hold half (in the 96,000-atom box with a 0.8 nm cutoff those long lists took the wide kernel 179 of the 421 us
// of both).  Where the cell grid serves (edges of at least three list cutoffs) the order is that of the x displacement,
// which gives every site half of its neighbors: the difference of the 32-bit box fractions wraps as the minimum image
// does, and as no two of three mutual neighbors are a third of the box apart it orders them without a cycle.
__device__ __forceinline__ bool siteAfter(const SiteCells& G, int byIndex, int a, int b) {
    const int d = byIndex ? 0 : (int)(G.order[b] - G.order[a]);
    return d > 0 || (d == 0 && b > a);
}
constexpr int kSiteCellMax = 8192;   // cells the one-block sort holds in shared memory
// sites up to this count are scattered and ordered in dynamic shared memory by the one-block sort (160 KB)
constexpr int kSiteSortSharedMax = 40000;

struct AtmBuffers {
    const int* siteOffsets;      // numSites + 1
    const int* siteParticles;
    const float4* siteParams;    // alpha, frequency, width, alchemical (0/1)
    const int* molecule;         // effective molecule (negative input already replaced by -1 - site)
    double* sitePos;             // numSites x 3
    double* siteRef;             // numSites x 3, at the last list build
    float4* chunkBox;            // 2 per chunk of 32 consecutive sites: box center (w = 1: usable) and half extents,
                                 // of the positions wrapped into a rectangular box; null: the list search scans all
    int* flag;                   // [0] rebuild, [1] neighbor overflow, [2] a list longer than the fast kernel takes,
                                 // [3] the lists are ordered by index (set by their build, see siteAfter)
    int* nbrCount;               // numSites
    int* nbr;                    // numSites x cap
    int cap;
    long long* siteForce;        // 3 x numSites, SoA fixed point
    long long* particleForce;    // 3 x numParticles, SoA fixed point (original order)
    int numParticles;
    double* energyPartials;      // one per warp of the fast triple kernel's grid, then one per warp of the wide one
    unsigned long long* tripleVisits;   // each interacting triple counts two (it is visited from two of its sites)
    SiteCells cells;
};

// Lists up to kAtmFast take the fast triple kernel, one warp per site: a longer one would hold its warp after the
// others have finished (a cluster's first site has all the others listed).  The cell grid's lists are all of about
// the same length, so there the fast kernel takes what its storage holds.
constexpr int kAtmFast = IX_TUNE_ATM_FAST;
constexpr int kAtmFastStaged = 2 * kAtmFast;
constexpr int kAtmFastWarps = 4;

// The longest list the fast kernel takes, by the order the lists were built in.
__device__ __forceinline__ int fastListMax(const AtmBuffers& A) { return A.flag[3] ? kAtmFast : kAtmFastStaged; }

// A site position as float, wrapped into a rectangular periodic box (unchanged otherwise): the frame of the chunk
// boxes, in which the minimum-image distance between a point and a box bounds that to every point in the box.
__device__ __forceinline__ float3 siteWrapped(const AtmConfig& C, double x, double y, double z) {
    float3 p = make_float3((float)x, (float)y, (float)z);
    if (C.periodic && !C.box.triclinic) {
        p.x -= C.boxf.a[0] * floorf(p.x * C.boxf.inv[0]);
        p.y -= C.boxf.b[1] * floorf(p.y * C.boxf.inv[1]);
        p.z -= C.boxf.c[2] * floorf(p.z * C.boxf.inv[2]);
    }
    return p;
}

// Squared minimum-image distance from a point to a box (0 inside it), both in the wrapped frame.
__device__ __forceinline__ float siteBoxDist2(const AtmConfig& C, float3 p, float4 c, float4 e) {
    float dx = c.x - p.x, dy = c.y - p.y, dz = c.z - p.z;
    if (C.periodic) {
        dx -= C.boxf.a[0] * rintf(dx * C.boxf.inv[0]);
        dy -= C.boxf.b[1] * rintf(dy * C.boxf.inv[1]);
        dz -= C.boxf.c[2] * rintf(dz * C.boxf.inv[2]);
    }
    dx = fmaxf(fabsf(dx) - e.x, 0.0f);
    dy = fmaxf(fabsf(dy) - e.y, 0.0f);
    dz = fmaxf(fabsf(dz) - e.z, 0.0f);
    return dx * dx + dy * dy + dz * dz;
}

__global__ void kSiteCentroids(AtmBuffers A, AtmConfig C, const double* pos) {
    dependentStart(C.numSites <= kEarlySites);
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    for (int k = s; k < C.zeroSlots; k += gridDim.x * blockDim.x) A.energyPartials[C.zeroOffset + k] = 0.0;
    bool moved = false;
    float3 w = make_float3(INFINITY, INFINITY, INFINITY), wMax = make_float3(-INFINITY, -INFINITY, -INFINITY);
    if (s < C.numSites) {
        double c[3] = {0.0, 0.0, 0.0};
        const int b = A.siteOffsets[s], e = A.siteOffsets[s + 1];
        for (int k = b; k < e; k++) {
            const int p = A.siteParticles[k];
            c[0] += pos[3 * p];
            c[1] += pos[3 * p + 1];
            c[2] += pos[3 * p + 2];
        }
        const double n = (double)(e - b);
        for (int d = 0; d < 3; d++) {
            c[d] /= n;
            A.sitePos[3 * s + d] = c[d];
            A.siteForce[d * C.numSites + s] = 0;   // the triple kernels of this evaluation accumulate from zero
        }
        const double dx = c[0] - A.siteRef[3 * s], dy = c[1] - A.siteRef[3 * s + 1], dz = c[2] - A.siteRef[3 * s + 2];
        moved = (float)(dx * dx + dy * dy + dz * dz) > C.maxMove2;
        w = siteWrapped(C, c[0], c[1], c[2]);
        wMax = w;
    }
    // a rebuild clears the long-list flag, which the lists set again (the host requests a rebuild by the flag alone)
    if (__any_sync(0xffffffffu, moved) && (threadIdx.x & 31) == 0) {
        atomicOr(A.flag, 1);
        A.flag[2] = 0;
    }
    else if (s == 0 && *(volatile int*)A.flag != 0) A.flag[2] = 0;
    if (A.chunkBox) {
        // the box of this warp's 32 sites (blocks are whole warps, so a warp is one chunk)
        const float lo[3] = {warpMinF(w.x), warpMinF(w.y), warpMinF(w.z)};
        const float hi[3] = {warpMaxF(wMax.x), warpMaxF(wMax.y), warpMaxF(wMax.z)};
        const int chunk = s >> 5;
        if ((threadIdx.x & 31) == 0 && 32 * chunk < C.numSites) {
            // the margin covers the float rounding of the wrapped positions
            const float m = 1e-4f;
            const bool usable = !(C.periodic && C.box.triclinic);
            A.chunkBox[2 * chunk] = make_float4(0.5f * (lo[0] + hi[0]), 0.5f * (lo[1] + hi[1]), 0.5f * (lo[2] + hi[2]),
                                                usable ? 1.0f : 0.0f);
            A.chunkBox[2 * chunk + 1] = make_float4(0.5f * (hi[0] - lo[0]) + m, 0.5f * (hi[1] - lo[1]) + m,
                                                    0.5f * (hi[2] - lo[2]) + m, 0.0f);
        }
    }
}

__device__ __forceinline__ void siteDelta(const AtmBuffers& A, const AtmConfig& C, int from, int to, double d[3]) {
    d[0] = A.sitePos[3 * to] - A.sitePos[3 * from];
    d[1] = A.sitePos[3 * to + 1] - A.sitePos[3 * from + 1];
    d[2] = A.sitePos[3 * to + 2] - A.sitePos[3 * from + 2];
    if (C.periodic) minimumImage(d[0], d[1], d[2], C.box);
}

// One warp per site A scans the sites above it, 32-site chunk by chunk, skipping the chunks whose box is farther
// than the list cutoff from A (when the centroid kernel wrote the chunk boxes).  The list is in increasing site order.
__global__ void kSiteNeighbors(AtmBuffers A, AtmConfig C) {
    dependentStart(C.numSites <= kEarlySites);
    if (*(volatile int*)A.flag == 0) return;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= C.numSites) return;
    const int a = warp;
    const int molA = A.molecule[a];
    const float3 pa = siteWrapped(C, A.sitePos[3 * a], A.sitePos[3 * a + 1], A.sitePos[3 * a + 2]);
    const float skip2 = C.listCutoff2 * (1.0f + 1e-4f);
    int count = 0;
    for (int b0 = (a + 1) & ~31; b0 < C.numSites; b0 += 32) {
        if (A.chunkBox) {
            const float4 c = A.chunkBox[2 * (b0 >> 5)];
            if (c.w != 0.0f && siteBoxDist2(C, pa, c, A.chunkBox[2 * (b0 >> 5) + 1]) >= skip2) continue;
        }
        const int b = b0 + lane;
        bool near = false;
        if (b > a && b < C.numSites && A.molecule[b] != molA) {
            double d[3];
            siteDelta(A, C, a, b, d);
            near = (float)(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]) < C.listCutoff2;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, near);
        if (near) {
            const int k = count + __popc(bal & laneMaskLt());
            if (k < A.cap) A.nbr[(size_t)a * A.cap + k] = b;
        }
        count += __popc(bal);
    }
    if (lane == 0) {
        // the full count: a site whose list overflowed its capacity is found by the wide triple kernel, which then
        // scans every later site instead of reading the list
        A.nbrCount[a] = count;
        if (count > A.cap) atomicOr(A.flag + 1, 1);
        // flag[2]: some site needs the wide triple kernel (cleared with each request of a build)
        if (count > kAtmFast || count > A.cap) atomicOr(A.flag + 2, 1);
        if (a == 0) A.flag[3] = 1;
    }
    for (int d = 0; d < 3; d++)
        if (lane == 0) A.siteRef[3 * a + d] = A.sitePos[3 * a + d];
}

// The sites binned into the cell grid (rebuild only), in one block: each site's cell from its wrapped position, the
// cell counts in shared memory, their scan, the scatter, and each cell's sites put in increasing order (so that the
// lists built from the cells come out the same on every run).  SHARED (at most kSiteSortSharedMax sites, the launch
// giving 4 bytes of dynamic shared memory per site): the scatter goes to shared memory and a warp per cell writes each
// site at its rank among the cell's sites; else each cell is insertion-sorted in place in global memory, which is why that
// form leaves the SM its cache (100,000 sites: 225 us, and 335 with all of the memory set aside for shared memory).
template <bool SHARED>
__global__ void __launch_bounds__(1024) kSiteCellSort(AtmBuffers A, AtmConfig C) {
    dependentStart(C.numSites <= kEarlySites);
    if (*(volatile int*)A.flag == 0) return;
    __shared__ int count[kSiteCellMax];
    __shared__ int threadSum[1024];
    extern __shared__ int scattered[];
    const SiteCells& G = A.cells;
    const int numCells = G.nc[0] * G.nc[1] * G.nc[2];
    const int t = threadIdx.x, T = blockDim.x;
    for (int c = t; c < numCells; c += T) count[c] = 0;
    __syncthreads();
    for (int s = t; s < C.numSites; s += T) {
        const float3 p = siteWrapped(C, A.sitePos[3 * s], A.sitePos[3 * s + 1], A.sitePos[3 * s + 2]);
        const int cx = min(max((int)(p.x * G.cellsPerNm[0]), 0), G.nc[0] - 1);
        const int cy = min(max((int)(p.y * G.cellsPerNm[1]), 0), G.nc[1] - 1);
        const int cz = min(max((int)(p.z * G.cellsPerNm[2]), 0), G.nc[2] - 1);
        const int cell = (cz * G.nc[1] + cy) * G.nc[0] + cx;
        G.siteCell[s] = cell;
        G.wrapped[s] = make_float4(p.x, p.y, p.z, __int_as_float(A.molecule[s]));
        const double f = A.sitePos[3 * s] * C.box.inv[0];
        G.order[s] = (unsigned)(unsigned long long)((f - floor(f)) * 4294967296.0);
        atomicAdd(&count[cell], 1);
    }
    __syncthreads();
    // exclusive scan: each thread a contiguous chunk of cells, then the chunk sums
    const int per = (numCells + T - 1) / T;
    const int c0 = min(t * per, numCells), c1 = min(c0 + per, numCells);
    int sum = 0;
    for (int c = c0; c < c1; c++) sum += count[c];
    threadSum[t] = sum;
    __syncthreads();
    for (int o = 1; o < T; o <<= 1) {
        const int v = t >= o ? threadSum[t - o] : 0;
        __syncthreads();
        threadSum[t] += v;
        __syncthreads();
    }
    int run = threadSum[t] - sum;
    for (int c = c0; c < c1; c++) {
        const int n = count[c];
        G.cellStart[c] = run;
        count[c] = run;          // the fill position from here on
        run += n;
    }
    if (t == T - 1) G.cellStart[numCells] = run;
    __syncthreads();
    int* dst = SHARED ? scattered : G.cellSites;
    for (int s = t; s < C.numSites; s += T) dst[atomicAdd(&count[G.siteCell[s]], 1)] = s;
    __syncthreads();
    if (SHARED) {
        // the sites are distinct, so each one's rank among its cell's sites is its place
        const int warp = t >> 5, lane = t & 31;
        for (int c = warp; c < numCells; c += T >> 5) {
            const int start = G.cellStart[c], n = G.cellStart[c + 1] - start;
            for (int e = lane; e < n; e += 32) {
                const int x = scattered[start + e];
                int rank = 0;
                for (int f = 0; f < n; f++) rank += scattered[start + f] < x;
                G.cellSites[start + rank] = x;
            }
        }
        return;
    }
    // insertion sort of each cell's sites (a few dozen at most)
    for (int c = t; c < numCells; c += T) {
        int* v = G.cellSites + G.cellStart[c];
        const int n = G.cellStart[c + 1] - G.cellStart[c];
        for (int i = 1; i < n; i++) {
            const int x = v[i];
            int j = i - 1;
            while (j >= 0 && v[j] > x) {
                v[j + 1] = v[j];
                j--;
            }
            v[j + 1] = x;
        }
    }
}

// The list search over the cell grid (rebuild only): one warp per site A takes the sites B after A (siteAfter) of
// other molecules within the list cutoff from the 27 cells around A's cell, in cell order.  The 27 cells' sites are taken as one
// sequence (a prefix over the cell sizes), so the lanes stay busy across cell boundaries.  The distance test uses the
// float wrapped positions of the cell sort with a margin of 1e-4 of the squared list cutoff, far above their rounding
// (a few 1e-6): the list may hold a pair at the very edge of the list cutoff that the double-precision distance would
// leave out, never the reverse, and the triple kernels test the cutoff itself in double.  The counts and flags are
// those of kSiteNeighbors.  Launched with 256-thread blocks.
__global__ void __launch_bounds__(256) kSiteNeighborsCells(AtmBuffers A, AtmConfig C) {
    dependentStart(C.numSites <= kEarlySites);
    if (*(volatile int*)A.flag == 0) return;
    __shared__ int cellFirst[8][32], cellEnd[8][32];   // per warp: each cell's first site and its end in the sequence
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const SiteCells& G = A.cells;
    for (int a = blockIdx.x * 8 + w; a < C.numSites; a += gridDim.x * 8) {
        const float4 pa = G.wrapped[a];
        const int molA = __float_as_int(pa.w);
        const float cut2 = C.listCutoff2 * (1.0f + 1e-4f);
        const int cell = G.siteCell[a];
        const int cx = cell % G.nc[0], cy = (cell / G.nc[0]) % G.nc[1], cz = cell / (G.nc[0] * G.nc[1]);
        // lane k < 27 takes the cell (dx, dy, dz) = (k % 3, k / 3 % 3, k / 9) - 1, the order of three nested loops
        int first = 0, n = 0;
        if (lane < 27) {
            const int x = (cx + lane % 3 - 1 + G.nc[0]) % G.nc[0], y = (cy + lane / 3 % 3 - 1 + G.nc[1]) % G.nc[1],
                      z = (cz + lane / 9 - 1 + G.nc[2]) % G.nc[2];
            const int c = (z * G.nc[1] + y) * G.nc[0] + x;
            first = G.cellStart[c];
            n = G.cellStart[c + 1] - first;
        }
        int end = n;
    #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += v;
        }
        const int total = __shfl_sync(0xffffffffu, end, 31);
        cellFirst[w][lane] = first;
        cellEnd[w][lane] = end;
        __syncwarp();
        int count = 0;
        for (int k0 = 0; k0 < total; k0 += 32) {
            const int k = k0 + lane;
            int b = -1;
            if (k < total) {
                // the cell holding entry k: the first whose end exceeds k (binary search over the 27 ends)
                int lo = 0, hi = 26;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (cellEnd[w][mid] > k) hi = mid;
                    else lo = mid + 1;
                }
                const int before = lo ? cellEnd[w][lo - 1] : 0;
                b = G.cellSites[cellFirst[w][lo] + (k - before)];
            }
            bool near = false;
            if (b >= 0 && siteAfter(G, 0, a, b)) {
                const float4 pb = G.wrapped[b];
                float dx = pb.x - pa.x, dy = pb.y - pa.y, dz = pb.z - pa.z;
                dx -= C.boxf.a[0] * rintf(dx * C.boxf.inv[0]);
                dy -= C.boxf.b[1] * rintf(dy * C.boxf.inv[1]);
                dz -= C.boxf.c[2] * rintf(dz * C.boxf.inv[2]);
                near = __float_as_int(pb.w) != molA && fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < cut2;
            }
            const unsigned bal = __ballot_sync(0xffffffffu, near);
            if (near) {
                const int slot = count + __popc(bal & laneMaskLt());
                if (slot < A.cap) A.nbr[(size_t)a * A.cap + slot] = b;
            }
            count += __popc(bal);
        }
        if (lane == 0) {
            A.nbrCount[a] = count;
            if (count > A.cap) atomicOr(A.flag + 1, 1);
            if (count > kAtmFastStaged || count > A.cap) atomicOr(A.flag + 2, 1);
            if (a == 0) A.flag[3] = 0;
            for (int d = 0; d < 3; d++) A.siteRef[3 * a + d] = A.sitePos[3 * a + d];
        }
        __syncwarp();
    }
}

// Tang-Toennies f_3 and its derivative (InteraxThreeBodyTerms.h:51-65); the series is exact to float for x < 2 at
// k = 16.
__device__ __forceinline__ void tangToennies3f(float x, float& f, float& df) {
    const float e = expNeg(x);
    const float t3 = x * x * x * (1.0f / 6.0f);
    df = e * t3;
    if (x < 2.0f) {
        float term = t3, tail = 0.0f;
#pragma unroll
        for (int k = 4; k <= 16; k++) {
            term *= x * (1.0f / k);
            tail += term;
        }
        f = e * tail;
    }
    else f = fmaf(-e, ((1.0f + x) + 0.5f * x * x) + t3, 1.0f);
}

// g = 1 - exp(-(r/R0)^6) and g' (InteraxThreeBodyTerms.h:71-77).
__device__ __forceinline__ void centroidDampingF(float r, float invR0, float& g, float& dg) {
    const float x = r * invR0;
    float x6 = x * x * x;
    x6 *= x6;
    const float e = expNeg(x6);
    g = x6 < 0.01f ? x6 * fmaf(-0.5f * x6, fmaf(-x6, 1.0f / 3.0f, 1.0f), 1.0f) : 1.0f - e;
    dg = 6.0f * x6 * e * rcpApprox(r);
}

// A staged neighbor k of site A.  pos: displacement from A and its squared length; par: frequency, the frequency and
// polarizability part of C9 that A and k make, alchemical (0/1), molecule (int bits); damp (damping only): width, the
// damping of the A-k distance, its r-derivative over the distance.
struct SiteDamping {
    float width, f, dfr;
};

// Damping of one distance: Tang-Toennies of the two widths' sum and the centroid damping (InteraxThreeBodyTerms.h:51-77),
// and its r-derivative divided by r.
__device__ __forceinline__ void siteDamping(const AtmConfig& C, float r2, float widths, float& f, float& dfr) {
    float invR;
    const float r = sqrtRefined(r2, invR);
    float df = 0.0f;
    f = 1.0f;
    if (C.useTangToennies) {
        const float rate = C.twoBeta * __fdividef(1.0f, widths);
        tangToennies3f(rate * r, f, df);
        df *= rate;
    }
    if (C.invCentroidRadius > 0.0f) {
        float g, dg;
        centroidDampingF(r, C.invCentroidRadius, g, dg);
        df = fmaf(df, g, f * dg);
        f *= g;
    }
    dfr = df * invR;
}

// What one warp stages per neighbor.
template <bool DAMP, int N>
struct TripleStorage {
    float4 pos[N];
    float4 par[N];
    int site[N];
    SiteDamping damp[DAMP ? N : 1];
};

template <bool DAMP, int N>
__device__ __forceinline__ void storeNeighbor(TripleStorage<DAMP, N>& S, const AtmBuffers& A, const AtmConfig& C,
                                              const float4& pa, int slot, int b, float x, float y, float z) {
    const float4 p = A.siteParams[b];
    const float u = fmaf(x, x, fmaf(y, y, z * z));
    const float sum = pa.y + p.y, inv = rcpApprox(sum), product = p.x * p.y, g = product * inv;
    S.pos[slot] = make_float4(x, y, z, u);
    // C9 = 3/2 aA aB aC wA wB wC (wA + wB + wC)/((wA + wB)(wB + wC)(wC + wA)) (InteraxThreeBodyForceImpl.h:69-72)
    //    = (3/2 aA wA) gB gC (1 + wA/(wB + wC)),  g = a w/(wA + w)
    S.par[slot] = make_float4(p.y, fmaf(fmaf(-sum, g, product), inv, g), p.w, __int_as_float(A.molecule[b]));
    S.site[slot] = b;
    if (DAMP) {
        SiteDamping d;
        d.width = p.z;
        siteDamping(C, u, pa.z + p.z, d.f, d.dfr);
        S.damp[slot] = d;
    }
}

// One warp's share of the triples of site A (parameters pa): the neighbors C of storage entries cFirst, cFirst +
// cStep, ... (8 at a time, below cEnd), each against every neighbor B of entries [bBegin, bEnd).  Four lanes take one
// C; lane s of them takes B = bBegin + s, + 4, ...  A triple is visited from both sides, and each visit adds the
// force on its own C only: the same number of warp iterations as visiting it once with half of the lanes idle, and
// a third of the arithmetic of all three forces.  The force on A is minus the sum of the others', in fixed point.
//   energy (InteraxThreeBodyTerms.h:97-146), with a = AB, b = AC, c = BC, p = a.b, q = a.c, s = b.c, P = (a b c)^2:
//     E = C9 (P^-3/2 - 3 p q s P^-5/2)
//     -force on C = b (R/b^2 + t) + c (R/c^2 + t) + a X s (p + q),
//     R = C9 (15 p q s P^-5/2 - 3 P^-3/2), X = -3 C9 P^-5/2, t = X p q
//   C9 with the scale and the alchemical factor (ReferenceInteraxThreeBodyIxn.cpp:116-120).
// Relative RMS errors of the three-body force against FP64 (means of six): 24,000 atoms 3.00e-7, 96,000 atoms 3.01e-7,
// 258 sites without a cutoff 2.62e-7.  With the sums of a lane in one row of up to 64, approximate quotients throughout and
// the force on A summed in float they were 3.16e-7, 3.22e-7 and 3.76e-7, in the same time; an energy is summed in FP64,
// one C's terms at a time.
// What bounds it: FP32 issue, about 75 instructions a visit, and for a few thousand sites the latency of the staging
// (list, position, parameters, three dependent loads).  The earlier form gave each lane a pair (B, C) of a flat
// triangular index, stored both forces in shared memory and gathered them per neighbor, 425 issue slots per 32 pairs.
// Kernel times on one B200, both triple kernels with a warp per site, before and now: 96,000-atom box, 0.8 nm, 13.6 M
// triples: 410 and 166 us; 24,000 atoms, 0.6 nm, 0.46 M triples: 27 and 25 us.  Beside the pair kernel, on two blocks an
// SM, the 24,000-atom launch takes 41 us of the pair kernel's 110 and is hidden behind it.
template <bool DAMP, bool IMAGE, bool ALCH, int N>
__device__ __forceinline__ void siteTriples(const TripleStorage<DAMP, N>& S, const AtmBuffers& A, const AtmConfig& C,
                                            const float4& pa, int cFirst, int cStep, int cEnd, int bBegin, int bEnd,
                                            int lane, long long& fa, double& energy,
                                            unsigned long long& visits) {
    unsigned seen = 0;
    const int s = lane & 3;
    const float kA = 1.5f * pa.x * pa.y * C.scale * (pa.w != 0.0f ? C.lambda : 1.0f);
    const float lambdaBC = pa.w != 0.0f ? 1.0f : C.lambda;
    for (int c0 = cFirst; c0 < cEnd; c0 += cStep) {
        const int k = c0 + (lane >> 2);
        const bool have = k < cEnd;
        const float4 xc = S.pos[have ? k : cFirst], pc = S.par[have ? k : cFirst];
        SiteDamping dc;
        if (DAMP) dc = S.damp[have ? k : cFirst];
        float invV = rcpApprox(xc.w);
        invV = fmaf(invV, fmaf(-xc.w, invV, 1.0f), invV);
        // along: the factor of xc, summed over B
        float gx = 0.0f, gy = 0.0f, gz = 0.0f, along = 0.0f, eC = 0.0f;
        auto visit = [&](int b) {
            const float4 xb = S.pos[b], pb = S.par[b];
            if (__float_as_int(pb.w) == __float_as_int(pc.w)) return;      // one molecule, B = C among them
            float cx = xc.x - xb.x, cy = xc.y - xb.y, cz = xc.z - xb.z;
            if (IMAGE) minimumImageF(cx, cy, cz, C.boxf);
            const float w = fmaf(cx, cx, fmaf(cy, cy, cz * cz));
            if (!(w < C.cutoff2)) return;
            float c9 = (pb.y * pc.y) * kA * fmaf(pa.y, rcpApprox(pb.x + pc.x), 1.0f);
            if (pb.z != 0.0f || pc.z != 0.0f) c9 *= lambdaBC;
            else if (ALCH && pa.w == 0.0f) return;
            if (c9 == 0.0f) return;
            const float p = fmaf(xb.x, xc.x, fmaf(xb.y, xc.y, xb.z * xc.z));
            const float q = fmaf(xb.x, cx, fmaf(xb.y, cy, xb.z * cz));
            const float r = fmaf(xc.x, cx, fmaf(xc.y, cy, xc.z * cz));
            const float P = xb.w * xc.w * w;
            float y = rsqrtApprox(P);
            y = fmaf(fmaf(-P * y, y, 1.0f), 0.5f * y, y);      // its fifth power is taken
            const float invP = y * y;
            const float invP32 = invP * y;
            const float invP52 = invP32 * invP;
            const float pq = p * q;
            const float pqr = pq * r;
            const float e = c9 * fmaf(-3.0f * pqr, invP52, invP32);
            const float radial = c9 * fmaf(15.0f * pqr, invP52, -3.0f * invP32);
            const float cross = -3.0f * c9 * invP52;
            const float t = cross * pq;
            float kb = fmaf(radial, invV, t), kc = fmaf(radial, rcpApprox(w), t), ka = cross * r * (p + q);
            if (DAMP) {
                const SiteDamping db = S.damp[b];
                float f, dfr;
                siteDamping(C, w, db.width + dc.width, f, dfr);
                const float fbc = db.f * f, damping = dc.f * fbc;
                kb = fmaf(kb, damping, e * fbc * dc.dfr);
                kc = fmaf(kc, damping, e * db.f * dc.f * dfr);
                ka *= damping;
                eC = fmaf(e, damping, eC);
            }
            else eC += e;
            along += kb;
            gx = fmaf(cx, kc, fmaf(xb.x, ka, gx));
            gy = fmaf(cy, kc, fmaf(xb.y, ka, gy));
            gz = fmaf(cz, kc, fmaf(xb.z, ka, gz));
            seen++;
        };
        const int first = have ? bBegin + s : bEnd;
        if constexpr (N > kAtmFastStaged)
            // a long list in runs of eight a lane, whose sums are added up
            for (int b0 = first; b0 < bEnd; b0 += 32) {
                const float sx = gx, sy = gy, sz = gz, sAlong = along;
                gx = gy = gz = along = 0.0f;
                for (int b = b0; b < min(b0 + 32, bEnd); b += 4) visit(b);
                gx += sx;
                gy += sy;
                gz += sz;
                along += sAlong;
            }
        else
            for (int b = first; b < bEnd; b += 4) visit(b);
        gx = fmaf(xc.x, along, gx);
        gy = fmaf(xc.y, along, gy);
        gz = fmaf(xc.z, along, gz);
        __syncwarp();
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            gx += __shfl_xor_sync(0xffffffffu, gx, o);
            gy += __shfl_xor_sync(0xffffffffu, gy, o);
            gz += __shfl_xor_sync(0xffffffffu, gz, o);
        }
        energy += (double)eC;
        // lane s of the four adds component s
        const long long g = have && s < 3 ? toFixed(s == 0 ? gx : (s == 1 ? gy : gz)) : 0;
        fa += g;
        if (g != 0) atomicAddFixed(A.siteForce + s * C.numSites + S.site[k], -g);
    }
    visits += seen;
}

// The force on A of a warp's share (lane s < 3 of every four holds component s).
__device__ __forceinline__ void addSiteForce(const AtmBuffers& A, const AtmConfig& C, int a, int lane, long long fa) {
    for (int o = 4; o < 32; o <<= 1) fa += __shfl_xor_sync(0xffffffffu, fa, o);
    if (lane < 3 && fa != 0) atomicAddFixed(A.siteForce + lane * C.numSites + a, fa);
}

// Stage the neighbors of site a that are within the cutoff (in list order) with their displacements from a and their
// parameters; returns how many there are (at most `capacity` are stored).
template <class Store>
__device__ __forceinline__ int stageTripleNeighbors(const AtmBuffers& A, const AtmConfig& C, int a, int n, int lane,
                                                    int first, int capacity, Store store) {
    int m = 0;
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int k = k0 + lane;
        bool in = false;
        double d[3];
        int b = -1;
        if (k < n) {
            b = A.nbr[(size_t)a * A.cap + k];
            siteDelta(A, C, a, b, d);
            in = (float)(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]) < C.cutoff2;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, in);
        if (in) {
            const int slot = m + __popc(bal & laneMaskLt()) - first;
            if (slot >= 0 && slot < capacity) store(slot, b, (float)d[0], (float)d[1], (float)d[2]);
        }
        m += __popc(bal);
    }
    return m;
}

// The same for a site whose list overflowed its capacity: every site after it (in the order of the lists' build) of
// another molecule is tested against the cutoff, which gives the same neighbors, so the same triples are evaluated.
// The reference falls back the same way
// (platforms/common/src/kernels/interaxThreeBody.cc:111-112, 437-438).
template <class Store>
__device__ __forceinline__ int stageTripleNeighborsScan(const AtmBuffers& A, const AtmConfig& C, int a, int lane,
                                                        int first, int capacity, Store store) {
    const int molA = A.molecule[a], byIndex = A.flag[3];
    int m = 0;
    for (int b0 = byIndex ? a + 1 : 0; b0 < C.numSites; b0 += 32) {
        const int b = b0 + lane;
        bool in = false;
        double d[3];
        if (b < C.numSites && A.molecule[b] != molA && siteAfter(A.cells, byIndex, a, b)) {
            siteDelta(A, C, a, b, d);
            in = (float)(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]) < C.cutoff2;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, in);
        if (in) {
            const int slot = m + __popc(bal & laneMaskLt()) - first;
            if (slot >= 0 && slot < capacity) store(slot, b, (float)d[0], (float)d[1], (float)d[2]);
        }
        m += __popc(bal);
    }
    return m;
}

static_assert(kAtmFastWarps * sizeof(TripleStorage<true, kAtmFastStaged>) < 48 * 1024, "static shared memory of a block");
static_assert((kAtmFastWarps * sizeof(TripleStorage<true, kAtmFastStaged>) + 1024) * IX_TUNE_ATM_MIN_BLOCKS <= 228 * 1024,
              "shared memory of the blocks an SM is asked to hold");

template <bool DAMP, bool IMAGE, bool ALCH>
__global__ void __launch_bounds__(32 * kAtmFastWarps, IX_TUNE_ATM_MIN_BLOCKS) kTriplesFast(AtmBuffers A, AtmConfig C) {
    dependentStart(false);
    __shared__ TripleStorage<DAMP, kAtmFastStaged> storage[kAtmFastWarps];
    auto& S = storage[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int warp = blockIdx.x * kAtmFastWarps + (threadIdx.x >> 5);
    const int fastMax = fastListMax(A);
    double eAcc = 0.0;
    unsigned long long visits = 0;
    for (int a = warp; a < C.numSites; a += gridDim.x * kAtmFastWarps) {
        const int n = A.nbrCount[a];
        if (n > fastMax || n > A.cap) continue;        // the wide kernel takes this site
        const float4 pa = A.siteParams[a];
        if (ALCH && pa.w == 0.0f) {
            // only the triples with an alchemical site: most sites have none
            bool any = false;
            for (int k = lane; k < n; k += 32) any |= A.siteParams[A.nbr[(size_t)a * A.cap + k]].w != 0.0f;
            if (!__any_sync(0xffffffffu, any)) continue;
        }
        __syncwarp();
        const int m = stageTripleNeighbors(A, C, a, n, lane, 0, kAtmFastStaged,
                                           [&](int slot, int b, float x, float y, float z) {
                                               storeNeighbor(S, A, C, pa, slot, b, x, y, z);
                                           });
        __syncwarp();
        long long fa = 0;
        siteTriples<DAMP, IMAGE, ALCH>(S, A, C, pa, 0, 8, m, 0, m, lane, fa, eAcc, visits);
        addSiteForce(A, C, a, lane, fa);
    }
    const double sum = 0.5 * warpSumD(eAcc);           // each triple was visited twice
    if (lane == 0) A.energyPartials[warp] = sum;
    for (int o = 16; o > 0; o >>= 1) visits += __shfl_xor_sync(0xffffffffu, visits, o);
    if (lane == 0 && visits) atomicAdd(A.tripleVisits, visits);
}

constexpr int kAtmWarps = 4;
constexpr int kAtmMaxStaged = 256;
constexpr int kAtmChunk = kAtmMaxStaged / 2;
static_assert(kAtmWarps * sizeof(TripleStorage<true, kAtmMaxStaged>) <= 48 * 1024,
              "dynamic shared memory of a block without asking for more than the default");
// Each long-list site is taken by this many warps, each evaluating every kAtmWideParts-th group of 8 of its neighbors:
// a site near the start of a large cluster has tens of thousands of (B, C) pairs, which one warp would take alone.
constexpr int kAtmWideParts = 8;

// Sites whose lists are longer than the fast kernel takes, in units (site, part) of kAtmWideParts parts per site.  A
// unit stages up to kAtmMaxStaged neighbors within the cutoff at once and evaluates its part of them against all; a
// longer list is taken in chunks of kAtmChunk, each pair of chunks staged side by side, so any length is handled.
// Energies go to energyPartials[partialsOffset + warp]: with a grid of one warp per unit, one slot per unit (unit =
// site x kAtmWideParts + part).
// `gate` (may be null): the kernel returns at once unless *gate is set (a list longer than the fast kernel takes).
template <bool DAMP, bool IMAGE, bool ALCH>
__global__ void __launch_bounds__(32 * kAtmWarps) kTriplesWide(AtmBuffers A, AtmConfig C, int partialsOffset,
                                                               const int* gate) {
    dependentStart(C.numSites <= kEarlySites);
    if (gate && *(volatile const int*)gate == 0) return;
    extern __shared__ float4 atmShared[];
    auto& S = reinterpret_cast<TripleStorage<DAMP, kAtmMaxStaged>*>(atmShared)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int fastMax = fastListMax(A);
    double eAcc = 0.0;
    unsigned long long visits = 0;
    const int units = C.numSites * kAtmWideParts;
    for (int u = blockIdx.x * kAtmWarps + (threadIdx.x >> 5); u < units; u += gridDim.x * kAtmWarps) {
        const int a = u / kAtmWideParts, part = u % kAtmWideParts;
        const int n = A.nbrCount[a];
        if (n <= fastMax && n <= A.cap) continue;      // the fast kernel takes this site
        const float4 pa = A.siteParams[a];
        const bool scan = n > A.cap;                   // the list overflowed: scan the sites
        auto stage = [&](int first, int base, int capacity) {
            auto store = [&](int slot, int b, float x, float y, float z) {
                storeNeighbor(S, A, C, pa, base + slot, b, x, y, z);
            };
            return scan ? stageTripleNeighborsScan(A, C, a, lane, first, capacity, store)
                        : stageTripleNeighbors(A, C, a, n, lane, first, capacity, store);
        };
        long long fa = 0;
        __syncwarp();
        const int m = stage(0, 0, kAtmMaxStaged);
        __syncwarp();
        if (m <= kAtmMaxStaged) {
            siteTriples<DAMP, IMAGE, ALCH>(S, A, C, pa, 8 * part, 8 * kAtmWideParts, m, 0, m, lane, fa, eAcc, visits);
        }
        else {
            const int chunks = (m + kAtmChunk - 1) / kAtmChunk;
            for (int I = 0; I < chunks; I++) {
                const int cI = min(kAtmChunk, m - I * kAtmChunk);
                for (int J = 0; J < chunks; J++) {
                    const int cJ = min(kAtmChunk, m - J * kAtmChunk);
                    __syncwarp();
                    stage(I * kAtmChunk, 0, kAtmChunk);
                    if (J != I) stage(J * kAtmChunk, kAtmChunk, kAtmChunk);
                    __syncwarp();
                    const int b0 = J == I ? 0 : kAtmChunk;
                    siteTriples<DAMP, IMAGE, ALCH>(S, A, C, pa, 8 * part, 8 * kAtmWideParts, cI, b0, b0 + cJ, lane, fa,
                                                   eAcc, visits);
                }
            }
        }
        addSiteForce(A, C, a, lane, fa);
        __syncwarp();
    }
    const double sum = 0.5 * warpSumD(eAcc);
    if (lane == 0) A.energyPartials[partialsOffset + blockIdx.x * kAtmWarps + (threadIdx.x >> 5)] = sum;
    for (int o = 16; o > 0; o >>= 1) visits += __shfl_xor_sync(0xffffffffu, visits, o);
    if (lane == 0 && visits) atomicAdd(A.tripleVisits, visits);
}

// The wide kernel where its grid is not empty, and the fast one.  The wide kernel mostly returns at once: it goes
// first, while there is room on the SMs; behind the fast one it waited for the pair kernel's last blocks.  `before` (may
// be null) is recorded ahead of the fast kernel.  ALCH: only the triples with an alchemical site.
template <bool DAMP, bool IMAGE, bool ALCH>
static void launchTriplesAs(const AtmBuffers& A, const AtmConfig& C, int fastBlocks, int wideBlocks, const int* gate,
                            cudaStream_t st, cudaEvent_t before, bool early) {
    if (wideBlocks > 0)
        launchNext(early, st, kTriplesWide<DAMP, IMAGE, ALCH>, wideBlocks, 32 * kAtmWarps,
                   kAtmWarps * sizeof(TripleStorage<DAMP, kAtmMaxStaged>), A, C, fastBlocks * kAtmFastWarps, gate);
    if (before) cudaEventRecord(before, st);
    launchNext(early && C.numSites <= kEarlySites, st, kTriplesFast<DAMP, IMAGE, ALCH>, fastBlocks, 32 * kAtmFastWarps, 0, A, C);
}
template <bool ALCH>
static void launchTriples(const AtmBuffers& A, const AtmConfig& C, int fastBlocks, int wideBlocks, const int* gate,
                          cudaStream_t st, cudaEvent_t before = nullptr, bool early = false) {
    const bool damp = C.useTangToennies || C.invCentroidRadius > 0.0f;
    if (damp && C.imageBC) launchTriplesAs<true, true, ALCH>(A, C, fastBlocks, wideBlocks, gate, st, before, early);
    else if (damp) launchTriplesAs<true, false, ALCH>(A, C, fastBlocks, wideBlocks, gate, st, before, early);
    else if (C.imageBC) launchTriplesAs<false, true, ALCH>(A, C, fastBlocks, wideBlocks, gate, st, before, early);
    else launchTriplesAs<false, false, ALCH>(A, C, fastBlocks, wideBlocks, gate, st, before, early);
}

// Each particle of a site receives the site force divided by the number of particles
// (ReferenceInteraxThreeBodyIxn.cpp:127-133).  The site forces are cleared as they are read.
__global__ void kSpreadSiteForces(AtmBuffers A, AtmConfig C) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= C.numSites) return;
    const int b = A.siteOffsets[s], e = A.siteOffsets[s + 1];
    const double inv = 1.0 / (double)(e - b);
    for (int d = 0; d < 3; d++) {
        const long long v = A.siteForce[d * C.numSites + s];
        if (v == 0) continue;
        A.siteForce[d * C.numSites + s] = 0;
        const long long share = __double2ll_rn((double)v * inv);
        for (int k = b; k < e; k++) atomicAddFixed(A.particleForce + (size_t)d * A.numParticles + A.siteParticles[k], share);
    }
}

}  // namespace ix
