// Device kd-tree build: the caller-side tree of the P2P pass (PhotoNs'
// build_kdtree / center_kdtree, src/fmm.c:69-122,231-327) built on the GPU
// with the same nodes, leaves, numbering and particle order.
//
// The reference splits a node of n particles at the mean of its coordinate
// on axis depth % 3 (sampled every max(1, n / 1e5)-th particle, summed in
// order) with an in-place two-pointer partition (bksort_inplace,
// src/fmm.c:69-122). That partition has a parallel form, used here: with nS
// the number of particles not above the mean, the k-th particle above the
// mean among the first nS slots swaps with the k-th particle not above it
// counted from the right among the last n - nS slots; the left child takes
// nS particles, or n - 1 when none lies above the mean; a node of two
// particles splits at their midpoint, swapping them when the first is above
// the second. Nodes are split level by level while they hold more than
// kTreeSmall particles (the partition by tiles of the node's slots, a level's
// children by one block, with no host between); smaller subtrees are built whole
// by one block each in shared memory. Nodes and leaves get build-order ids as they
// are made; the pre-order ids of the reference (son[0]'s subtree first, leaves
// numbered apart from nodes) and the node boxes follow from three passes: parents,
// counts from the leaves up, numbers and boxes from each node's path to the root.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace p2p {

constexpr int kTreeSmall = 2048;       // subtrees up to this size are built by one block
constexpr int kTreeTile = 2048;        // slots per tile of the level-wide partition
constexpr int kTreeThreads = 256;

// Status bits of the tree build.
enum : int {
    TB_NODE_CAP = 1,   // more nodes than the build's node capacity
    TB_LEAF_CAP = 2,   // more leaves than the leaf capacity
    TB_NUMBERING = 4,  // a pre-order id out of range (inconsistent records; nothing written)
};

// Build-order records (structure of arrays) of nodes and leaves.
struct TreeRec {
    // nodes
    double *split;
    int *son;      // 2 per node: build id of a leaf l -> 2l, of a node k -> 2k+1
    int *depth;
    int *nn, *nl;  // nodes and leaves in the node's subtree (itself included)
    int *pre;      // pre-order id
    int *first;    // pre-order id of the subtree's first leaf
    double *box;   // 6 per node: left[3], right[3]
    double *root;  // the root's
    int node_cap;
    // leaves
    int *lipart, *lnpart, *lid;  // particle range, pre-order leaf id
    int leaf_cap;
    int *counters;  // [0] nodes made, [1] leaves made, [2] status bits
};

// Particles being partitioned: SoA coordinates and original indices.
struct TreeParts {
    double *x, *y, *z;
    int *id;
};

__device__ __forceinline__ double tree_coord(const TreeParts &P, int axis, int i) {
    return axis == 0 ? P.x[i] : (axis == 1 ? P.y[i] : P.z[i]);
}

__device__ __forceinline__ void tree_swap(TreeParts &P, int i, int j) {
    const double tx = P.x[i], ty = P.y[i], tz = P.z[i];
    const int ti = P.id[i];
    P.x[i] = P.x[j]; P.y[i] = P.y[j]; P.z[i] = P.z[j]; P.id[i] = P.id[j];
    P.x[j] = tx; P.y[j] = ty; P.z[j] = tz; P.id[j] = ti;
}

// ------------------------------------------------------ the split value ---
//
// The reference's split value of a node of length >= 3 is the sampled mean,
// summed in slot order (src/fmm.c:88-97), so its rounding is that of a chain of
// up to 2e5 dependent FP64 additions. One thread makes one in 10 cycles (the
// addition takes 8.4), 0.87 ms a level of a 256^3 tree as it was and 12 of the
// tree's 26 ms. Short nodes keep the chain, many side by side; for long ones its
// result is found in parallel, bit for bit: while the running sum stays in one
// binade its unit in the last place u does not change, adding x moves it by x
// rounded to a multiple of u, which (S + x) - S gives exactly for any S of that
// binade, unless x lies half way between two multiples, where the chain rounds
// by its own parity. Those moves and their sums are multiples of u below 2^53
// of them, so FP64 adds them exactly in any order. A group of samples is
// therefore applied at once when it holds no half and S stays inside its binade
// whatever the order of the group's moves up and down; a group that might leave
// it goes through in shorter groups and, where need be, in the chain. Binades
// are left, and halves met, about log2(samples) times each.

// S after the n samples at s (shared memory: every lane reads the same word),
// added one by one.
__device__ __forceinline__ double mean_chain(const double *s, int n, double S) {
#pragma unroll 16
    for (int i = 0; i < n; ++i) S = __dadd_rn(S, s[i]);
    return S;
}

// The moves of a group of samples.
struct MeanMoves {
    double sum, size;  // their sum, and the sum of their magnitudes
    bool half;         // one of the samples rounds by parity
};

// S's binade as [lo, 2 lo) and half its unit; false where a chain must be
// followed sample by sample (zero, near-subnormal, huge or not finite).
__device__ __forceinline__ bool mean_binade(double S, double &lo, double &half_u) {
    const int e = (__double2hiint(S) >> 20) & 0x7ff;
    lo = __hiloint2double(e << 20, 0);
    half_u = __hiloint2double((e - 53) << 20, 0);
    return e >= 100 && e <= 2000;
}

__device__ __forceinline__ void mean_add(MeanMoves &g, double x, double S, double half_u) {
    const double move = __dsub_rn(__dadd_rn(S, x), S);
    g.sum = __dadd_rn(g.sum, move);
    g.size = __dadd_rn(g.size, fabs(move));
    g.half = g.half || fabs(__dsub_rn(x, move)) == half_u;
}

// Whether a group of moves may be applied to S at once (NaN and infinity fail):
// size + sum and size - sum are twice its moves up and down, exactly.
__device__ __forceinline__ bool mean_fits(double S, double lo, double sum, double size) {
    const double along = S < 0.0 ? -sum : sum, m = fabs(S);
    const double less = __dmul_rn(0.5, __dsub_rn(size, along)), more = __dmul_rn(0.5, __dadd_rn(size, along));
    return __dsub_rn(m, less) > lo && __dadd_rn(m, more) < __dadd_rn(lo, lo);
}

// The lanes' moves together (in every lane); half also where S might leave its
// binade under them.
__device__ __forceinline__ MeanMoves mean_gather(MeanMoves m, double S, double lo) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        m.sum = __dadd_rn(m.sum, __shfl_xor_sync(0xffffffffu, m.sum, off));
        m.size = __dadd_rn(m.size, __shfl_xor_sync(0xffffffffu, m.size, off));
    }
    m.half = __any_sync(0xffffffffu, m.half) || !mean_fits(S, lo, m.sum, m.size);
    return m;
}

// S after one warp's n samples at s (shared memory), 128 at a time.
__device__ __forceinline__ double mean_warp(const double *s, int n, double S) {
    const int lane = threadIdx.x & 31;
    for (int b = 0; b < n; b += 128) {
        const int m = min(128, n - b);
        double lo, half_u;
        if (mean_binade(S, lo, half_u)) {
            MeanMoves g = {0.0, 0.0, false};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (32 * i + lane < m) mean_add(g, s[b + 32 * i + lane], S, half_u);
            g = mean_gather(g, S, lo);
            if (!g.half) {
                S = __dadd_rn(S, g.sum);
                continue;
            }
        }
        S = mean_chain(s + b, m, S);
    }
    return S;
}

// -------------------------------------------------------------- inputs ---

// Copies the positions into the work arrays, ids = slot, and per-block
// min / max of the float-rounded coordinates (particle_combine's bounds,
// src/gravity.c:69-121).
__global__ void tree_init_kernel(const double *__restrict__ pos, int n, TreeParts P,
                                 float *__restrict__ block_lo, float *__restrict__ block_hi) {
    __shared__ float slo[3][kTreeThreads], shi[3][kTreeThreads];
    float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double c[3] = {pos[i], pos[(size_t)n + i], pos[2 * (size_t)n + i]};
        P.x[i] = c[0];
        P.y[i] = c[1];
        P.z[i] = c[2];
        P.id[i] = i;
        for (int d = 0; d < 3; ++d) {
            const float f = (float)c[d];
            lo[d] = fminf(lo[d], f);
            hi[d] = fmaxf(hi[d], f);
        }
    }
    for (int d = 0; d < 3; ++d) {
        slo[d][threadIdx.x] = lo[d];
        shi[d][threadIdx.x] = hi[d];
    }
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s)
            for (int d = 0; d < 3; ++d) {
                slo[d][threadIdx.x] = fminf(slo[d][threadIdx.x], slo[d][threadIdx.x + s]);
                shi[d][threadIdx.x] = fmaxf(shi[d][threadIdx.x], shi[d][threadIdx.x + s]);
            }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int d = 0; d < 3; ++d) {
            block_lo[3 * blockIdx.x + d] = slo[d][0];
            block_hi[3 * blockIdx.x + d] = shi[d][0];
        }
}

// The root box: boxL = min(boxsize, min float coordinate) - 1e-6 boxsize,
// boxH = max(0, max float coordinate) + 1e-6 boxsize, per axis (one block of
// three warps, one axis each).
__global__ void __launch_bounds__(96)
tree_root_box_kernel(const float *__restrict__ block_lo, const float *__restrict__ block_hi, int nblocks,
                     double boxsize, TreeRec R) {
    const int lane = threadIdx.x & 31, d = threadIdx.x >> 5;
    double lo = boxsize, hi = 0.0;
    for (int b = lane; b < nblocks; b += 32) {
        const double l = (double)block_lo[3 * b + d], h = (double)block_hi[3 * b + d];
        if (lo > l) lo = l;
        if (hi < h) hi = h;
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) {
        const double margin = __dmul_rn(0.000001, boxsize);
        R.root[d] = __dsub_rn(lo, margin);
        R.root[3 + d] = __dadd_rn(hi, margin);
    }
}

// ---------------------------------------------------- level-wide split ---

// A node split level-wide: its slots, axis, and (after the count) the number
// of its particles not above the mean.
struct TreeSeg {
    int ipart, length, axis, node;
    double mean;
    int nsmall, nbig;
    int tile0, before;  // its first tile; slots not above their means in the tiles before that
};

// Levels split level-wide: the counts of each, made by tree_level_kernel for the
// next one, so the levels are queued without the host reading between them.
constexpr int kTreeLevels = 4096;
struct TreeLevels {
    int nseg[kTreeLevels + 1], ntile[kTreeLevels + 1];
    int ntask;  // subtrees for one block each
};

// Segments whose chain of additions is made as it is, one warp per segment:
// short ones, and all of a level that has so many that they fill the GPU side
// by side (at 256^3 the levels of 512 and more segments took 4.4 ms with a block
// each).
constexpr int kMeanChainMax = 8192;
constexpr int kMeanChainSegs = 512;
__host__ __device__ __forceinline__ bool tree_takes_chain(int length, int nseg) {
    return length <= kMeanChainMax || (nseg >= kMeanChainSegs && length <= 100000);
}

__global__ void __launch_bounds__(128) tree_seg_chain_kernel(TreeSeg *segs, const TreeLevels *lv, int level,
                                                             TreeParts P, TreeRec R) {
    constexpr int kBatch = 256;
    __shared__ double batch[4][kBatch];
    const int lane = threadIdx.x & 31;
    const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nseg = lv->nseg[level];
    if (q >= nseg) return;
    const TreeSeg g = segs[q];
    if (!tree_takes_chain(g.length, nseg)) return;
    const double *c = (g.axis == 0 ? P.x : (g.axis == 1 ? P.y : P.z)) + g.ipart;
    double *s = batch[threadIdx.x >> 5];
    double S = 0.0, next[kBatch / 32];
#pragma unroll
    for (int i = 0; i < kBatch / 32; ++i) next[i] = 32 * i + lane < g.length ? c[32 * i + lane] : 0.0;
    for (int b = 0; b < g.length; b += kBatch) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kBatch / 32; ++i) s[32 * i + lane] = next[i];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kBatch / 32; ++i) {  // in flight during the additions
            const int k = b + kBatch + 32 * i + lane;
            next[i] = k < g.length ? c[k] : 0.0;
        }
        S = mean_chain(s, min(kBatch, g.length - b), S);
    }
    if (lane == 0) {
        const double mean = __ddiv_rn(S, (double)g.length);
        segs[q].mean = mean;
        R.split[g.node] = mean;
    }
}

// One block per longer segment: the split value, in windows of 8 groups of 512
// samples, a warp to a group (any lane may hold any of its samples: the loads
// are coalesced where the samples are contiguous). Groups that fit S's binade
// are applied by every thread; the owner of one that does not puts it in order
// in shared memory, works it out (mean_warp) and hands S on. The other groups'
// moves stay good while S stays in the binade they were found in.
constexpr int kMeanPerLane = 16;
constexpr int kMeanGroup = 32 * kMeanPerLane;
__global__ void __launch_bounds__(kTreeThreads, 3) tree_seg_mean_kernel(TreeSeg *segs, const TreeLevels *lv,
                                                                         int level, TreeParts P, TreeRec R) {
    constexpr int kWarps = kTreeThreads / 32;
    __shared__ MeanMoves groups[kWarps];
    __shared__ double s_sum;
    __shared__ double order[kMeanGroup];  // the group that is worked out
    const int nseg = lv->nseg[level];
    if ((int)blockIdx.x >= nseg) return;
    const TreeSeg g = segs[blockIdx.x];
    if (tree_takes_chain(g.length, nseg)) return;
    const double *c = (g.axis == 0 ? P.x : (g.axis == 1 ? P.y : P.z)) + g.ipart;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int mul = 1;
    if (g.length > 100000) mul = g.length / 100000;
    const int nsamp = (g.length + mul - 1) / mul;  // slots 0, mul, 2 mul, ... < length
    double S = 0.0;  // the same in every thread
    for (int s0 = 0; s0 < nsamp; s0 += kWarps * kMeanGroup) {
        double x[kMeanPerLane];
        const int first = s0 + w * kMeanGroup, last = min(nsamp, first + kMeanGroup);
#pragma unroll
        for (int i = 0; i < kMeanPerLane; ++i)
            x[i] = first + 32 * i + lane < last ? c[(size_t)(first + 32 * i + lane) * mul] : 0.0;
        const int ngroup = min(kWarps, (nsamp - s0 + kMeanGroup - 1) / kMeanGroup);
        int cur = 0;          // groups of the window already in S
        double found = -1.0;  // the binade that the window's moves belong to
        while (cur < ngroup) {
            double lo, half_u;
            if (mean_binade(S, lo, half_u)) {
                if (lo != found) {
                    if (w >= cur && w < ngroup) {
                        MeanMoves m = {0.0, 0.0, false};
#pragma unroll
                        for (int i = 0; i < kMeanPerLane; ++i)
                            if (first + 32 * i + lane < last) mean_add(m, x[i], S, half_u);
                        // moves found at this S hold at every S of the binade that they keep within it
                        m = mean_gather(m, S, lo);
                        if (lane == 0) groups[w] = m;
                    }
                    found = lo;
                    __syncthreads();
                }
                while (cur < ngroup && !groups[cur].half && mean_fits(S, lo, groups[cur].sum, groups[cur].size))
                    S = __dadd_rn(S, groups[cur++].sum);
            }
            if (cur < ngroup) {
                if (w == cur) {
#pragma unroll
                    for (int i = 0; i < kMeanPerLane; ++i) order[32 * i + lane] = x[i];
                    __syncwarp();
                    S = mean_warp(order, last - first, S);
                    if (lane == 0) s_sum = S;
                }
                __syncthreads();
                S = s_sum;
                ++cur;
            }
            __syncthreads();  // groups, order and s_sum are read before they are rewritten
        }
    }
    if (threadIdx.x == 0) {
        const double mean = __dmul_rn(__ddiv_rn(S, (double)g.length), (double)mul);
        segs[blockIdx.x].mean = mean;
        R.split[g.node] = mean;
    }
}

// Tiles of kTreeTile slots: tile t covers slots [tile_off[t], +kTreeTile) of
// segment tile_seg[t]. A warp holds kTileRounds x 32 consecutive slots, whose
// coordinates are all loaded before any is tested: one block barrier per tile,
// where a loop over 256-slot rounds paid two and a load latency for each (the
// swaps took 230 us per level at 256^3 and 28 us at any small size).
constexpr int kTileRounds = kTreeTile / kTreeThreads;

struct TileFlags {
    unsigned small[kTileRounds];  // round r's lanes whose slot is not above the mean
    int first;                    // this lane's slot in round 0 (relative to the segment)
    int before, total;            // slots not above the mean: in the warps before this one; in the tile
};

__device__ __forceinline__ TileFlags tree_tile_flags(const double *c, double mean, int off, int end, int *warp_tot) {
    TileFlags f;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    f.first = off + w * (32 * kTileRounds) + lane;
    double v[kTileRounds];
#pragma unroll
    for (int r = 0; r < kTileRounds; ++r) v[r] = f.first + 32 * r < end ? c[f.first + 32 * r] : 0.0;
    int cnt = 0;
#pragma unroll
    for (int r = 0; r < kTileRounds; ++r) {
        f.small[r] = __ballot_sync(0xffffffffu, f.first + 32 * r < end && !(v[r] > mean));
        cnt += __popc(f.small[r]);
    }
    if (lane == 0) warp_tot[w] = cnt;
    __syncthreads();
    f.before = f.total = 0;
#pragma unroll
    for (int q = 0; q < kTreeThreads / 32; ++q) {
        if (q < w) f.before += warp_tot[q];
        f.total += warp_tot[q];
    }
    return f;
}

// Counts the tile's slots not above the mean.
__global__ void __launch_bounds__(kTreeThreads)
tree_tile_count_kernel(const TreeSeg *__restrict__ segs, const TreeLevels *__restrict__ lv, int level,
                       const int *__restrict__ tile_seg, const int *__restrict__ tile_off, TreeParts P,
                       int *__restrict__ tile_small) {
    __shared__ int warp_tot[kTreeThreads / 32];
    if ((int)blockIdx.x >= lv->ntile[level]) return;
    const TreeSeg g = segs[tile_seg[blockIdx.x]];
    const int off = tile_off[blockIdx.x];
    const double *c = (g.axis == 0 ? P.x : (g.axis == 1 ? P.y : P.z)) + g.ipart;
    const TileFlags f = tree_tile_flags(c, g.mean, off, min(g.length, off + kTreeTile), warp_tot);
    if (threadIdx.x == 0) tile_small[blockIdx.x] = f.total;
}

// The swapped slots not above the mean: map[nsmall + q] = the slot of the
// (q+1)-th particle not above the mean counted from the right among the
// slots [nsmall, length) of the segment (relative slots). tile_pre[t] = slots
// not above the mean before tile t within its segment.
__global__ void __launch_bounds__(kTreeThreads)
tree_tile_map_kernel(const TreeSeg *__restrict__ segs, const TreeLevels *__restrict__ lv, int level,
                     const int *__restrict__ tile_seg, const int *__restrict__ tile_off,
                     const int *__restrict__ tile_pre, TreeParts P, int *__restrict__ map) {
    __shared__ int warp_tot[kTreeThreads / 32];
    if ((int)blockIdx.x >= lv->ntile[level]) return;
    const TreeSeg g = segs[tile_seg[blockIdx.x]];
    const int off = tile_off[blockIdx.x];
    const int end = min(g.length, off + kTreeTile);
    if (end <= g.nsmall) return;  // the whole tile lies in the left part (block-uniform)
    const double *c = (g.axis == 0 ? P.x : (g.axis == 1 ? P.y : P.z)) + g.ipart;
    const TileFlags f = tree_tile_flags(c, g.mean, off, end, warp_tot);
    const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
    int before = tile_pre[blockIdx.x] + f.before;
#pragma unroll
    for (int k = 0; k < kTileRounds; ++k) {
        const int r = f.first + 32 * k;
        const bool small = f.small[k] >> (threadIdx.x & 31) & 1u;
        if (small && r >= g.nsmall)
            map[g.ipart + g.nsmall + (g.nsmall - (before + __popc(f.small[k] & lt)) - 1)] = r;
        before += __popc(f.small[k]);
    }
}

// The swaps: the particle above the mean at slot r < nsmall, the (q+1)-th
// such from the left (q = r minus the slots not above the mean before r),
// with the slot map[nsmall + q]. Only the thread of slot r touches r and its
// partner; flags are read in [0, nsmall) only, which no other thread writes.
__global__ void __launch_bounds__(kTreeThreads)
tree_tile_swap_kernel(const TreeSeg *__restrict__ segs, const TreeLevels *__restrict__ lv, int level,
                      const int *__restrict__ tile_seg, const int *__restrict__ tile_off,
                      const int *__restrict__ tile_pre, TreeParts P, const int *__restrict__ map) {
    __shared__ int warp_tot[kTreeThreads / 32];
    if ((int)blockIdx.x >= lv->ntile[level]) return;
    const TreeSeg g = segs[tile_seg[blockIdx.x]];
    const int off = tile_off[blockIdx.x];
    const int end = min(min(g.length, off + kTreeTile), g.nsmall);
    if (end <= off) return;  // the whole tile lies in the right part (block-uniform)
    const double *c = (g.axis == 0 ? P.x : (g.axis == 1 ? P.y : P.z)) + g.ipart;
    const TileFlags f = tree_tile_flags(c, g.mean, off, end, warp_tot);
    const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
    int before = tile_pre[blockIdx.x] + f.before;
    int to[kTileRounds];  // the partner's slot, -1: stays
#pragma unroll
    for (int k = 0; k < kTileRounds; ++k) {
        const int r = f.first + 32 * k;
        const bool big = r < end && !(f.small[k] >> (threadIdx.x & 31) & 1u);
        to[k] = big ? map[g.ipart + g.nsmall + (r - (before + __popc(f.small[k] & lt)))] : -1;
        before += __popc(f.small[k]);
    }
    // four swaps' loads at a time, then their stores
#pragma unroll
    for (int k0 = 0; k0 < kTileRounds; k0 += 4) {
        double a[4][3], b[4][3];
        int ia[4], ib[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (to[k0 + k] < 0) continue;
            const int i = g.ipart + f.first + 32 * (k0 + k), j = g.ipart + to[k0 + k];
            a[k][0] = P.x[i]; a[k][1] = P.y[i]; a[k][2] = P.z[i]; ia[k] = P.id[i];
            b[k][0] = P.x[j]; b[k][1] = P.y[j]; b[k][2] = P.z[j]; ib[k] = P.id[j];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (to[k0 + k] < 0) continue;
            const int i = g.ipart + f.first + 32 * (k0 + k), j = g.ipart + to[k0 + k];
            P.x[i] = b[k][0]; P.y[i] = b[k][1]; P.z[i] = b[k][2]; P.id[i] = ib[k];
            P.x[j] = a[k][0]; P.y[j] = a[k][1]; P.z[j] = a[k][2]; P.id[j] = ia[k];
        }
    }
}

// ---------------------------------------------------- subtree per block ---

// A subtree to build in one block: slots, axis of its root, depth of its
// root, and where its root's code goes (son[2 * parent + side]).
struct TreeTask {
    int ipart, length, axis, depth, parent, side;
};

// The root as the first level (one segment over all tiles), or as the one
// subtree of a tree small enough for a block.
__global__ void __launch_bounds__(kTreeThreads)
tree_first_level_kernel(int n, TreeSeg *segs, int *__restrict__ tile_seg, int *__restrict__ tile_off, TreeTask *tasks,
                        TreeLevels *lv, TreeRec R) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, nt = (n + kTreeTile - 1) / kTreeTile;
    if (n > kTreeSmall && t < nt) {
        tile_seg[t] = 0;
        tile_off[t] = t * kTreeTile;
    }
    if (t > 0) return;
    if (n <= kTreeSmall) {
        tasks[0] = TreeTask{0, n, 0, 0, -1, 0};
        lv->ntask = 1;
        return;
    }
    segs[0] = TreeSeg{0, n, 0, 0, 0.0, 0, 0, 0, 0};
    lv->nseg[0] = 1;
    lv->ntile[0] = nt;
    R.depth[0] = 0;
    R.counters[0] = 1;
}

constexpr int kTreeLevelThreads = 1024;

// Exclusive prefix of v over a block of kTreeLevelThreads, and the total.
__device__ __forceinline__ int tree_level_scan(int v, int *warp_tot, int &total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    int t = warp_tot[lane];  // 32 warps
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, t, off);
        if (lane >= off) t += y;
    }
    total = __shfl_sync(0xffffffffu, t, 31);
    const int before = w > 0 ? __shfl_sync(0xffffffffu, t, w - 1) : 0;
    __syncthreads();  // warp_tot is rewritten by the next scan
    return before + x - v;
}

// After a level's tile counts, one block: the counts before each tile within its
// segment, every segment's split, its children (leaves, subtrees for one block,
// or the next level's segments and tiles) and the next level's counts.
__global__ void __launch_bounds__(kTreeLevelThreads)
tree_level_kernel(TreeSeg *segs, const int *__restrict__ tile_seg, const int *__restrict__ tile_small, int *tile_pre,
                  TreeSeg *next, int *__restrict__ next_tile_seg, int *__restrict__ next_tile_off, TreeTask *tasks,
                  TreeLevels *lv, int level, int maxleaf, int seg_cap, int task_cap, TreeRec R) {
    __shared__ int warp_tot[32];
    __shared__ int s_next, s_task, s_node, s_leaf;
    const int nseg = lv->nseg[level], ntile = lv->ntile[level];
    if (nseg == 0) return;
    if (threadIdx.x == 0) {
        s_next = 0;
        s_task = lv->ntask;
        s_node = R.counters[0];
        s_leaf = R.counters[1];
    }
    int carry = 0;
    for (int b = 0; b < ntile; b += kTreeLevelThreads) {
        const int t = b + threadIdx.x;
        int total;
        const int ex = tree_level_scan(t < ntile ? tile_small[t] : 0, warp_tot, total);
        if (t < ntile) tile_pre[t] = carry + ex;
        carry += total;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < nseg; q += kTreeLevelThreads) {
        TreeSeg g = segs[q];
        const int t1 = g.tile0 + (g.length + kTreeTile - 1) / kTreeTile;
        g.before = tile_pre[g.tile0];
        g.nsmall = (t1 < ntile ? tile_pre[t1] : carry) - g.before;
        g.nbig = g.length - g.nsmall;
        segs[q] = g;
        const int left = g.nbig == 0 ? g.length - 1 : g.nsmall;
        for (int c = 0; c < 2; ++c) {
            const int np = c ? g.length - left : left, ip = c ? g.ipart + left : g.ipart, axis = (g.axis + 1) % 3;
            int code = -1;
            if (np <= maxleaf) {
                const int l = atomicAdd(&s_leaf, 1);
                if (l < R.leaf_cap) {
                    R.lipart[l] = ip;
                    R.lnpart[l] = np;
                    code = 2 * l;
                } else {
                    atomicOr(&R.counters[2], TB_LEAF_CAP);
                }
            } else if (np <= kTreeSmall) {
                const int k = atomicAdd(&s_task, 1);
                if (k < task_cap) tasks[k] = TreeTask{ip, np, axis, level + 1, g.node, c};
                else atomicOr(&R.counters[2], TB_NODE_CAP);
                continue;  // the subtree's block records its root
            } else {
                const int k = atomicAdd(&s_node, 1), j = atomicAdd(&s_next, 1);
                if (k < R.node_cap && j < seg_cap) {
                    R.depth[k] = level + 1;
                    next[j] = TreeSeg{ip, np, axis, k, 0.0, 0, 0, 0, 0};
                    code = 2 * k + 1;
                } else {
                    atomicOr(&R.counters[2], TB_NODE_CAP);
                }
            }
            R.son[2 * g.node + c] = code;
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < ntile; t += kTreeLevelThreads) tile_pre[t] -= segs[tile_seg[t]].before;
    const int nnext = min(s_next, seg_cap);
    carry = 0;
    for (int b = 0; b < nnext; b += kTreeLevelThreads) {
        const int q = b + threadIdx.x;
        int total;
        const int ex = tree_level_scan(q < nnext ? (next[q].length + kTreeTile - 1) / kTreeTile : 0, warp_tot, total);
        if (q < nnext) next[q].tile0 = carry + ex;
        carry += total;
    }
    __syncthreads();
    for (int q = threadIdx.x >> 5; q < nnext; q += kTreeLevelThreads / 32) {
        const int t0 = next[q].tile0, nt = (next[q].length + kTreeTile - 1) / kTreeTile;
        for (int k = threadIdx.x & 31; k < nt; k += 32) {
            next_tile_seg[t0 + k] = q;
            next_tile_off[t0 + k] = k * kTreeTile;
        }
    }
    if (threadIdx.x == 0) {
        lv->nseg[level + 1] = nnext;
        lv->ntile[level + 1] = carry;
        lv->ntask = min(s_task, task_cap);
        R.counters[0] = min(s_node, R.node_cap);
        R.counters[1] = min(s_leaf, R.leaf_cap);
    }
}

struct SmallItem {
    int span;    // slot offset in the task (low 16 bits) and length (high 16 bits)
    int parent;  // build id of the parent node
    short depth;
    char axis, side;
};

constexpr int kTreeSmallThreads = 512;
// Nodes of one depth hold more than one particle each; they have two children.
constexpr int kTreeLevelItems = kTreeSmall / 2;
constexpr int kTreeLevelLeaves = kTreeSmall;

// A leaf made at the current depth: its slots in the task (as SmallItem::span)
// and its place, 2 x (index of the parent within the depth) + side.
struct SmallLeaf {
    int span, place;
};

// Dynamic shared memory of tree_small_kernel.
constexpr size_t kTreeSmallSmem = (size_t)kTreeSmall * (3 * sizeof(double) + sizeof(int) + sizeof(short)) +
                                  2 * (size_t)kTreeLevelItems * sizeof(SmallItem) +
                                  (size_t)kTreeLevelLeaves * sizeof(SmallLeaf);

// One block builds a whole subtree of at most kTreeSmall particles in shared
// memory, depth after depth, one warp per node, then writes the permuted
// particles back. Warps split their nodes with ballots and no block barrier,
// and the build ids of a depth's nodes and leaves (names only: the pre-order
// numbering is made afterwards) are taken with one atomic each. A block that
// split one node after another waited for each one's serial sum, ten barriers
// and three atomics on counters that all blocks share: 7.6 ms at 256^3.
__global__ void __launch_bounds__(kTreeSmallThreads)
tree_small_kernel(const TreeTask *__restrict__ tasks, TreeParts P, TreeRec R, int maxleaf) {
    extern __shared__ double tsm[];
    double *sx = tsm, *sy = sx + kTreeSmall, *sz = sy + kTreeSmall;
    int *sid = reinterpret_cast<int *>(sz + kTreeSmall);
    SmallItem *items = reinterpret_cast<SmallItem *>(sid + kTreeSmall);  // this depth's, then the next one's
    SmallLeaf *leaves = reinterpret_cast<SmallLeaf *>(items + 2 * kTreeLevelItems);
    short *smap = reinterpret_cast<short *>(leaves + kTreeLevelLeaves);
    __shared__ int s_count[2];  // items of each half
    __shared__ int s_nleaf, s_node0, s_leaf0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const TreeTask T = tasks[blockIdx.x];
    for (int i = threadIdx.x; i < T.length; i += blockDim.x) {
        sx[i] = P.x[T.ipart + i];
        sy[i] = P.y[T.ipart + i];
        sz[i] = P.z[T.ipart + i];
        sid[i] = P.id[T.ipart + i];
    }
    if (threadIdx.x == 0) {
        SmallItem it;
        it.span = T.length << 16;
        it.parent = T.parent;
        it.depth = (short)T.depth;
        it.axis = (char)T.axis;
        it.side = (char)T.side;
        items[0] = it;
        s_count[0] = 1;
        s_count[1] = 0;
        s_nleaf = 0;
        s_node0 = atomicAdd(&R.counters[0], 1);
    }
    __syncthreads();
    for (int half = 0;; half ^= 1) {
        const int count = s_count[half], node0 = s_node0;
        if (node0 + count > R.node_cap) {  // block-uniform
            if (threadIdx.x == 0) atomicOr(&R.counters[2], TB_NODE_CAP);
            break;
        }
        for (int q = w; q < count; q += kTreeSmallThreads / 32) {
            const SmallItem it = items[half * kTreeLevelItems + q];
            const int node = node0 + q;
            const int base = it.span & 0xffff, len = it.span >> 16, axis = it.axis;
            double *c = sx + axis * kTreeSmall + base;
            double split = 0.0;
            int nleft = 0;
            if (len == 2) {
                nleft = 1;
                split = __dmul_rn(0.5, __dadd_rn(c[0], c[1]));
                const bool swap = c[0] > c[1];
                __syncwarp();
                if (lane == 0 && swap) {
                    TreeParts Q{sx, sy, sz, sid};
                    tree_swap(Q, base, base + 1);
                }
            } else if (len > 2) {
                const double S = len <= 512 ? mean_chain(c, len, 0.0) : mean_warp(c, len, 0.0);
                const double mean = __ddiv_rn(S, (double)len);
                split = mean;
                int nsmall = 0;  // slots not above the mean
                for (int r0 = 0; r0 < len; r0 += 32)
                    nsmall += __popc(__ballot_sync(0xffffffffu, r0 + lane < len && !(c[r0 + lane] > mean)));
                // the swapped slots by rank: particles above the mean among the
                // first nsmall slots from the left, the others' from the right
                short *map = smap + base;
                int before = 0, kpairs = 0;
                for (int r0 = 0; r0 < len; r0 += 32) {
                    const int r = r0 + lane;
                    const bool in = r < len;
                    const bool small = in && !(c[r] > mean);
                    const unsigned m = __ballot_sync(0xffffffffu, small);
                    const int sb = before + __popc(m & lt);
                    if (in && !small && r < nsmall) map[r - sb] = (short)r;
                    else if (small && r >= nsmall) map[nsmall + (nsmall - sb - 1)] = (short)r;
                    const unsigned left = nsmall - r0 >= 32 ? 0xffffffffu : (nsmall > r0 ? (1u << (nsmall - r0)) - 1u : 0u);
                    kpairs += __popc(left & ~m);  // nsmall <= len: these lanes hold particles
                    before += __popc(m);
                }
                __syncwarp();
                TreeParts Q{sx, sy, sz, sid};
                for (int k = lane; k < kpairs; k += 32) tree_swap(Q, base + map[k], base + map[nsmall + k]);
                nleft = (len - nsmall) == 0 ? len - 1 : nsmall;
            }
            if (lane == 0) {
                R.split[node] = split;
                R.depth[node] = it.depth;
                if (it.parent >= 0) R.son[2 * it.parent + it.side] = 2 * node + 1;
            }
            if (lane < 2) {  // this lane's child
                const int np = lane ? len - nleft : nleft, ip = lane ? base + nleft : base;
                if (np <= maxleaf) {
                    SmallLeaf lf;
                    lf.span = ip | (np << 16);
                    lf.place = 2 * q + lane;
                    leaves[atomicAdd(&s_nleaf, 1)] = lf;
                } else {
                    SmallItem ch;
                    ch.span = ip | (np << 16);
                    ch.parent = node;
                    ch.depth = (short)(it.depth + 1);
                    ch.axis = (char)((axis + 1) % 3);
                    ch.side = (char)lane;
                    items[(half ^ 1) * kTreeLevelItems + atomicAdd(&s_count[half ^ 1], 1)] = ch;
                }
            }
        }
        __syncthreads();  // this depth is split; its leaves and the next depth's items are written
        const int nleaf = s_nleaf, more = s_count[half ^ 1];
        if (threadIdx.x == 0) {
            if (nleaf) s_leaf0 = atomicAdd(&R.counters[1], nleaf);
            if (more) s_node0 = atomicAdd(&R.counters[0], more);
        }
        __syncthreads();
        if (threadIdx.x == 0) s_nleaf = s_count[half] = 0;
        if (nleaf && s_leaf0 + nleaf > R.leaf_cap) {  // block-uniform
            if (threadIdx.x == 0) atomicOr(&R.counters[2], TB_LEAF_CAP);
            break;
        }
        for (int i = threadIdx.x; i < nleaf; i += blockDim.x) {
            const SmallLeaf lf = leaves[i];
            const int l = s_leaf0 + i;
            R.lipart[l] = T.ipart + (lf.span & 0xffff);
            R.lnpart[l] = lf.span >> 16;
            R.son[2 * (node0 + (lf.place >> 1)) + (lf.place & 1)] = 2 * l;
        }
        if (!more) break;
        __syncthreads();  // the leaves are read, the counts are reset
    }
    __syncthreads();
    for (int i = threadIdx.x; i < T.length; i += blockDim.x) {
        P.x[T.ipart + i] = sx[i];
        P.y[T.ipart + i] = sy[i];
        P.z[T.ipart + i] = sz[i];
        P.id[T.ipart + i] = sid[i];
    }
}

// ------------------------------------------------- numbering and boxes ---

// Three passes whatever the tree's depth (one launch per depth, twice, took 26 to
// 52 launches, a tenth of a small step).

// Each box's parent as 2 x node + side (-1: the root), nodes' arrival counts 0.
__global__ void tree_link_kernel(TreeRec R, int nnode, int nleaf, int *__restrict__ parent,
                                 int *__restrict__ lparent, int *__restrict__ arrived) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnode; k += gridDim.x * blockDim.x) {
        arrived[k] = 0;
        if (k == 0) parent[0] = -1;
        for (int n = 0; n < 2; ++n) {
            const int c = R.son[2 * k + n];
            if (c < 0 || c == 1 || ((c & 1) ? (c >> 1) >= nnode : (c >> 1) >= nleaf)) {  // a child never recorded
                atomicOr(&R.counters[2], TB_NUMBERING);
                continue;
            }
            if (c & 1) parent[c >> 1] = 2 * k + n;
            else lparent[c >> 1] = 2 * k + n;
        }
    }
}

// Subtree node and leaf counts: a thread per leaf climbs while it is the second
// of a node's two children to arrive.
__global__ void tree_count_kernel(TreeRec R, int nnode, int nleaf, const int *__restrict__ parent,
                                  const int *__restrict__ lparent, int *__restrict__ arrived) {
    if (R.counters[2] & TB_NUMBERING) return;
    for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < nleaf; l += gridDim.x * blockDim.x) {
        for (int p = lparent[l]; p >= 0;) {
            const int k = p >> 1;
            __threadfence();
            if (atomicAdd(&arrived[k], 1) == 0) break;
            __threadfence();
            int nn = 1, nl = 0;
            for (int n = 0; n < 2; ++n) {
                const int c = R.son[2 * k + n];
                nn += (c & 1) ? __ldcg(&R.nn[c >> 1]) : 0;
                nl += (c & 1) ? __ldcg(&R.nl[c >> 1]) : 1;
            }
            R.nn[k] = nn;
            R.nl[k] = nl;
            p = parent[k];
        }
    }
}

// Every node's pre-order id, first leaf and box from its path to the root, and
// the ids of its leaves (center_kdtree, src/fmm.c:273-327: an ancestor split on
// an axis bounds the box on the side it was left by, the nearest one counts).
__global__ void tree_order_kernel(TreeRec R, int nnode, const int *__restrict__ parent) {
    if (R.counters[2] & TB_NUMBERING) return;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnode; k += gridDim.x * blockDim.x) {
        double box[6];
        unsigned known = 0;
        int pre = 0, first = 0, steps = 0;
        for (int p = parent[k]; p >= 0; p = parent[p >> 1]) {
            if (++steps > nnode) break;
            const int a = p >> 1, right = p & 1;
            const int side = R.depth[a] % 3 + (right ? 0 : 3);  // left child: right[axis] = split
            if (!(known >> side & 1u)) {
                known |= 1u << side;
                const double split = R.split[a];
#pragma unroll
                for (int q = 0; q < 6; ++q)
                    if (q == side) box[q] = split;
            }
            pre += 1;
            if (right) {
                const int c = R.son[2 * a];
                pre += (c & 1) ? R.nn[c >> 1] : 0;
                first += (c & 1) ? R.nl[c >> 1] : 1;
            }
        }
        double root[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) root[q] = R.root[q];
#pragma unroll
        for (int q = 0; q < 6; ++q) R.box[6 * (size_t)k + q] = known >> q & 1u ? box[q] : root[q];
        R.pre[k] = pre;
        R.first[k] = first;
        const int c0 = R.son[2 * k], c1 = R.son[2 * k + 1];
        if (!(c0 & 1)) R.lid[c0 >> 1] = first;
        if (!(c1 & 1)) R.lid[c1 >> 1] = first + ((c0 & 1) ? R.nl[c0 >> 1] : 1);
        if (steps > nnode) atomicOr(&R.counters[2], TB_NUMBERING);
    }
}

// Output tables in pre-order: node child codes in final ids, first leaves,
// centres and widths (AoS); leaf ranges, centres and widths (from the
// parent's box, the split axis cut at the split).
__global__ void tree_emit_kernel(TreeRec R, int nnode, int nleaf, int *__restrict__ son,
                                 int *__restrict__ node_first, double *__restrict__ node_center,
                                 double *__restrict__ node_width, int *__restrict__ leaf_ipart,
                                 int *__restrict__ leaf_npart, double *__restrict__ leaf_center,
                                 double *__restrict__ leaf_width) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnode; k += gridDim.x * blockDim.x) {
        const int pre = R.pre[k];
        if ((unsigned)pre >= (unsigned)nnode) {
            atomicOr(&R.counters[2], TB_NUMBERING);
            continue;
        }
        const int axis = R.depth[k] % 3;
        const double *bx = R.box + 6 * (size_t)k;
        double w[3], ctr[3];
        for (int q = 0; q < 3; ++q) {
            w[q] = __dsub_rn(bx[3 + q], bx[q]);
            ctr[q] = __dmul_rn(0.5, __dadd_rn(bx[3 + q], bx[q]));
            node_center[3 * (size_t)pre + q] = ctr[q];
            node_width[3 * (size_t)pre + q] = w[q];
        }
        node_first[pre] = R.first[k];
        const double split = R.split[k];
        for (int n = 0; n < 2; ++n) {
            const int c = R.son[2 * k + n];
            if (c & 1) {
                son[2 * pre + n] = 2 * R.pre[c >> 1] + 1;
            } else {
                const int l = c >> 1, id = R.lid[l];
                if ((unsigned)l >= (unsigned)R.leaf_cap || (unsigned)id >= (unsigned)nleaf) {
                    atomicOr(&R.counters[2], TB_NUMBERING);
                    continue;
                }
                son[2 * pre + n] = 2 * id;
                leaf_ipart[id] = R.lipart[l];
                leaf_npart[id] = R.lnpart[l];
                for (int q = 0; q < 3; ++q) {
                    leaf_width[3 * (size_t)id + q] = w[q];
                    leaf_center[3 * (size_t)id + q] = ctr[q];
                }
                if (n == 0) {
                    leaf_width[3 * (size_t)id + axis] = __dsub_rn(split, bx[axis]);
                    leaf_center[3 * (size_t)id + axis] = __dmul_rn(0.5, __dadd_rn(bx[axis], split));
                } else {
                    leaf_width[3 * (size_t)id + axis] = __dsub_rn(bx[3 + axis], split);
                    leaf_center[3 * (size_t)id + axis] = __dmul_rn(0.5, __dadd_rn(bx[3 + axis], split));
                }
            }
        }
    }
}

// leaf.active (src/fmm.c:1226-1236): 0 when the leaf holds a local particle
// (tag 1), else -1; one warp per leaf.
__global__ void tree_active_kernel(const int *__restrict__ leaf_ipart, const int *__restrict__ leaf_npart,
                                   int nleaf, const int *__restrict__ id, const int *__restrict__ tag,
                                   int *__restrict__ active) {
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < nleaf; l += nw) {
        const int ip = leaf_ipart[l], np = leaf_npart[l];
        bool any = false;
        for (int q = lane; q < np; q += 32) any = any || (tag ? tag[id[ip + q]] == 1 : true);
        any = __any_sync(0xffffffffu, any);
        if (lane == 0) active[l] = any ? 0 : -1;
    }
}

// A per-particle SoA result in tree order back to input order:
// out[d * n + perm[i]] = in[d * n + i].
__global__ void tree_unpermute_kernel(const double *__restrict__ in, const int *__restrict__ perm, int n,
                                      double *__restrict__ out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int j = perm[i];
        if ((unsigned)j >= (unsigned)n) continue;
        out[j] = in[i];
        out[(size_t)n + j] = in[(size_t)n + i];
        out[2 * (size_t)n + j] = in[2 * (size_t)n + i];
    }
}

// Positions in tree order (SoA) from the work arrays.
__global__ void tree_pos_out_kernel(TreeParts P, int n, double *__restrict__ pos) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        pos[i] = P.x[i];
        pos[(size_t)n + i] = P.y[i];
        pos[2 * (size_t)n + i] = P.z[i];
    }
}

}  // namespace p2p
