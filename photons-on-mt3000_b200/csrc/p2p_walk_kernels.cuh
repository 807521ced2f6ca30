// Device interaction-list walks on the kd-tree: the P2P lists of PhotoNs'
// dual-tree walk (walk_task_p2p, src/fmm.c:656-792) straight into CSR rows, and
// the M2L tasks of its walk_task_m2l (src/fmm.c:812-957), both with the
// LONGSHORT acceptance test of src/fmm.c:409-479.
//
// The serial walks recurse over box pairs (A, B) from (root, root): a pair of
// boxes is dropped or accepted, or the larger box is opened; (A, A) opens on
// both sides. How a pair goes on depends on the pair alone. So the sink side
// is taken depth by depth (walk_level_kernel, one launch per depth, one warp
// per box A): A receives its parent's list of undecided boxes B, in leaf
// order; opens those B that are to be opened until each is dropped, accepted,
// kept (A is to be opened: both children of A receive the kept list) or, for
// two leaves, emitted. A pair is tested once for all the leaves below A, where
// a walk per sink leaf tests it again for each of them (51 ms at 256^3), and A's
// box is in registers, so a test reads one 32-byte record: the test is bounded
// in FP32 (p2p_walk_test.h) and repeated in FP64 only where the bound does not
// decide. A dependent FP64 operation takes about 16 cycles and a test has some
// 25 in a row, so in FP64 the warps mostly waited for it.
//
// Order: the serial walk emits a sink's sources in pre-order of the source
// side, i.e. in increasing leaf id (leaves are numbered in pre-order and
// son[0]'s subtree is walked before son[1]'s). A warp keeps the boxes in that
// order: it takes up to 32 of the first ones (from a stack of opened boxes with
// the first on top, then from the input list), writes out the decided ones
// that precede every box still to be opened, and puts the rest back with
// opened boxes replaced by their children. Rows come out sorted and equal those
// the list path builds, entry for entry, with no sort (20 ms at 256^3).
//
// A tree much deeper than a balanced one, or one whose opened boxes outgrow a
// warp's stack, is walked by sink leaf instead (walk_sink_kernel).
//
// Lists are chains of chunks of a pool, as their lengths are not known before
// they are made. The acceptance arithmetic is written with explicitly rounded
// FP64 operations (no contraction), the ISO C evaluation of the reference's
// code.
#pragma once

#include <algorithm>

#include "p2p_device_common.cuh"
#include "p2p_walk_test.h"

namespace p2p {

// The tree as the walks' other users see it.
struct WalkArgs {
    int nnode, nleaf;
    const int *son;           // 2 * nnode encoded children: leaf l -> 2l, node k -> 2k + 1
    const int *node_first;    // nnode: smallest leaf id in the node's subtree
    const int *leaf_active;   // nleaf: >= 0 for leaves holding a local particle (sinks)
    const double *node_center, *node_width;  // 3 * nnode
    const double *leaf_center, *leaf_width;  // 3 * nleaf
    double cutoff, open_angle;
};

enum : int {
    ST_WALK_STACK = 4,    // a warp's opened boxes exceeded its stack (the host walks by sink leaf, or enlarges that walk's)
    ST_WALK_ROW = 8,      // a row came out longer than it was counted (or, in the FMM, offsets out of order)
    ST_WALK_TREE = 16,    // a child code outside the tree, leaves not in pre-order, or a walk longer than any tree allows
    ST_WALK_LISTS = 32,   // the pool of undecided lists is full (the host enlarges it and repeats the walk)
    ST_WALK_OUT = 64,     // the pool of rows (or M2L tasks) is full
    ST_WALK_LONG = 128,   // a walk by sink leaf met more pairs than it may
};

__device__ __forceinline__ const double *walk_center(const WalkArgs &w, int c) {
    return (c & 1) ? w.node_center + 3 * (size_t)(c >> 1) : w.leaf_center + 3 * (size_t)(c >> 1);
}

__device__ __forceinline__ bool walk_valid(const WalkArgs &w, int c) {
    return c >= 0 && ((c & 1) ? (c >> 1) < w.nnode : (c >> 1) < w.nleaf);
}

// The child of node code A whose subtree holds leaf L (pre-order leaf ids:
// son[0]'s leaves precede son[1]'s); -1 for a child code outside the tree.
__device__ __forceinline__ int walk_child_toward(const WalkArgs &w, int A, int L) {
    const int k = A >> 1;
    const int s1 = w.son[2 * k + 1];
    if (!walk_valid(w, s1)) return -1;
    const int f1 = (s1 & 1) ? w.node_first[s1 >> 1] : (s1 >> 1);
    return L < f1 ? w.son[2 * k] : s1;
}

// acceptance (LONGSHORT), src/fmm.c:409-479: 0 open, 1 accept (M2L), -1 drop.
__device__ __forceinline__ int walk_acceptance(const WalkBox &i, const WalkBox &j, double cutoff, double open_angle) {
    double dist[3], w[3], mn[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        dist[d] = __dsub_rn(i.c[d], j.c[d]);
        w[d] = __dmul_rn(__dadd_rn(i.w[d], j.w[d]), 0.5);
    }
    const double dd2 = __dadd_rn(__dadd_rn(__dmul_rn(dist[0], dist[0]), __dmul_rn(dist[1], dist[1])),
                                 __dmul_rn(dist[2], dist[2]));
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double m = dist[d] < 0.0 ? -dist[d] : dist[d];
        m = __dsub_rn(m, w[d]);
        mn[d] = m <= 0.0 ? 0.0 : m;
    }
    if (__dadd_rn(__dadd_rn(mn[0], mn[1]), mn[2]) < 1.0e-15) return 0;
    const double dm2 = __dadd_rn(__dadd_rn(__dmul_rn(mn[0], mn[0]), __dmul_rn(mn[1], mn[1])),
                                 __dmul_rn(mn[2], mn[2]));
    if (dm2 > __dmul_rn(cutoff, cutoff)) return -1;
    double wmax = w[0];
    if (w[1] > wmax) wmax = w[1];
    if (w[2] > wmax) wmax = w[2];
    wmax = fabs(wmax);
    wmax = __dmul_rn(wmax, 2.0);
    if (__dmul_rn(wmax, wmax) < __dmul_rn(__dmul_rn(open_angle, open_angle), dd2)) return 1;
    return 0;
}

constexpr int kWalkWarps = 4;      // boxes in flight per block
constexpr int kWalkStack = 1024;   // opened boxes per warp (shared memory)
constexpr int kWalkChunk = 64;     // ids per chunk of a list of undecided boxes or of a row
constexpr int kWalkTaskChunk = 16; // ids per chunk of a sink's M2L tasks (about 10 at open angle 0.4)
constexpr int kWalkGrab = 16;      // chunks a warp takes from a pool at a time
constexpr int kWalkLevels = 96;    // most depths of a walk by depth
// Depths beyond walk_first_depths before a tree is walked by sink leaf. Clustered
// particles need none; 20^3 particles, 48 of them at one point, take 1.3 ms by depth
// and 0.6 by sink leaf, 300 of them 3.5 ms by sink leaf after what this many depths took.
constexpr int kWalkExtraDepths = 12;

// A sink-side box to be walked at a depth.
struct WalkItem {
    int code, parent;  // the box, and the node it is a child of (-1: the root)
    int lo, hi;        // leaf ids of its subtree [lo, hi) (P2P walk)
    int head, len;     // its parent's undecided boxes
};

struct WalkPool {
    int *ids;   // cap chunks
    int *next;  // cap: the chunk after this one in its list
    int cap;
};

// Device counters of one walk.
struct WalkCtrl {
    int items[kWalkLevels + 1];   // boxes of each depth
    int lists[kWalkLevels + 1];   // chunks taken by each depth's undecided lists
    int taken[kWalkLevels + 1];   // boxes of each depth taken by warps beyond their first
    int out;                      // chunks taken by rows or tasks
    int status;                   // ST_WALK_* bits of this walk
    unsigned long long ntask;     // M2L tasks
};

enum WalkMode {
    WALK_ROWS = 0,   // P2P rows into the pool of chunks
    WALK_COUNT = 1,  // P2P row lengths only
    WALK_FILL = 2,   // P2P rows into row_src[row_off[L] ...]
    WALK_M2L = 3,    // M2L tasks of every box into the pool of chunks
};

struct WalkRun {
    int nnode, nleaf;
    const WalkBox *box;        // box code c at index c
    const WalkBox32 *box32;
    float cut2, th2;           // squares of cutoff and open angle
    const int64_t *active;     // nleaf + 1: active leaves before each leaf (P2P)
    const int *node_first;
    double cutoff, open_angle;
    WalkItem *items[2];        // this depth's boxes, the next one's
    WalkPool lists[2];         // the lists they receive, those they leave
    WalkPool out;
    int *out_head, *out_len;   // per leaf (P2P) or per sink, leaves then nodes (M2L)
    const int64_t *row_off;    // WALK_FILL
    int *row_src;
    WalkCtrl *ctrl;
};

// The boxes' records, the leaves' active flags and the first depth (the root
// with itself as its one undecided box).
template <bool M2L>
__global__ void __launch_bounds__(256)
walk_pack_kernel(const WalkArgs w, WalkBox *__restrict__ box, WalkBox32 *__restrict__ box32,
                 int *__restrict__ flag, WalkItem *items,
                 int *lists, WalkCtrl *ctrl) {
    const int n = w.nnode + w.nleaf;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const bool leaf = i < w.nleaf;
        const int k = leaf ? i : i - w.nleaf;
        const double *c = leaf ? w.leaf_center + 3 * (size_t)k : w.node_center + 3 * (size_t)k;
        const double *v = leaf ? w.leaf_width + 3 * (size_t)k : w.node_width + 3 * (size_t)k;
        WalkBox b;
        WalkBox32 f;
        for (int d = 0; d < 3; ++d) {
            b.c[d] = c[d];
            b.w[d] = v[d];
            f.c[d] = (float)c[d];
            f.w[d] = (float)v[d];
        }
        b.sum = __dadd_rn(__dadd_rn(v[0], v[1]), v[2]);
        b.pad = 0.0;
        f.son[0] = leaf ? -1 : w.son[2 * k];
        f.son[1] = leaf ? -1 : w.son[2 * k + 1];
        const int code = leaf ? 2 * k : 2 * k + 1;
        box[code] = b;
        box32[code] = f;
        if (!M2L && leaf) flag[k] = w.leaf_active[k] >= 0 ? 1 : 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        items[0] = WalkItem{1, -1, 0, w.nleaf, 0, 1};
        lists[0] = 1;  // the root's code
        ctrl->items[0] = 1;
    }
}

__device__ __forceinline__ WalkBox32 walk_load(const WalkBox32 *p) {
    WalkBox32 b;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(b.c[0]), "=f"(b.c[1]), "=f"(b.c[2]), "=f"(b.w[0]), "=f"(b.w[1]), "=f"(b.w[2]),
          "=f"(reinterpret_cast<float &>(b.son[0])), "=f"(reinterpret_cast<float &>(b.son[1]))
        : "l"(__cvta_generic_to_global(p)));
    return b;
}

// The exact test where the bound does not decide: the same outcomes.
static __device__ __noinline__ int walk_exact(const WalkBox *box, int A, int B, double cutoff, double open_angle) {
    const WalkBox a = box[A], b = box[B];
    const int t = walk_acceptance(a, b, cutoff, open_angle);
    if (t != 0) return t == 1 ? WALK_ACCEPT : WALK_DROP;
    return (A & 1) && (!(B & 1) || a.sum > b.sum) ? WALK_OPEN_A : WALK_OPEN_B;
}

// One warp's list being written: ids appended in order, CHUNK per chunk.
template <int CHUNK>
struct WalkWriter {
    int head, cur, n;  // first and current chunk, ids so far
    int base, left;    // chunks taken from the pool and not yet used (kept between lists)
    __device__ __forceinline__ void start() { n = 0; head = cur = -1; }
    // Appends the ids of the lanes in mask, in lane order; false when the pool is full.
    __device__ __forceinline__ bool append(unsigned mask, int id, const WalkPool &p, int *taken) {
        const int k = __popc(mask);
        if (k == 0) return true;
        const int lane = threadIdx.x & 31;
        const int off = n % CHUNK;
        int room = off ? CHUNK - off : 0;  // left in the current chunk
        const int rank = __popc(mask & ((1u << lane) - 1u));
        const bool mine = mask >> lane & 1u;
        if (mine && rank < room) p.ids[(size_t)cur * CHUNK + off + rank] = id;
        while (k > room) {  // at most once where CHUNK >= 32
            if (left == 0) {
                if (lane == 0) base = atomicAdd(taken, kWalkGrab);
                base = __shfl_sync(kFull, base, 0);
                left = kWalkGrab;
                if (base < 0 || base > p.cap - kWalkGrab) {
                    left = 0;
                    return false;
                }
            }
            const int c = base++;
            --left;
            if (cur < 0) head = c;
            else if (lane == 0) p.next[cur] = c;
            cur = c;
            if (mine && rank >= room && rank < room + CHUNK) p.ids[(size_t)c * CHUNK + rank - room] = id;
            room += CHUNK;
        }
        n += k;
        return true;
    }
};

template <int MODE>
__global__ void __launch_bounds__(kWalkWarps * 32, 8) walk_level_kernel(const WalkRun g, int level) {
    constexpr bool M2L = MODE == WALK_M2L;
    constexpr int OUT = M2L ? kWalkTaskChunk : kWalkChunk;
    __shared__ int stacks[kWalkWarps][kWalkStack];
    __shared__ WalkItem pushed[kWalkWarps][32];  // children for the next depth, written 31 or more at a time
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u, above = ~(lt | (1u << lane));
    const int count = g.ctrl->items[level];
    int i = blockIdx.x * kWalkWarps + wid;
    if (i >= count || g.ctrl->status) return;  // (a walk that failed is not continued)
    int *stk = stacks[wid];
    const WalkItem *in = g.items[level & 1];
    WalkItem *next_items = g.items[(level & 1) ^ 1];
    const WalkPool from = g.lists[level & 1], to = g.lists[(level & 1) ^ 1];
    WalkWriter<kWalkChunk> kept;
    WalkWriter<OUT> out;
    kept.base = kept.left = out.base = out.left = 0;
    int npushed = 0, fault = 0;
    unsigned long long ntask = 0;
    auto flush = [&]() {
        int at = 0;
        if (lane == 0) at = atomicAdd(&g.ctrl->items[level + 1], npushed);
        at = __shfl_sync(kFull, at, 0);
        // disjoint subtrees: at most nleaf boxes a depth in a well-formed tree
        if (at < 0 || at + npushed > g.nleaf) fault |= ST_WALK_TREE;
        else if (lane < npushed) next_items[at + lane] = pushed[wid][lane];
        npushed = 0;
        __syncwarp();
    };
    // lists differ by a factor of a hundred between voids and halos, so warps
    // take boxes as they get free, each one's next asked for before it is needed
    int after = 0;
    for (; i < count && !fault; i = gridDim.x * kWalkWarps + __shfl_sync(kFull, after, 0)) {
        if (lane == 0) after = atomicAdd(&g.ctrl->taken[level], 1);
        const WalkItem it = in[i];
        const int A = it.code;
        const bool a_leaf = !(A & 1);
        const WalkBox32 a = walk_load(g.box32 + A);
        const bool fill = MODE == WALK_FILL && a_leaf;
        const int64_t row = fill ? g.row_off[A >> 1] : 0;
        const int cap = fill ? (int)(g.row_off[(A >> 1) + 1] - row) : 0;
        int chunk = it.head, chunk_next = it.len > kWalkChunk ? from.next[it.head] : 0;
        int sp = 0, pos = 0, emitted = 0;
        kept.start();
        out.start();
        // a pair is met at most once: a longer walk means a malformed tree
        long long budget = 2LL * ((long long)g.nnode + g.nleaf) + 64;
        while (sp > 0 || pos < it.len) {
            // the first boxes: from the stack, then from the input
            const int ns = min(32, sp), ni = min(32 - ns, it.len - pos);
            int v = 0;
            if (lane < ns) {
                v = stk[sp - 1 - lane];
            } else if (lane < ns + ni) {
                const int o = (pos & (kWalkChunk - 1)) + lane - ns;
                v = o < kWalkChunk ? from.ids[(size_t)chunk * kWalkChunk + o]
                                   : from.ids[(size_t)chunk_next * kWalkChunk + o - kWalkChunk];
            }
            __syncwarp();  // the boxes are read before others are put in their places
            sp -= ns;
            if ((pos & (kWalkChunk - 1)) + ni >= kWalkChunk) {
                chunk = chunk_next;
                if (it.len - (pos + ni) > kWalkChunk - ((pos + ni) & (kWalkChunk - 1))) chunk_next = from.next[chunk];
            }
            pos += ni;
            budget -= ni;
            // 0 dropped, 1 decided (emitted or kept), 2 opened
            int cls = 0, c0 = -1, c1 = -1, B = v;
            bool task = false;
            if (lane < ns + ni) {
                if (v < 0) {  // decided before
                    B = ~v;
                    cls = 1;
                } else if (a_leaf && !(B & 1)) {
                    cls = M2L ? 0 : 1;
                } else if (A == B) {
                    cls = 1;
                } else {
                    const WalkBox32 b = walk_load(g.box32 + B);
                    if (B == it.parent) {  // (parent, parent) opened on both sides
                        cls = 2;
                    } else {
                        int t = walk_bound(a, b, !a_leaf, B & 1, g.cut2, g.th2);
                        if (t == WALK_UNDECIDED) t = walk_exact(g.box, A, B, g.cutoff, g.open_angle);
                        cls = t == WALK_OPEN_A ? 1 : (t == WALK_OPEN_B ? 2 : 0);
                        task = M2L && t == WALK_ACCEPT;
                    }
                    c0 = b.son[0];
                    c1 = b.son[1];
                }
            }
            int nc = 0;
            if (cls == 2) {
                const bool v0 = c0 >= 0 && ((c0 & 1) ? (c0 >> 1) < g.nnode : (c0 >> 1) < g.nleaf);
                const bool v1 = c1 >= 0 && ((c1 & 1) ? (c1 >> 1) < g.nnode : (c1 >> 1) < g.nleaf);
                // the M2L walk passes over absent children
                if ((!v0 && (!M2L || c0 >= 0)) || (!v1 && (!M2L || c1 >= 0))) fault = ST_WALK_TREE;
                if (!v0) c0 = c1;
                nc = (v0 ? 1 : 0) + (v1 ? 1 : 0);
            }
            const unsigned open = __ballot_sync(kFull, cls == 2);
            // written out: the lanes before the first opened box (M2L lists need no
            // order, only the same one on every run)
            const unsigned ready = M2L || !open ? kFull : (open & (0u - open)) - 1u;
            const unsigned done = __ballot_sync(kFull, cls == 1);
            if (M2L) {
                const unsigned tm = __ballot_sync(kFull, task);
                if (!out.append(tm, B, g.out, &g.ctrl->out)) fault |= ST_WALK_OUT;
                if (!a_leaf && !kept.append(done & ready, B, to, &g.ctrl->lists[level])) fault |= ST_WALK_LISTS;
            } else if (!a_leaf) {
                if (!kept.append(done & ready, B, to, &g.ctrl->lists[level])) fault |= ST_WALK_LISTS;
            } else {
                const unsigned m = done & ready;
                if (MODE == WALK_ROWS) {
                    if (!out.append(m, B >> 1, g.out, &g.ctrl->out)) fault |= ST_WALK_OUT;
                } else if (MODE == WALK_FILL && (m >> lane & 1u)) {
                    const int slot = emitted + __popc(m & lt);
                    if (slot < cap) g.row_src[row + slot] = B >> 1;
                    else fault |= ST_WALK_ROW;
                }
                emitted += __popc(m);
            }
            // the others back on the stack, the first on top
            const unsigned back = done & ~ready;
            const unsigned one = __ballot_sync(kFull, nc >= 1), two = __ballot_sync(kFull, nc == 2);
            const int total = __popc(back) + __popc(one) + __popc(two);
            if (sp + total > kWalkStack) {
                fault |= ST_WALK_STACK;
            } else {
                const int at = sp + __popc(back & above) + __popc(one & above) + __popc(two & above);
                if (back >> lane & 1u) stk[at] = ~B;
                if (nc == 1) stk[at] = c0;
                if (nc == 2) {
                    stk[at] = c1;
                    stk[at + 1] = c0;
                }
                sp += total;
            }
            budget -= __popc(one) + __popc(two);
            if (budget < 0) fault |= ST_WALK_TREE;
            fault = __reduce_or_sync(kFull, fault);
            __syncwarp();
            if (fault) break;  // warp-uniform
        }
        if (fault) break;
        if (M2L) {
            if (lane == 0) {
                const int s = a_leaf ? A >> 1 : g.nleaf + (A >> 1);
                g.out_head[s] = out.head;
                g.out_len[s] = out.n;
            }
            ntask += (unsigned)out.n;
        } else if (a_leaf) {
            if (MODE != WALK_FILL && lane == 0) {
                if (MODE == WALK_ROWS) g.out_head[A >> 1] = out.head;
                g.out_len[A >> 1] = emitted;
            }
            if (fill && emitted != cap) fault |= ST_WALK_ROW;
        }
        if (!a_leaf && kept.n > 0) {  // A's children receive its undecided boxes
            const int s0 = a.son[0], s1 = a.son[1];
            int mid = it.lo;
            bool go0 = s0 >= 0, go1 = s1 >= 0;
            const bool v0 = s0 >= 0 && ((s0 & 1) ? (s0 >> 1) < g.nnode : (s0 >> 1) < g.nleaf);
            const bool v1 = s1 >= 0 && ((s1 & 1) ? (s1 >> 1) < g.nnode : (s1 >> 1) < g.nleaf);
            if ((!v0 && (!M2L || s0 >= 0)) || (!v1 && (!M2L || s1 >= 0))) fault |= ST_WALK_TREE;
            if (!M2L && !fault) {
                mid = (s1 & 1) ? g.node_first[s1 >> 1] : s1 >> 1;
                // pre-order leaves: both subtrees hold some, a leaf holds itself
                if (mid <= it.lo || mid >= it.hi) fault |= ST_WALK_TREE;
                else if ((!(s0 & 1) && (s0 >> 1 != it.lo || mid != it.lo + 1)) || (!(s1 & 1) && it.hi != mid + 1))
                    fault |= ST_WALK_TREE;
                if (!fault) {  // subtrees without a sink need no walk
                    go0 = g.active[mid] > g.active[it.lo];
                    go1 = g.active[it.hi] > g.active[mid];
                }
            }
            if (!fault) {
                if (lane == 0) {
                    if (go0) pushed[wid][npushed] = WalkItem{s0, A, it.lo, mid, kept.head, kept.n};
                    if (go1) pushed[wid][npushed + (go0 ? 1 : 0)] = WalkItem{s1, A, mid, it.hi, kept.head, kept.n};
                }
                npushed += (go0 ? 1 : 0) + (go1 ? 1 : 0);
                __syncwarp();
                if (npushed > 30) flush();
            }
        }
    }
    if (!fault && npushed) flush();
    fault = __reduce_or_sync(kFull, fault);
    if (lane == 0) {
        if (fault) atomicOr(&g.ctrl->status, fault);
        if (M2L && ntask) atomicAdd(&g.ctrl->ntask, ntask);
    }
}

// ---------------------------------------------------------- deep trees ---
//
// By depth, a leaf's warp follows what it opens alone while the next depth waits,
// and decided leaves wait on the stack for the open boxes before them. Particles at
// one point make a chain of splits that each peel off one particle: D depths of up
// to D - d steps each, and up to D leaves waiting. Such trees are walked by sink
// leaf: one warp per leaf L takes the pairs (A, B) from (root, root) that lead to
// L's entries, A on L's path, so no leaf waits for another, with a stack in global
// memory that the host enlarges as needed. Each pair is tested again for every
// leaf below A (7.6 ms for 128^3 clustered particles, 3.1 by depth).

// Whether every box is the child of one node at most, and the root of none: what
// the walk meets from the root then ends, whatever the codes.
static __global__ void __launch_bounds__(256)
walk_refs_kernel(const int *__restrict__ son, int nnode, int nleaf, int *__restrict__ refs, WalkCtrl *ctrl) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 2 * nnode; i += gridDim.x * blockDim.x) {
        const int c = son[i];
        if (c < 0 || ((c & 1) ? (c >> 1) >= nnode : (c >> 1) >= nleaf)) continue;  // reported where it is met
        if (c == 1 || atomicAdd(&refs[(c & 1) ? nleaf + (c >> 1) : c >> 1], 1) > 0)
            atomicOr(&ctrl->status, ST_WALK_TREE);
    }
}

// MODE: WALK_COUNT, WALK_FILL (rows in leaf order, as walk_level_kernel) or
// WALK_M2L (a box's tasks belong to the warp of its first leaf, which appends them
// one by one in the order of its walk; tail: per sink, its last chunk).
// A leaf's walk ends after kWalkSinkPairs pairs, or 64 a box in larger trees: some
// seconds, three times what the deepest chain that the tree build makes takes (6,143
// splits, 19 million pairs). Stacks: cap pairs per warp. Pairs lie on the stack in
// leaf order of B, whose subtrees do not overlap, the first on top.
constexpr long long kWalkSinkPairs = 1LL << 26;

template <int MODE>
__global__ void __launch_bounds__(kWalkWarps * 32)
walk_sink_kernel(const WalkRun g, int2 *stacks, int cap, int *__restrict__ tail) {
    constexpr bool M2L = MODE == WALK_M2L;
    const int lane = threadIdx.x & 31, warp = blockIdx.x * kWalkWarps + (threadIdx.x >> 5);
    const unsigned lt = (1u << lane) - 1u, above = ~(lt | (1u << lane));
    int2 *stk = stacks + (size_t)warp * cap;
    int fault = 0, depths = 0;
    unsigned long long ntask = 0;
    auto valid = [&](int c) { return c >= 0 && ((c & 1) ? (c >> 1) < g.nnode : (c >> 1) < g.nleaf); };
    auto first_leaf = [&](int c) { return (c & 1) ? g.node_first[c >> 1] : c >> 1; };
    const volatile int &failed = g.ctrl->status;  // (a walk that failed is not continued)
    for (int L = warp; L < g.nleaf; L += gridDim.x * kWalkWarps) {
        if (__any_sync(kFull, failed)) break;
        if (!M2L && g.active[L + 1] == g.active[L]) continue;  // (its count is 0)
        const int64_t row = MODE == WALK_FILL ? g.row_off[L] : 0;
        const int room = MODE == WALK_FILL ? (int)(g.row_off[L + 1] - row) : 0;
        // the child of a node on L's path that leads on to L (-1: none)
        auto toward = [&](const int son[2]) {
            const int s0 = son[0], s1 = son[1];
            int c = s0;
            if (s1 >= 0 || !M2L) {  // (the M2L walk passes over absent children)
                if (!valid(s1)) return -1;
                if (s0 < 0 || L >= first_leaf(s1)) c = s1;
            }
            return valid(c) && ((c & 1) || c >> 1 == L) ? c : -1;
        };
        if (lane == 0) stk[0] = make_int2(1, 1);
        __syncwarp();
        int sp = 1, emitted = 0;
        long long budget = max(kWalkSinkPairs, 64LL * ((long long)g.nnode + g.nleaf));
        while (sp > 0) {
            const int ns = min(32, sp);
            int2 v = make_int2(0, 0);
            if (lane < ns) v = stk[sp - 1 - lane];
            __syncwarp();  // the pairs are read before others are put in their places
            sp -= ns;
            budget -= ns;
            const int A = v.x;
            int B = v.y, cls = 0;  // 0 dropped, 1 decided, 2 opened
            int nc = 0, ca = A, c0 = -1, c1 = -1;  // the opened pair's nc pairs: (ca, c0), (ca, c1)
            bool task = false;
            if (lane < ns) {
                if (B < 0) {  // decided before
                    B = ~B;
                    cls = 1;
                } else if (!(A & 1) && !(B & 1)) {
                    cls = M2L ? 0 : 1;
                } else {
                    const WalkBox32 a = walk_load(g.box32 + A), b = walk_load(g.box32 + B);
                    int t = WALK_OPEN_B;
                    if (A != B) {
                        t = walk_bound(a, b, A & 1, B & 1, g.cut2, g.th2);
                        if (t == WALK_UNDECIDED) t = walk_exact(g.box, A, B, g.cutoff, g.open_angle);
                    }
                    task = M2L && t == WALK_ACCEPT && first_leaf(A) == L;
                    if (t == WALK_OPEN_A || A == B) {
                        ca = toward(a.son);
                        if (ca < 0) fault = ST_WALK_TREE;
                    }
                    if (t == WALK_OPEN_A) {
                        cls = 2;
                        nc = 1;
                        c0 = B;
                    } else if (t == WALK_OPEN_B) {  // (A, A) is opened on both sides
                        cls = 2;
                        c0 = b.son[0];
                        c1 = b.son[1];
                        const bool v0 = valid(c0), v1 = valid(c1);
                        if ((!v0 && (!M2L || c0 >= 0)) || (!v1 && (!M2L || c1 >= 0))) fault = ST_WALK_TREE;
                        if (!v0) c0 = c1;
                        nc = (v0 ? 1 : 0) + (v1 ? 1 : 0);
                    }
                }
            }
            const unsigned open = __ballot_sync(kFull, cls == 2), done = __ballot_sync(kFull, cls == 1);
            const unsigned ready = !open ? kFull : (open & (0u - open)) - 1u;
            if (M2L) {
                for (unsigned m = __ballot_sync(kFull, task); m; m &= m - 1u) {
                    const int from = __ffs(m) - 1;
                    const int a = __shfl_sync(kFull, A, from), b = __shfl_sync(kFull, B, from);
                    if (lane == 0 && !fault) {
                        const int s = (a & 1) ? g.nleaf + (a >> 1) : a >> 1, n = g.out_len[s];
                        int c;
                        if (n % kWalkTaskChunk) {
                            c = tail[s];
                        } else {
                            c = atomicAdd(&g.ctrl->out, 1);
                            if (c < 0 || c >= g.out.cap) {
                                fault = ST_WALK_OUT;
                            } else {
                                if (n == 0) g.out_head[s] = c;
                                else g.out.next[tail[s]] = c;
                                tail[s] = c;
                            }
                        }
                        if (!fault) {
                            g.out.ids[(size_t)c * kWalkTaskChunk + n % kWalkTaskChunk] = b;
                            g.out_len[s] = n + 1;
                            ++ntask;
                        }
                    }
                }
            } else {
                const unsigned m = done & ready;
                if (MODE == WALK_FILL && (m >> lane & 1u)) {
                    const int slot = emitted + __popc(m & lt);
                    if (slot < room) g.row_src[row + slot] = B >> 1;
                    else fault = ST_WALK_ROW;
                }
                emitted += __popc(m);
            }
            // the others back on the stack, the first on top
            const unsigned back = done & ~ready;
            const unsigned one = __ballot_sync(kFull, nc >= 1), two = __ballot_sync(kFull, nc == 2);
            const int total = __popc(back) + __popc(one) + __popc(two);
            if (budget < 0) fault |= ST_WALK_LONG;
            if (sp > cap - total) {
                fault |= ST_WALK_STACK;
            } else {
                const int at = sp + __popc(back & above) + __popc(one & above) + __popc(two & above);
                if (back >> lane & 1u) stk[at] = make_int2(A, ~B);
                if (nc == 1) stk[at] = make_int2(ca, c0);
                if (nc == 2) {
                    stk[at] = make_int2(ca, c1);
                    stk[at + 1] = make_int2(ca, c0);
                }
                sp += total;
            }
            fault = __reduce_or_sync(kFull, fault);
            __syncwarp();
            if (fault) break;  // warp-uniform
        }
        if (fault) break;
        if (MODE == WALK_COUNT && lane == 0) g.out_len[L] = emitted;
        if (MODE == WALK_FILL && emitted != room) fault = ST_WALK_ROW;
        if (M2L) {  // L's depth: its path's nodes and itself
            int d = 1;
            for (int c = 1; c >= 0 && (c & 1) && d <= g.nnode + 1; ++d) c = toward(g.box32[c].son);
            depths = max(depths, d);
        }
    }
    if (lane == 0) {
        if (fault) atomicOr(&g.ctrl->status, fault);
        if (M2L && ntask) atomicAdd(&g.ctrl->ntask, ntask);
        if (M2L && depths) atomicMax(&g.ctrl->items[0], depths);
    }
}

// Rows from the pool into their CSR places (CHAINS; else they are there
// already), and their pair counts (with skipped, the pairs of entries wholly
// beyond the FP32 forms' cutoff too). One warp per leaf.
template <bool CHAINS>
__global__ void __launch_bounds__(256)
walk_gather_kernel(const int *__restrict__ len, const int *__restrict__ head, const int64_t *__restrict__ row_off,
                   int nleaf, const WalkPool pool, int *__restrict__ row_src, const int *__restrict__ leaf_npart,
                   const LeafMeta *__restrict__ meta, double cscale, float uout,
                   unsigned long long *__restrict__ pairs, unsigned long long *__restrict__ skipped) {
    const int lane = threadIdx.x & 31;
    const int nw = (int)(((int64_t)gridDim.x * blockDim.x) >> 5);
    unsigned long long my_pairs = 0, my_skip = 0;
    for (int L = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); L < nleaf; L += nw) {
        const int n = len[L];
        if (n <= 0) continue;  // warp-uniform
        const int64_t base = row_off[L];
        const long long np_t = leaf_npart[L];
        LeafMeta mt{};
        if (skipped) mt = meta[L];
        int chunk = CHAINS ? head[L] : 0;
        for (int b = 0; b < n; b += kWalkChunk) {
            const int after = CHAINS && b + kWalkChunk < n ? pool.next[chunk] : 0;
#pragma unroll
            for (int h = 0; h < kWalkChunk; h += 32) {
                const int i = b + h + lane;
                if (i >= n) continue;
                int S;
                if (CHAINS) row_src[base + i] = S = pool.ids[(size_t)chunk * kWalkChunk + h + lane];
                else S = row_src[base + i];
                const unsigned long long np = (unsigned long long)(np_t * (long long)leaf_npart[S]);
                my_pairs += np;
                if (skipped) {
                    const LeafMeta ms = meta[S];
                    float ox, oy, oz;
                    entry_offset(ms, mt, cscale, ox, oy, oz);
                    if (entry_u_min(ms, mt, ox, oy, oz) > uout) my_skip += np;
                }
            }
            chunk = after;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        my_pairs += __shfl_xor_sync(kFull, my_pairs, off);
        my_skip += __shfl_xor_sync(kFull, my_skip, off);
    }
    if (lane == 0) {
        if (my_pairs) atomicAdd(pairs, my_pairs);
        if (skipped && my_skip) atomicAdd(skipped, my_skip);
    }
}

// ------------------------------------------------------------- launching ---

// Blocks of a launch: a depth has at most one box per leaf.
inline int walk_blocks(int sm_count, int boxes) {
    return std::min(sm_count * 8, (boxes + kWalkWarps - 1) / kWalkWarps);
}

// Enqueues depths [lv, lv + n) of a walk.
template <int MODE>
inline cudaError_t walk_depths(cudaStream_t st, const WalkRun &g, int sm_count, int lv, int n) {
    const int blocks = walk_blocks(sm_count, g.nleaf);
    for (int l = lv; l < lv + n; ++l) walk_level_kernel<MODE><<<blocks, kWalkWarps * 32, 0, st>>>(g, l);
    return cudaGetLastError();
}

// Depths enqueued before the host looks whether boxes are left: mean splits
// of clustered particles go about six depths below a balanced tree (26 for
// 828,182 leaves); an empty depth costs 2 us, another look 20.
inline int walk_first_depths(int nleaf) {
    int lg = 0;
    while (lg < 30 && (1 << lg) < nleaf) ++lg;
    return lg + 6;
}

// Blocks of a walk by sink leaf and its stacks' memory, at most 1 GB unless a
// single block's takes more.
constexpr int kWalkSinkStack = 2048;  // pairs a warp at first
inline int walk_sink_blocks(int sm_count, int nleaf, int cap) {
    const int64_t block = (int64_t)kWalkWarps * cap * (int64_t)sizeof(int2);
    return (int)std::max<int64_t>(1, std::min<int64_t>(walk_blocks(sm_count, nleaf), ((int64_t)1 << 30) / block));
}
inline size_t walk_sink_bytes(int blocks, int cap) { return (size_t)blocks * kWalkWarps * cap * sizeof(int2); }

// Enqueues a walk by sink leaf: refs (nnode + nleaf ints) is cleared here.
template <int MODE>
inline cudaError_t walk_sinks(cudaStream_t st, const WalkRun &g, const int *son, int *refs, int blocks, int2 *stacks,
                              int cap, int *tail) {
    cudaError_t e = cudaMemsetAsync(refs, 0, sizeof(int) * ((size_t)g.nnode + g.nleaf), st);
    if (e != cudaSuccess) return e;
    walk_refs_kernel<<<std::min((2 * (int64_t)g.nnode + 255) / 256, (int64_t)4096), 256, 0, st>>>(son, g.nnode, g.nleaf,
                                                                                                 refs, g.ctrl);
    walk_sink_kernel<MODE><<<blocks, kWalkWarps * 32, 0, st>>>(g, stacks, cap, tail);
    return cudaGetLastError();
}

inline float walk_th2(double open_angle) {
    return open_angle > 0.0 ? std::max((float)(open_angle * open_angle), 1.1754944e-38f) : 0.f;
}
inline size_t walk_pool_bytes(int64_t cap, int chunk) { return (size_t)cap * (size_t)(chunk + 1) * sizeof(int); }
inline WalkPool walk_pool(void *p, int64_t cap, int chunk) {
    return WalkPool{(int *)p, (int *)p + (size_t)cap * chunk, (int)cap};
}
// Chunks that warps hold without having used them, for `boxes` boxes with lists:
// 16 a box, 75,776 (20 MB of lists) where they fill the GPU.
inline int64_t walk_pool_slack(int sm_count, int boxes) {
    return (int64_t)walk_blocks(sm_count, boxes) * kWalkWarps * kWalkGrab;
}

}  // namespace p2p
