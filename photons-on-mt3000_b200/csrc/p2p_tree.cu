// Device kd-tree build (C ABI p2p_dtree_*; kernels in p2p_tree_kernels.cuh).
//
// Replaces the caller's build_kdtree / center_kdtree (src/fmm.c:69-122,
// 231-327) plus the leaf.active marking (src/fmm.c:1226-1236) on the GPU,
// producing the same tree: nodes and leaves in the reference's pre-order
// numbering, the same particle order, node and leaf boxes, active flags.
// The result feeds p2p_pass_begin_device (positions in tree order, leaf
// ranges) and p2p_pass_submit_walk (the node and leaf tables) directly.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "photons_p2p.h"
#include "p2p_host_shared.h"
#include "p2p_tree_kernels.cuh"

#define P2P_API extern "C" __attribute__((visibility("default")))

using namespace p2p;

struct p2p_dtree {
    int device = 0;
    int npart = 0, nleaf = 0, nnode = 0;
    double *pos = nullptr;  // SoA, tree order
    int *perm = nullptr;    // tree slot -> input index
    int *leaf_ipart = nullptr, *leaf_npart = nullptr, *leaf_active = nullptr;
    double *leaf_center = nullptr, *leaf_width = nullptr;  // AoS, 3 per leaf
    int *son = nullptr, *node_first = nullptr;
    double *node_center = nullptr, *node_width = nullptr;  // AoS, 3 per node
    float build_ms = 0.f;
    int cap_part = 0, cap_leaf = 0, cap_node = 0;  // sizes the arrays were allocated for
};

namespace {

void free_tree(p2p_dtree *t) {
    void *ptrs[] = {t->pos, t->perm, t->leaf_ipart, t->leaf_npart, t->leaf_active, t->leaf_center,
                    t->leaf_width, t->son, t->node_first, t->node_center, t->node_width};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    t->pos = t->leaf_center = t->leaf_width = t->node_center = t->node_width = nullptr;
    t->perm = t->leaf_ipart = t->leaf_npart = t->leaf_active = t->son = t->node_first = nullptr;
    t->cap_part = t->cap_leaf = t->cap_node = 0;
    t->npart = t->nleaf = t->nnode = 0;
}

// Temporaries of one build, in the session's grow-only scratch (one slot
// per request, numbered in request order): a rebuild of the same size
// allocates and frees nothing. The build returns only after its last kernel
// has finished, so the next build may reuse every slot.
struct Scratch {
    p2p_session *s;
    int next = 0;
    template <class T>
    bool get(T **out, size_t count) {
        void *p = session_scratch(s, next++, sizeof(T) * (count > 0 ? count : 1));
        if (!p) return false;
        *out = (T *)p;
        return true;
    }
};

template <class T>
bool dev_alloc(T **out, size_t count) {
    void *p = nullptr;
    if (cudaMalloc(&p, sizeof(T) * (count > 0 ? count : 1)) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    *out = (T *)p;
    return true;
}

int cuda_fail(cudaError_t e, const char *what) {
    char msg[256];
    snprintf(msg, sizeof(msg), "%s: %s", what, cudaGetErrorString(e));
    cudaGetLastError();
    return report_error(P2P_ERR_CUDA, msg);
}

#define TREE_CUDA(expr)                                  \
    do {                                                 \
        cudaError_t _e = (expr);                         \
        if (_e != cudaSuccess) return cuda_fail(_e, #expr); \
    } while (0)

int grid(int64_t n, int threads, int cap) {
    int64_t b = (n + threads - 1) / threads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, cap));
}

}  // namespace

namespace {

int check_build_args(p2p_session *s, int npart, const double *d_pos, int maxleaf, double boxsize) {
    if (!s) return report_error(P2P_ERR_ARG, "null argument");
    if (npart <= 0 || !d_pos) return report_error(P2P_ERR_ARG, "tree build needs particles");
    if (maxleaf <= 0) return report_error(P2P_ERR_ARG, "maxleaf must be positive");
    if (!(boxsize > 0.0)) return report_error(P2P_ERR_ARG, "boxsize must be positive");
    return P2P_OK;
}

// The tree's arrays for npart particles, nleaf leaves and nnode nodes: kept
// where they are large enough, else reallocated (with an eighth to spare,
// so rebuilds whose sizes drift reallocate rarely).
bool fit_tree(p2p_dtree *tree, int n, int nleaf, int nnode) {
    auto more = [](int c) { return (int)std::min<int64_t>((int64_t)c + c / 8 + 16, INT32_MAX); };
    bool ok = true;
    if (n > tree->cap_part) {
        cudaFree(tree->pos);
        cudaFree(tree->perm);
        tree->pos = nullptr;
        tree->perm = nullptr;
        const int c = more(n);
        ok = ok && dev_alloc(&tree->pos, 3 * (size_t)c) && dev_alloc(&tree->perm, c);
        tree->cap_part = ok ? c : 0;
    }
    if (ok && nleaf > tree->cap_leaf) {
        int **iv[] = {&tree->leaf_ipart, &tree->leaf_npart, &tree->leaf_active};
        double **dv[] = {&tree->leaf_center, &tree->leaf_width};
        for (int **p : iv) { cudaFree(*p); *p = nullptr; }
        for (double **p : dv) { cudaFree(*p); *p = nullptr; }
        const int c = more(nleaf);
        for (int **p : iv) ok = ok && dev_alloc(p, c);
        for (double **p : dv) ok = ok && dev_alloc(p, 3 * (size_t)c);
        tree->cap_leaf = ok ? c : 0;
    }
    if (ok && nnode > tree->cap_node) {
        cudaFree(tree->son);
        cudaFree(tree->node_first);
        cudaFree(tree->node_center);
        cudaFree(tree->node_width);
        tree->son = tree->node_first = nullptr;
        tree->node_center = tree->node_width = nullptr;
        const int c = more(nnode);
        ok = ok && dev_alloc(&tree->son, 2 * (size_t)c) && dev_alloc(&tree->node_first, c) &&
             dev_alloc(&tree->node_center, 3 * (size_t)c) && dev_alloc(&tree->node_width, 3 * (size_t)c);
        tree->cap_node = ok ? c : 0;
    }
    return ok;
}

// Builds into tree (its arrays reused where large enough). On an error the
// caller discards the tree's contents.
int build_into(p2p_session *s, p2p_dtree *tree, int npart, const double *d_pos, const int *d_tag, int maxleaf,
               double boxsize) {
    TREE_CUDA(cudaSetDevice(session_device(s)));
    cudaStream_t st = (cudaStream_t)p2p_session_stream(s);
    cudaEvent_t e0, e1;
    TREE_CUDA(cudaEventCreate(&e0));
    TREE_CUDA(cudaEventCreate(&e1));
    struct Events {
        cudaEvent_t a, b;
        ~Events() {
            cudaEventDestroy(a);
            cudaEventDestroy(b);
        }
    } evs{e0, e1};
    TREE_CUDA(cudaEventRecord(e0, st));
    int launches = 0;

    const int n = npart;
    // Nodes and leaves: a binary tree has one leaf more than nodes; leaves
    // hold up to maxleaf particles and mean splits keep most of them over
    // half full. The capacity allows 8 / maxleaf of a leaf per particle.
    const int64_t cap64 = std::min<int64_t>((int64_t)n + 1, 8LL * n / maxleaf + 1024);
    const int cap = (int)cap64;

    Scratch S{s};
    TreeParts P;
    TreeRec R;
    std::memset(&R, 0, sizeof(R));
    int *map = nullptr, *parent = nullptr, *lparent = nullptr, *arrived = nullptr;
    float *blo = nullptr, *bhi = nullptr;
    const int init_blocks = grid(n, kTreeThreads, 1024);
    bool ok = S.get(&P.x, n) && S.get(&P.y, n) && S.get(&P.z, n) && S.get(&P.id, n) && S.get(&map, n) &&
              S.get(&blo, 3 * (size_t)init_blocks) && S.get(&bhi, 3 * (size_t)init_blocks) &&
              S.get(&R.split, cap) && S.get(&R.son, 2 * (size_t)cap) && S.get(&R.depth, cap) &&
              S.get(&R.nn, cap) && S.get(&R.nl, cap) && S.get(&R.pre, cap) && S.get(&R.first, cap) &&
              S.get(&R.box, 6 * (size_t)cap) && S.get(&R.root, 6) && S.get(&R.lipart, cap) && S.get(&R.lnpart, cap) &&
              S.get(&R.lid, cap) && S.get(&parent, cap) && S.get(&lparent, cap) && S.get(&arrived, cap) &&
              S.get(&R.counters, 3);
    if (!ok) return report_error(P2P_ERR_NOMEM, "tree build: device allocation failed");
    R.node_cap = cap;
    R.leaf_cap = cap;

    tree_init_kernel<<<init_blocks, kTreeThreads, 0, st>>>(d_pos, n, P, blo, bhi);
    tree_root_box_kernel<<<1, 96, 0, st>>>(blo, bhi, init_blocks, boxsize, R);
    launches += 2;

    // ---- nodes above kTreeSmall particles, level by level; the host reads the
    // counts once the levels that such a tree has are queued (an empty level
    // costs its launches, a look at the counts about as much as two levels) ----
    const int seg_cap = n / (kTreeSmall + 1) + 1, task_cap = (int)(n / ((int64_t)maxleaf + 1)) + 1;
    const int tile_cap = (n + kTreeTile - 1) / kTreeTile + seg_cap;
    TreeSeg *segs[2] = {nullptr, nullptr};
    int *tile_seg[2] = {nullptr, nullptr}, *tile_off[2] = {nullptr, nullptr}, *tile_small = nullptr, *tile_pre = nullptr;
    TreeTask *tasks = nullptr;
    TreeLevels *lv = nullptr;
    for (int k = 0; k < 2; ++k)
        ok = ok && S.get(&segs[k], seg_cap) && S.get(&tile_seg[k], tile_cap) && S.get(&tile_off[k], tile_cap);
    ok = ok && S.get(&tile_small, tile_cap) && S.get(&tile_pre, tile_cap) && S.get(&tasks, task_cap) && S.get(&lv, 1);
    if (!ok) return report_error(P2P_ERR_NOMEM, "tree build: device allocation failed");
    TREE_CUDA(cudaMemsetAsync(lv, 0, sizeof(TreeLevels), st));
    TREE_CUDA(cudaMemsetAsync(R.counters, 0, 3 * sizeof(int), st));
    tree_first_level_kernel<<<grid((n + kTreeTile - 1) / kTreeTile, kTreeThreads, INT32_MAX), kTreeThreads, 0, st>>>(
        n, segs[0], tile_seg[0], tile_off[0], tasks, lv, R);
    launches += 1;
    int hc[3] = {0, 0, 0}, ntask = 0, left = 0, level = 0;
    int batch = 0;
    while (n > kTreeSmall && ((int64_t)kTreeSmall << batch) < n) ++batch;
    for (batch = n > kTreeSmall ? batch + 2 : 0;; batch = 2) {
        for (const int end = std::min(level + batch, kTreeLevels); level < end; ++level) {
            const int a = level & 1, b = a ^ 1;
            const int nseg = level < 30 ? std::min(1 << level, seg_cap) : seg_cap;
            const int ntile = std::min(n / kTreeTile + nseg, tile_cap);
            tree_seg_mean_kernel<<<nseg, kTreeThreads, 0, st>>>(segs[a], lv, level, P, R);
            tree_seg_chain_kernel<<<(nseg + 3) / 4, 128, 0, st>>>(segs[a], lv, level, P, R);
            tree_tile_count_kernel<<<ntile, kTreeThreads, 0, st>>>(segs[a], lv, level, tile_seg[a], tile_off[a], P,
                                                                   tile_small);
            tree_level_kernel<<<1, kTreeLevelThreads, 0, st>>>(segs[a], tile_seg[a], tile_small, tile_pre, segs[b],
                                                              tile_seg[b], tile_off[b], tasks, lv, level, maxleaf, seg_cap,
                                                              task_cap, R);
            tree_tile_map_kernel<<<ntile, kTreeThreads, 0, st>>>(segs[a], lv, level, tile_seg[a], tile_off[a], tile_pre, P,
                                                                 map);
            tree_tile_swap_kernel<<<ntile, kTreeThreads, 0, st>>>(segs[a], lv, level, tile_seg[a], tile_off[a], tile_pre,
                                                                  P, map);
            launches += 6;
        }
        TREE_CUDA(cudaGetLastError());
        TREE_CUDA(cudaMemcpyAsync(&left, &lv->nseg[level], sizeof(int), cudaMemcpyDeviceToHost, st));
        TREE_CUDA(cudaMemcpyAsync(&ntask, &lv->ntask, sizeof(int), cudaMemcpyDeviceToHost, st));
        TREE_CUDA(cudaMemcpyAsync(hc, R.counters, sizeof(hc), cudaMemcpyDeviceToHost, st));
        TREE_CUDA(cudaStreamSynchronize(st));
        if (hc[2] & (TB_NODE_CAP | TB_LEAF_CAP)) return report_error(P2P_ERR_CAPACITY, "tree build: node capacity");
        if (left == 0) break;
        if (level == kTreeLevels)
            return report_error(P2P_ERR_CAPACITY, "tree build: more than 4096 levels above 2048 particles");
    }

    // ---- subtrees of at most kTreeSmall particles, one block each ----
    if (ntask > 0) {
        TREE_CUDA(cudaFuncSetAttribute(tree_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kTreeSmallSmem));
        tree_small_kernel<<<ntask, kTreeSmallThreads, kTreeSmallSmem, st>>>(tasks, P, R, maxleaf);
        launches += 1;
        TREE_CUDA(cudaGetLastError());
    }
    TREE_CUDA(cudaMemcpyAsync(hc, R.counters, sizeof(hc), cudaMemcpyDeviceToHost, st));
    TREE_CUDA(cudaStreamSynchronize(st));
    if (hc[2] & (TB_NODE_CAP | TB_LEAF_CAP))
        return report_error(P2P_ERR_CAPACITY, "tree build: more nodes or leaves than the build's capacity");
    const int nnode = hc[0], nleaf = hc[1];

    // ---- pre-order numbering and boxes ----
    const int gn = grid(nnode, 256, 4096);
    tree_link_kernel<<<gn, 256, 0, st>>>(R, nnode, nleaf, parent, lparent, arrived);
    tree_count_kernel<<<grid(nleaf, 256, 4096), 256, 0, st>>>(R, nnode, nleaf, parent, lparent, arrived);
    tree_order_kernel<<<gn, 256, 0, st>>>(R, nnode, parent);
    launches += 3;

    p2p_dtree *t = tree;
    t->device = session_device(s);
    if (!fit_tree(t, n, nleaf, nnode)) return report_error(P2P_ERR_NOMEM, "tree build: device allocation failed");
    t->npart = n;
    t->nleaf = nleaf;
    t->nnode = nnode;
    tree_emit_kernel<<<gn, 256, 0, st>>>(R, nnode, nleaf, t->son, t->node_first, t->node_center, t->node_width,
                                         t->leaf_ipart, t->leaf_npart, t->leaf_center, t->leaf_width);
    {   // the numbering is consistent before the leaf tables are read
        int status = 0;
        cudaError_t ce = cudaMemcpyAsync(&status, R.counters + 2, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
        if (ce != cudaSuccess || (status & TB_NUMBERING)) {
            if (ce != cudaSuccess) return cuda_fail(ce, "tree build");
            return report_error(P2P_ERR_STATE, "tree build: inconsistent node records");
        }
    }
    tree_active_kernel<<<grid((int64_t)nleaf * 32, 256, 8192), 256, 0, st>>>(t->leaf_ipart, t->leaf_npart, nleaf,
                                                                            P.id, d_tag, t->leaf_active);
    tree_pos_out_kernel<<<grid(n, 256, 8192), 256, 0, st>>>(P, n, t->pos);
    launches += 3;
    cudaError_t e = cudaMemcpyAsync(t->perm, P.id, sizeof(int) * (size_t)n, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaEventRecord(e1, st);
    if (e == cudaSuccess) e = cudaEventSynchronize(e1);  // the next build may reuse the scratch
    if (e == cudaSuccess) e = cudaEventElapsedTime(&t->build_ms, e0, e1);
    if (e != cudaSuccess) return cuda_fail(e, "tree build");
    count_launches(launches);
    return P2P_OK;
}

}  // namespace

P2P_API int p2p_dtree_build(p2p_session *s, int npart, const double *d_pos, const int *d_tag, int maxleaf,
                            double boxsize, p2p_dtree **out) {
    if (!out) return report_error(P2P_ERR_ARG, "null argument");
    *out = nullptr;
    const int st = check_build_args(s, npart, d_pos, maxleaf, boxsize);
    if (st != P2P_OK) return st;
    p2p_dtree *t = new p2p_dtree();
    const int r = build_into(s, t, npart, d_pos, d_tag, maxleaf, boxsize);
    if (r != P2P_OK) {
        cudaSetDevice(t->device);
        free_tree(t);
        delete t;
        return r;
    }
    *out = t;
    return P2P_OK;
}

P2P_API int p2p_dtree_rebuild(p2p_session *s, p2p_dtree *t, int npart, const double *d_pos, const int *d_tag,
                              int maxleaf, double boxsize) {
    if (!t) return report_error(P2P_ERR_ARG, "null tree");
    const int st = check_build_args(s, npart, d_pos, maxleaf, boxsize);
    if (st != P2P_OK) return st;
    if ((t->pos || t->son) && t->device != session_device(s))
        return report_error(P2P_ERR_ARG, "tree and session are on different devices");
    const int r = build_into(s, t, npart, d_pos, d_tag, maxleaf, boxsize);
    if (r != P2P_OK) t->npart = t->nleaf = t->nnode = 0;  // no tree; its arrays stay for the next rebuild
    return r;
}

P2P_API int p2p_dtree_free(p2p_dtree *t) {
    if (!t) return P2P_OK;
    cudaSetDevice(t->device);
    free_tree(t);
    delete t;
    return P2P_OK;
}

P2P_API int p2p_dtree_counts(const p2p_dtree *t, int *npart, int *nleaf, int *nnode, float *build_ms) {
    if (!t) return report_error(P2P_ERR_ARG, "null tree");
    if (npart) *npart = t->npart;
    if (nleaf) *nleaf = t->nleaf;
    if (nnode) *nnode = t->nnode;
    if (build_ms) *build_ms = t->build_ms;
    return P2P_OK;
}

P2P_API int p2p_dtree_device_arrays(const p2p_dtree *t, const double **d_pos, const int **d_perm,
                                    const int **d_leaf_ipart, const int **d_leaf_npart) {
    if (!t) return report_error(P2P_ERR_ARG, "null tree");
    if (d_pos) *d_pos = t->pos;
    if (d_perm) *d_perm = t->perm;
    if (d_leaf_ipart) *d_leaf_ipart = t->leaf_ipart;
    if (d_leaf_npart) *d_leaf_npart = t->leaf_npart;
    return P2P_OK;
}

P2P_API int p2p_dtree_walk_tree(const p2p_dtree *t, p2p_walk_tree *w) {
    if (!t || !w) return report_error(P2P_ERR_ARG, "null argument");
    w->nnode = t->nnode;
    w->nleaf = t->nleaf;
    w->son = t->son;
    w->node_first = t->node_first;
    w->node_center = t->node_center;
    w->node_width = t->node_width;
    w->leaf_center = t->leaf_center;
    w->leaf_width = t->leaf_width;
    w->leaf_active = t->leaf_active;
    return P2P_OK;
}

P2P_API int p2p_dtree_unpermute(const p2p_dtree *t, p2p_session *s, const double *d_in, double *d_out) {
    if (!t || !s || !d_in || !d_out) return report_error(P2P_ERR_ARG, "null argument");
    if (d_in == d_out) return report_error(P2P_ERR_ARG, "unpermute needs distinct buffers");
    TREE_CUDA(cudaSetDevice(t->device));
    cudaStream_t st = (cudaStream_t)p2p_session_stream(s);
    tree_unpermute_kernel<<<grid(t->npart, 256, 8192), 256, 0, st>>>(d_in, t->perm, t->npart, d_out);
    TREE_CUDA(cudaGetLastError());
    count_launches(1);
    return P2P_OK;
}

P2P_API int p2p_dtree_download(const p2p_dtree *t, double *pos, int *perm, int *leaf_ipart, int *leaf_npart,
                               int *leaf_active, double *leaf_center, double *leaf_width, int *son,
                               int *node_first, double *node_center, double *node_width) {
    if (!t) return report_error(P2P_ERR_ARG, "null tree");
    TREE_CUDA(cudaSetDevice(t->device));
    struct Item {
        void *dst;
        const void *src;
        size_t bytes;
    } items[] = {{pos, t->pos, sizeof(double) * 3 * (size_t)t->npart},
                 {perm, t->perm, sizeof(int) * (size_t)t->npart},
                 {leaf_ipart, t->leaf_ipart, sizeof(int) * (size_t)t->nleaf},
                 {leaf_npart, t->leaf_npart, sizeof(int) * (size_t)t->nleaf},
                 {leaf_active, t->leaf_active, sizeof(int) * (size_t)t->nleaf},
                 {leaf_center, t->leaf_center, sizeof(double) * 3 * (size_t)t->nleaf},
                 {leaf_width, t->leaf_width, sizeof(double) * 3 * (size_t)t->nleaf},
                 {son, t->son, sizeof(int) * 2 * (size_t)t->nnode},
                 {node_first, t->node_first, sizeof(int) * (size_t)t->nnode},
                 {node_center, t->node_center, sizeof(double) * 3 * (size_t)t->nnode},
                 {node_width, t->node_width, sizeof(double) * 3 * (size_t)t->nnode}};
    for (const Item &it : items)
        if (it.dst && it.bytes) TREE_CUDA(cudaMemcpy(it.dst, it.src, it.bytes, cudaMemcpyDeviceToHost));
    return P2P_OK;
}
