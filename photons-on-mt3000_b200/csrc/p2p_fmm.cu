// Far field of the short-range force on the GPU (C ABI p2p_fmm_*): the
// multipole part of PhotoNs' FMM within the cutoff sphere, the complement of
// the P2P pass on the same kd-tree.
//
//   p2m + m2m  every leaf's multipole to octupole order about its box centre
//              (p2m, src/operator.c:14-97), then each node's from its two
//              children's, shifted to its centre (m2m / walk_m2m, :102-199):
//              one thread per leaf, climbing while it is the last of a
//              node's children to finish
//   M2L walk   the reference's dual-tree recursion from (root, root)
//              (walk_task_m2l, src/fmm.c:812-957, with the acceptance test
//              of :409-479) depth by depth of the sink side on the GPU
//              (walk_level_kernel; deep trees by sink leaf, walk_sink_kernel),
//              each sink's accepted sources in a list
//   M2L        each sink (leaf or node), half a warp, sums over its list, in the
//              order the walk leaves it, the source multipole's contribution
//              to its local expansion with the erfc-truncated kernel's derivatives
//              (m2l with LONGSHORT, src/operator.c:331-475)
//   l2l + l2p  each leaf takes its ancestors' locals down its path from the
//              root (l2l / walk_l2l, :477-606) and, if it holds a local
//              particle, evaluates the gradient at its particles (l2p,
//              :203-262; called for active leaves at src/gravity.c:427-428)
//
// Expansions are 20 coefficients per box in the reference's index order
// (inc/operator.h): 1, x, y, z, xx, xy, xz, yy, yz, zz, xxx, xxy, xxz, xyy,
// xyz, xzz, yyy, yyz, yzz, zzz. Multipole coefficients carry (-1)^n / a!b!c!
// and the locals are the derivatives, so a shift or a contraction is a sum
// over multi-indices with the monomials d^g / g! of the shift (mono below).
//
// The reference's m2l returns early when `abs(r2) <= 1e-15` with the integer
// abs() of <stdlib.h> (src/operator.c:340-344): every task with r2 < 1 in
// the caller's length unit contributes nothing. min_r2 keeps that behaviour
// selectable: 1 reproduces the reference, 1e-15 the evident intent.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "photons_p2p.h"
#include "p2p_host_shared.h"
#include "p2p_internal.h"

#include "p2p_walk_kernels.cuh"

#define P2P_API extern "C" __attribute__((visibility("default")))

using namespace p2p;

namespace {

constexpr int kNC = 20;  // coefficients per expansion (octupole)

// Exponents (a, b, c) of coefficient k.
__host__ __device__ constexpr int ex(int k, int d) {
    constexpr int t[kNC][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {2, 0, 0}, {1, 1, 0}, {1, 0, 1},
                               {0, 2, 0}, {0, 1, 1}, {0, 0, 2}, {3, 0, 0}, {2, 1, 0}, {2, 0, 1}, {1, 2, 0},
                               {1, 1, 1}, {1, 0, 2}, {0, 3, 0}, {0, 2, 1}, {0, 1, 2}, {0, 0, 3}};
    return t[k][d];
}
__host__ __device__ constexpr int order(int k) { return ex(k, 0) + ex(k, 1) + ex(k, 2); }
// Index of the coefficient with exponents (a, b, c), a + b + c <= 3; -1 otherwise.
__host__ __device__ constexpr int idx(int a, int b, int c) {
    if (a < 0 || b < 0 || c < 0 || a + b + c > 3) return -1;
    for (int k = 0; k < kNC; ++k)
        if (ex(k, 0) == a && ex(k, 1) == b && ex(k, 2) == c) return k;
    return -1;
}
__host__ __device__ constexpr int sum_idx(int k, int j) {
    return idx(ex(k, 0) + ex(j, 0), ex(k, 1) + ex(j, 1), ex(k, 2) + ex(j, 2));
}
__host__ __device__ constexpr int diff_idx(int k, int j) {  // k - j, -1 unless j <= k componentwise
    return idx(ex(k, 0) - ex(j, 0), ex(k, 1) - ex(j, 1), ex(k, 2) - ex(j, 2));
}

// d^g / g! for every multi-index g.
__device__ __forceinline__ void mono(double dx, double dy, double dz, double *p) {
    const double x2 = dx * dx * 0.5, y2 = dy * dy * 0.5, z2 = dz * dz * 0.5;
    p[0] = 1.0;
    p[1] = dx; p[2] = dy; p[3] = dz;
    p[4] = x2; p[5] = dx * dy; p[6] = dx * dz; p[7] = y2; p[8] = dy * dz; p[9] = z2;
    p[10] = x2 * dx * (1.0 / 3.0); p[11] = x2 * dy; p[12] = x2 * dz; p[13] = dx * y2; p[14] = dx * dy * dz;
    p[15] = dx * z2; p[16] = y2 * dy * (1.0 / 3.0); p[17] = y2 * dz; p[18] = dy * z2; p[19] = z2 * dz * (1.0 / 3.0);
}

// Multipole shift: out[a] += sum_{b <= a} m[b] p[a - b].
__device__ __forceinline__ void shift_m(const double *m, const double *p, double *out) {
#pragma unroll
    for (int a = 0; a < kNC; ++a) {
        double s = 0.0;
#pragma unroll
        for (int b = 0; b < kNC; ++b)
            if (diff_idx(a, b) >= 0) s += m[b] * p[diff_idx(a, b)];
        out[a] += s;
    }
}

// Local shift: out[a] += sum_{b >= a} l[b] p[b - a].
__device__ __forceinline__ void shift_l(const double *l, const double *p, double *out) {
#pragma unroll
    for (int a = 0; a < kNC; ++a) {
        double s = 0.0;
#pragma unroll
        for (int b = 0; b < kNC; ++b)
            if (diff_idx(b, a) >= 0) s += l[b] * p[diff_idx(b, a)];
        out[a] += s;
    }
}

// Derivatives to third order of phi(r) = erfc(r / (2 r_s)) / r at r = (x, y,
// z), the radial factors of m2l's LONGSHORT branch.
__device__ __forceinline__ void kernel_derivs(double x, double y, double z, double r2, double irs, double *D) {
    const double dr = sqrt(r2), ir = 1.0 / dr;
    const double ir2 = ir * ir, ir3 = ir2 * ir, ir4 = ir2 * ir2, ir5 = ir4 * ir, ir6 = ir4 * ir2, ir7 = ir6 * ir;
    const double irs3 = irs * irs * irs, irs5 = irs3 * irs * irs;
    const double u = 0.5 * dr * irs;
    const double ec = exp(-u * u) * 0.56418958354775628695;  // exp(-u^2) / sqrt(pi)
    const double c = erfc(u);
    const double f0 = ir * c;
    const double f1 = -ir3 * (c + dr * ec * irs);
    const double f2 = 3.0 * ir5 * c + (3.0 * irs * ir4 + 0.5 * ir2 * irs3) * ec;
    const double f3 = -15.0 * ir7 * c - (15.0 * ir6 * irs + 2.5 * ir4 * irs3 + 0.25 * ir2 * irs5) * ec;
    const double v[3] = {x, y, z};
    D[0] = f0;
#pragma unroll
    for (int k = 1; k < kNC; ++k) {
        // the axes of coefficient k as an index list i <= j <= l
        int ax[3], n = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int r = 0; r < ex(k, d); ++r) ax[n++] = d;
        if (order(k) == 1) {
            D[k] = f1 * v[ax[0]];
        } else if (order(k) == 2) {
            D[k] = f2 * v[ax[0]] * v[ax[1]] + (ax[0] == ax[1] ? f1 : 0.0);
        } else {
            double t = 0.0;
            if (ax[1] == ax[2]) t += v[ax[0]];
            if (ax[0] == ax[2]) t += v[ax[1]];
            if (ax[0] == ax[1]) t += v[ax[2]];
            D[k] = f3 * v[ax[0]] * v[ax[1]] * v[ax[2]] + f2 * t;
        }
    }
}

struct FmmArgs {
    WalkArgs w;
    const double *pos;       // 3 * npart SoA, tree order
    const int *leaf_ip, *leaf_np;
    int npart;
    double mass, irs, min_r2;
    int *leaf_parent, *node_parent, *nchild, *arrive;
    double *leafM, *nodeM;   // 20 per box
    double *sinkL;           // 20 per sink: leaves then nodes
    double *leafL;           // 20 per leaf: final locals
    int *status;
};

__device__ __forceinline__ const double *box_center(const WalkArgs &w, int c) { return walk_center(w, c); }
__device__ __forceinline__ int sink_index(const WalkArgs &w, int c) { return (c & 1) ? w.nleaf + (c >> 1) : (c >> 1); }

__global__ void fmm_parent_kernel(FmmArgs f) {
    const WalkArgs &w = f.w;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nnode; k += gridDim.x * blockDim.x) {
        int n = 0;
        for (int s = 0; s < 2; ++s) {
            const int c = w.son[2 * k + s];
            if (c < 0) continue;
            if (!walk_valid(w, c)) {
                atomicOr(f.status, ST_WALK_TREE);
                continue;
            }
            if (c & 1)
                f.node_parent[c >> 1] = k;
            else
                f.leaf_parent[c >> 1] = k;
            ++n;
        }
        f.nchild[k] = n;
        f.arrive[k] = 0;
    }
}

// Multipole of leaf l (p2m), then up the tree while this thread is the last
// of a node's children to arrive: the node's multipole from its children's,
// son[0]'s first.
__global__ void fmm_upward_kernel(FmmArgs f) {
    const WalkArgs &w = f.w;
    for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < w.nleaf; l += gridDim.x * blockDim.x) {
        double M[kNC];
#pragma unroll
        for (int k = 0; k < kNC; ++k) M[k] = 0.0;
        const double *c = w.leaf_center + 3 * (size_t)l;
        const int ip = f.leaf_ip[l], np = f.leaf_np[l];
        const size_t n = (size_t)f.npart;
        for (int i = ip; i < ip + np; ++i) {
            double p[kNC];
            mono(f.pos[i] - c[0], f.pos[n + i] - c[1], f.pos[2 * n + i] - c[2], p);
#pragma unroll
            for (int k = 0; k < kNC; ++k) M[k] += ((order(k) & 1) ? -f.mass : f.mass) * p[k];
        }
#pragma unroll
        for (int k = 0; k < kNC; ++k) f.leafM[(size_t)kNC * l + k] = M[k];
        int node = f.leaf_parent[l], guard = 0;
        while (node >= 0) {
            if (++guard > 4096) {  // deeper than any tree the builders make: a cycle
                atomicOr(f.status, ST_WALK_TREE);
                break;
            }
            __threadfence();
            if (atomicAdd(&f.arrive[node], 1) != f.nchild[node] - 1) break;
            __threadfence();
            double T[kNC];
#pragma unroll
            for (int k = 0; k < kNC; ++k) T[k] = 0.0;
            const double *pc = w.node_center + 3 * (size_t)node;
            for (int s = 0; s < 2; ++s) {
                const int ch = w.son[2 * node + s];
                if (ch < 0 || !walk_valid(w, ch)) continue;
                const double *cc = box_center(w, ch);
                const double *src = (ch & 1) ? f.nodeM + (size_t)kNC * (ch >> 1) : f.leafM + (size_t)kNC * (ch >> 1);
                double m[kNC], p[kNC];
#pragma unroll
                for (int k = 0; k < kNC; ++k) m[k] = __ldcg(src + k);
                mono(pc[0] - cc[0], pc[1] - cc[1], pc[2] - cc[2], p);
                shift_m(m, p, T);
            }
#pragma unroll
            for (int k = 0; k < kNC; ++k) f.nodeM[(size_t)kNC * node + k] = T[k];
            node = f.node_parent[node];
        }
    }
}

// M2L: half a warp per sink (a sink has about 10 tasks at open angle 0.4),
// lane j takes tasks j, j + 16, ... of its list, in the order the walk left
// them (which does not vary between runs), and the lanes' partial locals are
// summed by a fixed shuffle tree: the same sum on every run. The walk keeps a sink's tasks together, so nothing is sorted.
constexpr int kM2LThreads = 128;

__global__ void __launch_bounds__(kM2LThreads)
fmm_m2l_kernel(FmmArgs f, const int *__restrict__ head, const int *__restrict__ len, const WalkPool pool,
               unsigned long long *applied) {
    const WalkArgs &w = f.w;
    constexpr int H = kWalkTaskChunk;  // lanes per sink, tasks per chunk
    static_assert(H == 16, "a chunk of tasks is one per lane of a half warp");
    const int lane = threadIdx.x & (H - 1);
    const int nsink = w.nleaf + w.nnode;
    const int nhalf = gridDim.x * (blockDim.x / H);
    unsigned used = 0;
    // whole warps stay in the loop (the shuffles below)
    for (int s0 = (blockIdx.x * blockDim.x + threadIdx.x) / H; (s0 & ~1) < nsink; s0 += nhalf) {
        const int s = min(s0, nsink - 1);
        const int k = s0 < nsink ? len[s] : 0;
        double L[kNC];
#pragma unroll
        for (int c = 0; c < kNC; ++c) L[c] = 0.0;
        const int code = s < w.nleaf ? 2 * s : 2 * (s - w.nleaf) + 1;
        const double *cs = box_center(w, code);
        int chunk = k ? head[s] : 0;
        for (int b = 0; b < k; b += H) {
            const int t = chunk;
            if (b + H < k) chunk = pool.next[t];
            if (b + lane >= k) continue;
            const int sc = pool.ids[(size_t)t * H + lane];
            const double *cb = box_center(w, sc);
            const double x = cs[0] - cb[0], y = cs[1] - cb[1], z = cs[2] - cb[2];
            const double r2 = x * x + y * y + z * z;
            if (!(r2 >= f.min_r2)) continue;
            ++used;
            const double *Msrc = (sc & 1) ? f.nodeM + (size_t)kNC * (sc >> 1) : f.leafM + (size_t)kNC * (sc >> 1);
            double m[kNC], D[kNC];
#pragma unroll
            for (int c = 0; c < kNC; ++c) m[c] = Msrc[c];
            kernel_derivs(x, y, z, r2, f.irs, D);
#pragma unroll
            for (int c = 0; c < kNC; ++c) {
                double acc = 0.0;
#pragma unroll
                for (int j = 0; j < kNC; ++j)
                    if (sum_idx(c, j) >= 0) acc += m[j] * D[sum_idx(c, j)];
                L[c] += acc;
            }
        }
        __syncwarp();
#pragma unroll
        for (int o = H / 2; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < kNC; ++c) L[c] += __shfl_down_sync(kFull, L[c], o, H);
        if (lane == 0 && s0 < nsink) {
#pragma unroll
            for (int c = 0; c < kNC; ++c) f.sinkL[(size_t)kNC * s + c] = L[c];
        }
    }
    used = __reduce_add_sync(kFull, used);
    if ((threadIdx.x & 31) == 0 && used) atomicAdd(applied, (unsigned long long)used);
}

// Locals down each leaf's path from the root, then the gradient at the
// leaf's particles (active leaves; zero for the others).
__global__ void fmm_downward_kernel(FmmArgs f, double *__restrict__ acc) {
    const WalkArgs &w = f.w;
    const size_t n = (size_t)f.npart;
    for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < w.nleaf; l += gridDim.x * blockDim.x) {
        double L[kNC];
        int A;
        if (w.nnode > 0) {
            A = 1;  // the root node
#pragma unroll
            for (int k = 0; k < kNC; ++k) L[k] = f.sinkL[(size_t)kNC * w.nleaf + k];
            int guard = 0;
            while ((A & 1) && guard++ < 4096) {
                const int ch = walk_child_toward(w, A, l);
                if (ch < 0 || !walk_valid(w, ch)) {
                    atomicOr(f.status, ST_WALK_TREE);
                    break;
                }
                const double *pc = box_center(w, A), *cc = box_center(w, ch);
                double T[kNC], p[kNC];
                const double *own = f.sinkL + (size_t)kNC * sink_index(w, ch);
#pragma unroll
                for (int k = 0; k < kNC; ++k) T[k] = own[k];
                mono(cc[0] - pc[0], cc[1] - pc[1], cc[2] - pc[2], p);
                shift_l(L, p, T);
#pragma unroll
                for (int k = 0; k < kNC; ++k) L[k] = T[k];
                A = ch;
            }
            if (A != 2 * l) atomicOr(f.status, ST_WALK_TREE);
        } else {
#pragma unroll
            for (int k = 0; k < kNC; ++k) L[k] = f.sinkL[(size_t)kNC * l + k];
        }
#pragma unroll
        for (int k = 0; k < kNC; ++k) f.leafL[(size_t)kNC * l + k] = L[k];
        const int ip = f.leaf_ip[l], np = f.leaf_np[l];
        const bool active = w.leaf_active[l] >= 0;
        const double *c = w.leaf_center + 3 * (size_t)l;
        for (int i = ip; i < ip + np; ++i) {
            double g[3] = {0.0, 0.0, 0.0};
            if (active) {
                double p[kNC];
                mono(f.pos[i] - c[0], f.pos[n + i] - c[1], f.pos[2 * n + i] - c[2], p);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    // d/dx_d of sum_b L[b] x^b / b!: sum over b with b_d >= 1 of L[b] x^(b - e_d) / (b - e_d)!
#pragma unroll
                    for (int b = 1; b < kNC; ++b) {
                        const int r = idx(ex(b, 0) - (d == 0), ex(b, 1) - (d == 1), ex(b, 2) - (d == 2));
                        if (r >= 0) g[d] += L[b] * p[r];
                    }
                }
            }
            acc[i] = g[0];
            acc[n + i] = g[1];
            acc[2 * n + i] = g[2];
        }
    }
}

struct DevBufF {
    void *p = nullptr;
    size_t cap = 0;
};

int grow(DevBufF &b, size_t bytes) {
    if (bytes == 0) bytes = 16;
    if (b.cap >= bytes) return P2P_OK;
    if (b.p) cudaFree(b.p);
    b.p = nullptr;
    b.cap = 0;
    const size_t want = bytes + bytes / 4;
    if (cudaMalloc(&b.p, want) != cudaSuccess) {
        cudaGetLastError();
        return report_error(P2P_ERR_NOMEM, "FMM scratch allocation failed");
    }
    b.cap = want;
    return P2P_OK;
}

int fail_cuda(cudaError_t e, const char *what) {
    char msg[256];
    snprintf(msg, sizeof(msg), "%s: %s", what, cudaGetErrorString(e));
    cudaGetLastError();
    return report_error(P2P_ERR_CUDA, msg);
}

int blocks_for(long long n, int threads) {
    long long b = (n + threads - 1) / threads;
    return (int)std::max(1LL, std::min(b, 148LL * 32));
}

}  // namespace

struct p2p_fmm {
    int device = 0;
    cudaStream_t stream = nullptr;
    DevBufF parents, leafM, nodeM, sinkL, leafL, counts, ctrl;
    DevBufF box, items, lists[2], tasks, tails, walk_ctrl;  // the M2L walk
    WalkLimits limits;
    cudaEvent_t ev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    long long n_m2l = 0, n_applied = 0;
    int levels = 0, nleaf = 0, nnode = 0;
};

#define FMM_TRY(expr)                \
    do {                             \
        int _s = (expr);             \
        if (_s != P2P_OK) return _s; \
    } while (0)
#define FMM_CUDA(expr, what)                        \
    do {                                            \
        cudaError_t _e = (expr);                    \
        if (_e != cudaSuccess) return fail_cuda(_e, what); \
    } while (0)

P2P_API int p2p_fmm_create(p2p_session *s, p2p_fmm **out) {
    if (!s || !out) return report_error(P2P_ERR_ARG, "null argument");
    *out = nullptr;
    FMM_CUDA(cudaSetDevice(session_device(s)), "cudaSetDevice");
    p2p_fmm *f = new p2p_fmm();
    f->device = session_device(s);
    f->stream = (cudaStream_t)p2p_session_stream(s);
    f->limits = session_walk_limits(s);
    for (cudaEvent_t &e : f->ev) {
        if (cudaEventCreate(&e) != cudaSuccess) {
            cudaGetLastError();
            p2p_fmm_destroy(f);
            return report_error(P2P_ERR_CUDA, "FMM event creation failed");
        }
    }
    *out = f;
    return P2P_OK;
}

P2P_API int p2p_fmm_destroy(p2p_fmm *f) {
    if (!f) return P2P_OK;
    cudaSetDevice(f->device);
    cudaStreamSynchronize(f->stream);
    DevBufF *bufs[] = {&f->parents, &f->leafM, &f->nodeM, &f->sinkL, &f->leafL, &f->counts, &f->ctrl, &f->box,
                       &f->items, &f->lists[0], &f->lists[1], &f->tasks, &f->tails, &f->walk_ctrl};
    for (DevBufF *b : bufs)
        if (b->p) cudaFree(b->p);
    for (cudaEvent_t e : f->ev)
        if (e) cudaEventDestroy(e);
    delete f;
    return P2P_OK;
}

P2P_API int p2p_fmm_far(p2p_fmm *f, const p2p_walk_tree *t, int npart, const double *d_pos, const int *d_leaf_ipart,
                        const int *d_leaf_npart, double mass, double split_radius, double cutoff, double open_angle,
                        double min_r2, double *d_acc) {
    if (!f || !t) return report_error(P2P_ERR_ARG, "null argument");
    if (npart < 0 || t->nleaf < 0 || t->nnode < 0) return report_error(P2P_ERR_ARG, "negative size");
    if (npart > 0 && (!d_pos || !d_acc || !d_leaf_ipart || !d_leaf_npart))
        return report_error(P2P_ERR_ARG, "null device array");
    if ((t->nnode > 0 && (!t->son || !t->node_first || !t->node_center || !t->node_width)) ||
        (t->nleaf > 0 && (!t->leaf_center || !t->leaf_width || !t->leaf_active)))
        return report_error(P2P_ERR_ARG, "null tree array");
    if (!(split_radius > 0.0) || !(cutoff >= 0.0) || !(open_angle >= 0.0) || !(min_r2 >= 0.0) ||
        !std::isfinite(mass))
        return report_error(P2P_ERR_ARG, "bad split radius, cutoff, open angle, min_r2 or mass");
    FMM_CUDA(cudaSetDevice(f->device), "cudaSetDevice");
    const int nleaf = t->nleaf, nnode = t->nnode, nsink = nleaf + nnode;
    f->nleaf = nleaf;
    f->nnode = nnode;
    f->n_m2l = f->n_applied = 0;
    f->levels = 0;
    cudaStream_t st = f->stream;
    const int threads = 256;
    FMM_CUDA(cudaEventRecord(f->ev[0], st), "FMM");
    if (nleaf == 0) {
        if (npart) FMM_CUDA(cudaMemsetAsync(d_acc, 0, sizeof(double) * 3 * (size_t)npart, st), "FMM");
        for (int k = 1; k < 5; ++k) FMM_CUDA(cudaEventRecord(f->ev[k], st), "FMM");
        return P2P_OK;
    }
    FMM_TRY(grow(f->parents, sizeof(int) * ((size_t)nleaf + 3 * (size_t)nnode)));
    FMM_TRY(grow(f->leafM, sizeof(double) * kNC * (size_t)nleaf));
    FMM_TRY(grow(f->nodeM, sizeof(double) * kNC * (size_t)std::max(nnode, 1)));
    FMM_TRY(grow(f->sinkL, sizeof(double) * kNC * (size_t)nsink));
    FMM_TRY(grow(f->leafL, sizeof(double) * kNC * (size_t)nleaf));
    FMM_TRY(grow(f->counts, sizeof(int) * 2 * (size_t)nsink));
    FMM_TRY(grow(f->ctrl, 64));
    FmmArgs a;
    a.w.nnode = nnode;
    a.w.nleaf = nleaf;
    a.w.son = t->son;
    a.w.node_first = t->node_first;
    a.w.leaf_active = t->leaf_active;
    a.w.node_center = t->node_center;
    a.w.node_width = t->node_width;
    a.w.leaf_center = t->leaf_center;
    a.w.leaf_width = t->leaf_width;
    a.w.cutoff = cutoff;
    a.w.open_angle = open_angle;
    a.pos = d_pos;
    a.leaf_ip = d_leaf_ipart;
    a.leaf_np = d_leaf_npart;
    a.npart = npart;
    a.mass = mass;
    a.irs = 1.0 / split_radius;
    a.min_r2 = min_r2;
    int *par = (int *)f->parents.p;
    a.leaf_parent = par;
    a.node_parent = par + nleaf;
    a.nchild = par + nleaf + nnode;
    a.arrive = par + nleaf + 2 * nnode;
    a.leafM = (double *)f->leafM.p;
    a.nodeM = (double *)f->nodeM.p;
    a.sinkL = (double *)f->sinkL.p;
    a.leafL = (double *)f->leafL.p;
    unsigned long long *ctrl = (unsigned long long *)f->ctrl.p;  // [0] nout [1] ntask [2] applied [3] status
    a.status = (int *)(ctrl + 3);
    FMM_CUDA(cudaMemsetAsync(ctrl, 0, 64, st), "FMM");
    FMM_CUDA(cudaMemsetAsync(par, 0xff, sizeof(int) * ((size_t)nleaf + nnode), st), "FMM");  // parents -1
    if (nnode) fmm_parent_kernel<<<blocks_for(nnode, threads), threads, 0, st>>>(a);
    fmm_upward_kernel<<<blocks_for(nleaf, threads), threads, 0, st>>>(a);
    FMM_CUDA(cudaEventRecord(f->ev[1], st), "FMM upward");

    // M2L walk, one depth of sinks per launch: every sink's tasks into a pool
    // of chunks (sizes are first guesses, or what the buffers hold from earlier
    // walks: a walk that runs out of one is repeated with twice the size; only the
    // buffers outlive the call)
    int *head = (int *)f->counts.p, *len = head + nsink;
    if (!nnode) FMM_CUDA(cudaMemsetAsync(len, 0, sizeof(int) * (size_t)nsink, st), "FMM walk");
    WalkRun g;
    std::memset(&g, 0, sizeof(g));
    unsigned long long ntask = 0;
    if (nnode) {
        int sms = 0;
        FMM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, f->device), "FMM walk");
        const WalkLimits &lim = f->limits;
        int64_t list_cap = lim.list_chunks ? lim.list_chunks : 2 * (int64_t)nnode + walk_pool_slack(sms, nleaf);
        int64_t task_cap = lim.out_chunks ? lim.out_chunks : 3 * (int64_t)nsink / 2 + walk_pool_slack(sms, nsink);
        const size_t lists_held = std::min(f->lists[0].cap, f->lists[1].cap);
        list_cap = std::max(list_cap, (int64_t)(lists_held / walk_pool_bytes(1, kWalkChunk)));
        task_cap = std::max(task_cap, (int64_t)(f->tasks.cap / walk_pool_bytes(1, kWalkTaskChunk)));
        g.nnode = nnode;
        g.nleaf = nleaf;
        g.node_first = t->node_first;
        g.cutoff = cutoff;
        g.open_angle = open_angle;
        g.cut2 = (float)(cutoff * cutoff);
        g.th2 = walk_th2(open_angle);
        g.out_head = head;
        g.out_len = len;
        const size_t nbox = 2 * ((size_t)std::max(nleaf, nnode) + 1);
        FMM_TRY(grow(f->box, (sizeof(WalkBox) + sizeof(WalkBox32)) * nbox));
        FMM_TRY(grow(f->items, sizeof(WalkItem) * 2 * (size_t)nleaf));
        FMM_TRY(grow(f->walk_ctrl, sizeof(WalkCtrl)));
        g.box = (const WalkBox *)f->box.p;
        g.box32 = (const WalkBox32 *)(g.box + nbox);
        g.items[0] = (WalkItem *)f->items.p;
        g.items[1] = g.items[0] + nleaf;
        g.ctrl = (WalkCtrl *)f->walk_ctrl.p;
        const int depths = lim.depths ? std::min(lim.depths, kWalkLevels) : walk_first_depths(nleaf) + kWalkExtraDepths;
        bool by_sink = false;  // a deep tree (walk_sink_kernel)
        int stack_cap = kWalkSinkStack;
        for (;;) {
            const int sink_blocks = walk_sink_blocks(sms, nleaf, stack_cap);
            if (by_sink) {
                FMM_TRY(grow(f->lists[0], walk_sink_bytes(sink_blocks, stack_cap)));
                FMM_TRY(grow(f->lists[1], sizeof(int) * (size_t)nsink));
                FMM_TRY(grow(f->tails, sizeof(int) * (size_t)nsink));
            } else {
                for (int k = 0; k < 2; ++k) FMM_TRY(grow(f->lists[k], walk_pool_bytes(list_cap, kWalkChunk)));
            }
            for (int k = 0; k < 2; ++k) g.lists[k] = walk_pool(f->lists[k].p, list_cap, kWalkChunk);
            FMM_TRY(grow(f->tasks, walk_pool_bytes(task_cap, kWalkTaskChunk)));
            g.out = walk_pool(f->tasks.p, task_cap, kWalkTaskChunk);
            FMM_CUDA(cudaMemsetAsync(len, 0, sizeof(int) * (size_t)nsink, st), "FMM walk");
            FMM_CUDA(cudaMemsetAsync(g.ctrl, 0, sizeof(WalkCtrl), st), "FMM walk");
            walk_pack_kernel<true><<<blocks_for((long long)nnode + nleaf, threads), threads, 0, st>>>(
                a.w, (WalkBox *)f->box.p, (WalkBox32 *)((WalkBox *)f->box.p + nbox), nullptr, g.items[0], g.lists[0].ids, g.ctrl);
            int status = 0, lv = 0;
            std::vector<int> boxes;  // of each depth
            for (int n = walk_first_depths(nleaf);; n = 4) {
                n = by_sink ? 0 : std::min(n, depths - lv);
                if (by_sink)
                    FMM_CUDA(walk_sinks<WALK_M2L>(st, g, t->son, (int *)f->lists[1].p, sink_blocks, (int2 *)f->lists[0].p,
                                                  stack_cap, (int *)f->tails.p), "FMM walk");
                else
                    FMM_CUDA(walk_depths<WALK_M2L>(st, g, sms, lv, n), "FMM walk");
                count_launches(by_sink ? 2 : n);
                lv += n;
                boxes.resize(lv + 1);
                FMM_CUDA(cudaMemcpyAsync(boxes.data(), g.ctrl->items, sizeof(int) * (lv + 1), cudaMemcpyDeviceToHost, st),
                         "FMM walk");
                FMM_CUDA(cudaMemcpyAsync(&status, &g.ctrl->status, sizeof(int), cudaMemcpyDeviceToHost, st), "FMM walk");
                FMM_CUDA(cudaMemcpyAsync(&ntask, &g.ctrl->ntask, sizeof(ntask), cudaMemcpyDeviceToHost, st), "FMM walk");
                FMM_CUDA(cudaStreamSynchronize(st), "FMM walk");
                if (status || by_sink || boxes[lv] == 0 || lv == depths) break;
            }
            if (status & ST_WALK_TREE) return report_error(P2P_ERR_ARG, "FMM: a child code outside the tree");
            if (status & ST_WALK_LONG)
                return report_error(P2P_ERR_CAPACITY, "FMM walk: a leaf's walk met more pairs than it may");
            if (!status && (by_sink || boxes[lv] == 0)) {
                f->levels = by_sink ? boxes[0] : lv - (int)std::count(boxes.begin(), boxes.begin() + lv, 0);
                break;
            }
            if (status & ST_WALK_LISTS) list_cap *= 2;
            if (status & ST_WALK_OUT) task_cap *= 2;
            if (std::max(list_cap, task_cap) > INT32_MAX)
                return report_error(P2P_ERR_CAPACITY, "FMM walk: more lists than a pool can hold");
            if (!by_sink) {
                by_sink = (status & ST_WALK_STACK) || !status;  // (boxes are left below the last depth)
            } else if (status & ST_WALK_STACK) {
                if (stack_cap > (1 << 28)) return report_error(P2P_ERR_CAPACITY, "FMM walk: a sink's walk exceeded its stack");
                stack_cap *= 2;
            }
        }
    }
    f->n_m2l = (long long)ntask;
    FMM_CUDA(cudaEventRecord(f->ev[2], st), "FMM walk");

    // M2L: each sink's sum over its tasks
    fmm_m2l_kernel<<<(int)std::min<long long>(((long long)nsink * kWalkTaskChunk + kM2LThreads - 1) / kM2LThreads, 148LL * 16),
                     kM2LThreads, 0, st>>>(a, head, len, g.out, ctrl + 2);
    FMM_CUDA(cudaEventRecord(f->ev[3], st), "FMM m2l");
    fmm_downward_kernel<<<blocks_for(nleaf, 128), 128, 0, st>>>(a, d_acc);
    FMM_CUDA(cudaEventRecord(f->ev[4], st), "FMM downward");
    FMM_CUDA(cudaGetLastError(), "FMM launch");
    unsigned long long h2[2];
    FMM_CUDA(cudaMemcpyAsync(h2, ctrl + 2, sizeof(h2), cudaMemcpyDeviceToHost, st), "FMM");
    FMM_CUDA(cudaStreamSynchronize(st), "FMM");
    f->n_applied = (long long)h2[0];
    count_launches(nnode ? 5 : 3);
    if ((int)h2[1] & ST_WALK_TREE) return report_error(P2P_ERR_ARG, "FMM: a child code outside the tree");
    return P2P_OK;
}

P2P_API int p2p_fmm_stats(p2p_fmm *f, int64_t *n_m2l, int64_t *n_applied, int *levels, float *ms) {
    if (!f) return report_error(P2P_ERR_ARG, "null argument");
    if (n_m2l) *n_m2l = f->n_m2l;
    if (n_applied) *n_applied = f->n_applied;
    if (levels) *levels = f->levels;
    if (ms) {
        cudaError_t e = cudaEventSynchronize(f->ev[4]);
        for (int k = 0; k < 4 && e == cudaSuccess; ++k) e = cudaEventElapsedTime(&ms[k], f->ev[k], f->ev[k + 1]);
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms[4], f->ev[0], f->ev[4]);
        if (e != cudaSuccess) return fail_cuda(e, "FMM timings");
    }
    return P2P_OK;
}

P2P_API int p2p_fmm_download(p2p_fmm *f, double *leaf_M, double *leaf_L) {
    if (!f) return report_error(P2P_ERR_ARG, "null argument");
    FMM_CUDA(cudaSetDevice(f->device), "cudaSetDevice");
    FMM_CUDA(cudaStreamSynchronize(f->stream), "FMM download");
    const size_t bytes = sizeof(double) * kNC * (size_t)f->nleaf;
    if (leaf_M && bytes) FMM_CUDA(cudaMemcpy(leaf_M, f->leafM.p, bytes, cudaMemcpyDeviceToHost), "FMM download");
    if (leaf_L && bytes) FMM_CUDA(cudaMemcpy(leaf_L, f->leafL.p, bytes, cudaMemcpyDeviceToHost), "FMM download");
    return P2P_OK;
}
