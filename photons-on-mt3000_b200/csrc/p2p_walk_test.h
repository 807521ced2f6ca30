// The pair test of the walks (acceptance, src/fmm.c:409-479, with LONGSHORT):
// in FP64 as the reference's C evaluates it, and a bound on it in FP32 that
// decides almost every pair from a 32-byte record per box.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define P2P_HD __host__ __device__ __forceinline__
#else
#define P2P_HD inline
#endif

namespace p2p {

// A box for the exact test.
struct alignas(64) WalkBox {
    double c[3], w[3];  // centre, width
    double sum;         // (w[0] + w[1]) + w[2], the opening rule's size
    double pad;
};

// The same rounded to FP32, with its children: one 32-byte access.
struct alignas(32) WalkBox32 {
    float c[3], w[3];
    int son[2];  // child codes (-1 for a leaf)
};

// What becomes of a pair of different boxes.
enum { WALK_DROP = -1, WALK_OPEN_B = 0, WALK_ACCEPT = 1, WALK_OPEN_A = 2, WALK_UNDECIDED = 3 };

// max(v, 0) that keeps NaN (fmaxf gives 0 and would leave a pair with a NaN gap to
// its other axes); one instruction on the device.
P2P_HD float walk_max0(float v) {
#ifdef __CUDA_ARCH__
    asm("max.NaN.f32 %0, %0, 0f00000000;" : "+f"(v));
    return v;
#else
    return v < 0.f ? 0.f : v;
#endif
}

// The pair (a, b) bounded in FP32: WALK_UNDECIDED unless the exact test's
// outcome is certain. a_node, b_node: the boxes are nodes (a larger node a is
// opened before b; a leaf is never opened). cut2, th2: the squares of cutoff
// and open angle rounded to FP32.
//
// Errors: a centre or width is rounded once (2^-24 of it) and each difference,
// sum and product again, so one axis's gap |dist| - width is off by less than
// slack = 2^-21 (|ca| + |cb| + wa + wb); squares and sums of bounds, and the two
// constants, by less than 1e-6 of themselves. A gap bounded to be at most zero
// is zero in the exact test too. An open angle whose square vanishes in FP32 is
// not 0: th2 is then passed as the smallest normal number. A pair with NaN or
// infinity in either box is undecided: its gap's bounds are NaN on that axis, which
// walk_max0 keeps, and no comparison with their sums holds.
P2P_HD int walk_bound(const WalkBox32 &a, const WalkBox32 &b, bool a_node, bool b_node, float cut2, float th2) {
    constexpr float kSlack = 4.76837158e-7f, kUp = 1.0f + 2.0e-6f, kDown = 1.0f - 2.0e-6f;
    float dist[3], w[3], slack[3], lo2 = 0.f, hi2 = 0.f, lo1 = 0.f;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int d = 0; d < 3; ++d) {
        dist[d] = fabsf(a.c[d] - b.c[d]);
        w[d] = (a.w[d] + b.w[d]) * 0.5f;
        slack[d] = kSlack * (fabsf(a.c[d]) + fabsf(b.c[d]) + 2.0f * w[d]);
        const float gap = dist[d] - w[d];
        const float lo = walk_max0(gap - slack[d]), hi = walk_max0(gap + slack[d]);
        lo1 += lo;
        lo2 += lo * lo;
        hi2 += hi * hi;
    }
    if (lo2 * kDown > cut2 * kUp && lo1 > 1.0e-14f) return WALK_DROP;
    if (!(hi2 * kUp < cut2 * kDown)) return WALK_UNDECIDED;
    // not dropped: accepted (never at open angle 0) or opened
    if (th2 > 0.f) {
        float d2lo = 0.f, d2hi = 0.f, wlo = 0.f, whi = 0.f;
#ifdef __CUDACC__
#pragma unroll
#endif
        for (int d = 0; d < 3; ++d) {
            const float dl = fmaxf(dist[d] - slack[d], 0.f), dh = dist[d] + slack[d];
            d2lo += dl * dl;
            d2hi += dh * dh;
            wlo = fmaxf(wlo, w[d] - slack[d]);
            whi = fmaxf(whi, w[d] + slack[d]);
        }
        const float t_lo = 2.f * wlo, t_hi = 2.f * whi, most = th2 * d2hi * kUp;
        if (t_hi * t_hi * kUp < th2 * d2lo * kDown && lo1 > 1.0e-14f) return WALK_ACCEPT;
        if (!(t_lo * t_lo * kDown >= most) || !(most < 3.0e38f)) return WALK_UNDECIDED;  // (an overflow decides nothing)
    }
    if (!a_node) return WALK_OPEN_B;
    if (!b_node) return WALK_OPEN_A;
    const float sa = a.w[0] + a.w[1] + a.w[2], sb = b.w[0] + b.w[1] + b.w[2];
    if (sa * kDown > sb * kUp) return WALK_OPEN_A;
    if (sa * kUp < sb * kDown) return WALK_OPEN_B;
    return WALK_UNDECIDED;
}

}  // namespace p2p
