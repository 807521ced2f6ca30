// FP64 pair kernel for passes with a cutoff (pair_fp64_kernel).
//
// The general kernel (pair_plain_kernel) evaluates rsqrt, a division, erfc and
// exp per pair: 183 FP64 flops, 62% of the FP64 pipe at 256^3 and one warp per
// sink leaf, so small passes wait for their longest row. Here
//   - the pair factor comes from the polynomials of p2p_fit64.h: 28 FP64
//     instructions for a near pair, 50 for a far one, 6 for one beyond the
//     cutoff. Their coefficients are the same for every lane, so they are
//     operands from the constant bank; a table of short polynomials per region
//     needs half the instructions but a gathered shared-memory load for each
//     coefficient, whose bank conflicts made it slower (65^3: 12.9 ms);
//   - near, inside and beyond are decided on the high word of r^2, off the
//     FP64 pipe; a warp whose pairs are all near, or all beyond, skips the rest.
//     Half of the instructions were not FP64, and issue and the FP64 pipe were
//     about equally busy (58% and 54%), so those count too: the decisions by
//     minima over the lane's pairs, a clamp that runs only where a pair is near
//     the softening and 32-bit shared addresses took a 65^3 pass from 10.5 to
//     9.5 ms (33 ms in the general kernel);
//   - a lane keeps four sinks in registers (the sink-register layout of the
//     FP32 forms: G = ceil(ns / 4) groups of sinks, J = 32 / G source phases),
//     so a source read from shared memory serves four independent chains;
//   - the row's sources are copied into shared memory asynchronously
//     (cp.async, 8 bytes a lane and coordinate) one chunk ahead of the chunk
//     being evaluated;
//   - the warps of a block share one sink leaf's row, each a contiguous share
//     of its entries, and their partial sums are added in warp and phase
//     order: a row takes a quarter of the time at four warps, and the result
//     repeats bit for bit; with leaf_warps = -P (few leaves) P blocks share a
//     row, their sums in P arrays that sum_parts_kernel adds in order.
// Pairs whose r^2 has the cutoff's high word, and those with r^2 not finite, go
// through the general arithmetic (plain_factor), so which pairs are inside, and
// what NaN and infinity give, is decided exactly as there.
#pragma once

#include "p2p_fit64.h"
#include "p2p_launch.h"
#include "p2p_pair_kernels.cuh"

namespace p2p {

constexpr int kFp64Sinks = 4;  // sinks per lane

// The general kernel's factor of one pair, from r2 = |d|^2 + eps^2 (Plummer) or
// max(|d|^2, eps^2) (clamp); keep = false beyond the cutoff.
template <int SOFT>
__device__ __noinline__ double plain_factor(const double r2, const PairArgs &a, bool &keep) {
    double dr, drs;
    if (SOFT == SOFT_CLAMP) {
        dr = a.soft;
        if (r2 > a.soft * a.soft) dr = rsqrt(r2) * r2;
        drs = dr * a.hrrs;
    } else {
        dr = sqrt(r2);
        drs = 0.5 * dr * a.rrs;
    }
    keep = !(drs > a.xcut);
    return 1.0 / (dr * dr * dr) * (erfc(drs) + a.coeff * drs * exp(-drs * drs));
}

struct Fp64Lane {
    double px[kFp64Sinks], py[kFp64Sinks], pz[kFp64Sinks];
    double ax[kFp64Sinks], ay[kFp64Sinks], az[kFp64Sinks];
};

// 1 / sqrt(v) for v in the normal range: the hardware's approximation (about
// 2^-20) and one step of Householder's third-order iteration for y^-2 = v.
__device__ __forceinline__ double fp64_rsqrt(const double v) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    const double h = fma(-(v * y), y, 1.0);
    return fma(y * h, fma(h, 0.375, 0.5), y);
}

__device__ __forceinline__ unsigned fp64_hi(const double v) { return (unsigned)__double2hiint(v); }

// One source against the lane's sinks.
template <int SOFT, bool MASSES, int NF>
__device__ __forceinline__ void fp64_eval(const double sx, const double sy, const double sz, const double sw,
                                          Fp64Lane &L, const PairArgs &a, const Fit64 &F) {
    constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer
    constexpr int N = kFp64Sinks;
    double dx[N], dy[N], dz[N], r2[N];
    // Which kinds of pair there are, from the least and largest high words: a
    // minimum of (high word - start of a range) below the range's length says
    // that one lies in it. Two predicates and a combination a pair and kind, and
    // a 64-bit maximum a pair for the clamp, were a sixth of the instructions.
    unsigned least = 0xffffffffu, most = 0u;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        dx[k] = sx - L.px[k];
        dy[k] = sy - L.py[k];
        dz[k] = sz - L.pz[k];
        if (SOFT == SOFT_CLAMP)
            r2[k] = fma(dz[k], dz[k], fma(dy[k], dy[k], dx[k] * dx[k]));
        else
            r2[k] = fma(dz[k], dz[k], fma(dy[k], dy[k], fma(dx[k], dx[k], a.eps2_box)));
        least = min(least, fp64_hi(r2[k]));
        most = max(most, fp64_hi(r2[k]));
    }
    if (SOFT == SOFT_CLAMP && (least <= fp64_hi(a.eps2_box) || most >= 0x7ff00000u)) {
        least = 0xffffffffu;
        most = 0u;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            r2[k] = fmax(r2[k], a.eps2_box);
            least = min(least, fp64_hi(r2[k]));
            most = max(most, fp64_hi(r2[k]));
        }
    }
    unsigned past_near = 0xffffffffu, past_in = 0xffffffffu;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        past_near = min(past_near, fp64_hi(r2[k]) - F.hi_near);
        past_in = min(past_in, fp64_hi(r2[k]) - F.hi_in);
    }
    const bool near = least < F.hi_near, far = past_near < F.hi_in - F.hi_near;
    if (past_in <= F.hi_out - F.hi_in || most >= 0x7ff00000u) {  // rare
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const unsigned hi = fp64_hi(r2[k]);
            if (!(hi >= F.hi_in && (hi <= F.hi_out || hi >= 0x7ff00000u))) continue;
            bool keep;
            double f = plain_factor<SOFT>(r2[k], a, keep);
            if (keep) {
                if (MASSES) f *= sw;
                L.ax[k] = fma(dx[k], f, L.ax[k]);
                L.ay[k] = fma(dy[k], f, L.ay[k]);
                L.az[k] = fma(dz[k], f, L.az[k]);
            }
            dx[k] = dy[k] = dz[k] = 0.0;  // (an infinite one times the zero below would be NaN)
        }
    }
    if (near || far) {
        double y[N], p[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
            y[k] = fp64_rsqrt(r2[k]);
            p[k] = 0.0;
        }
        if (near) {
            double q[N];
#pragma unroll
            for (int k = 0; k < N; ++k) q[k] = F.near[kFit64Near - 1];
#pragma unroll
            for (int c = kFit64Near - 2; c >= 0; --c)
#pragma unroll
                for (int k = 0; k < N; ++k) q[k] = fma(q[k], r2[k] - F.near_mid, F.near[c]);
#pragma unroll
            for (int k = 0; k < N; ++k) {
                double f = fma(y[k] * y[k], y[k], q[k]);
                if (MASSES) f *= sw;
                p[k] = fp64_hi(r2[k]) < F.hi_near ? f : 0.0;
            }
        }
        if (far) {
            double f[N], e[N], q[N];
            int n[N];
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const double m = fma(r2[k], F.e_hi, kMagic), whole = m - kMagic;
                n[k] = __double2loint(m);
                f[k] = fma(r2[k], F.e_lo, fma(r2[k], F.e_hi, -whole));
                e[k] = F.exp2[kFit64Exp - 1];
            }
#pragma unroll
            for (int c = kFit64Exp - 2; c >= 0; --c)
#pragma unroll
                for (int k = 0; k < N; ++k) e[k] = fma(e[k], f[k], F.exp2[c]);
#pragma unroll
            for (int k = 0; k < N; ++k) {
                f[k] = fma(r2[k], y[k], -F.far_mid);
                q[k] = F.far[NF - 1];
            }
#pragma unroll
            for (int c = NF - 2; c >= 0; --c)
#pragma unroll
                for (int k = 0; k < N; ++k) q[k] = fma(q[k], f[k], F.far[c]);
#pragma unroll
            for (int k = 0; k < N; ++k) {
                // 2^n by the exponent field: a far pair's n lies in [-24, -1], so nothing leaves
                // the normal range; what other lanes make of it is not used
                e[k] = __hiloint2double(__double2hiint(e[k]) + (n[k] << 20), __double2loint(e[k]));
                double v = (y[k] * y[k]) * y[k] * (e[k] * q[k]);
                if (MASSES) v *= sw;
                p[k] = fp64_hi(r2[k]) - F.hi_near < F.hi_in - F.hi_near ? v : p[k];
            }
        }
#pragma unroll
        for (int k = 0; k < N; ++k) {
            L.ax[k] = fma(dx[k], p[k], L.ax[k]);
            L.ay[k] = fma(dy[k], p[k], L.ay[k]);
            L.az[k] = fma(dz[k], p[k], L.az[k]);
        }
    }
}

__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

__device__ __forceinline__ double load_shared(const unsigned at) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
    return v;
}

// Shared memory of one warp: two chunks of cap / 2 sources (x, y, z and mass
// rows), the partial sums of its lanes' sinks.
__host__ __device__ constexpr size_t fp64_warp_bytes(int cap) {
    return (size_t)cap * 4 * sizeof(double) + (size_t)32 * 3 * kFp64Sinks * sizeof(double);
}

template <int SOFT, bool MASSES, int NF>
__global__ void __launch_bounds__(256, 2)
pair_fp64_kernel(const __grid_constant__ PairArgs a, const __grid_constant__ Fit64 F, const int cap) {
    extern __shared__ double smem_d[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int wdoubles = (int)(fp64_warp_bytes(cap) / sizeof(double));
    double *const wbase = smem_d + w * wdoubles;
    const unsigned wshared = (unsigned)__cvta_generic_to_shared(wbase);
    const int chunk = cap / 2;
    double *const sums = wbase + 4 * (size_t)cap;  // [component and sink][lane]
    __shared__ int s_item;
    const int parts = a.leaf_warps < 0 ? -a.leaf_warps : 1;  // blocks sharing a row, each with sums of its own
    const size_t n3 = 3 * (size_t)a.npart;
    const double *X = a.pos, *Y = a.pos + a.npart, *Z = a.pos + 2 * (size_t)a.npart;
    for (;;) {
        __syncthreads();  // the previous item is read
        if (threadIdx.x == 0) s_item = atomicAdd(a.queue, 1);
        __syncthreads();
        const int item = s_item;
        if (item >= a.nleaf * parts) break;
        const int li = item_leaf(a, item / parts, lane), part = item % parts;
        const int64_t r0 = a.row_off[li], len = a.row_off[li + 1] - r0;
        if (len <= 0) continue;
        // this warp's contiguous share of the row's entries
        const int64_t shares = (int64_t)parts * W, share = (int64_t)part * W + w;
        const int64_t rb = r0 + len * share / shares, re = r0 + len * (share + 1) / shares;
        const LeafMeta mt = a.leaf[li];
        for (int s0 = 0; s0 < mt.npart; s0 += 8 * kFp64Sinks) {
            const int ns = min(8 * kFp64Sinks, mt.npart - s0);
            const int G = (ns + kFp64Sinks - 1) / kFp64Sinks, J = 32 / G;
            const int g = lane % G, jl = lane / G;
            const int first = mt.ipart + s0;
            Fp64Lane L;
#pragma unroll
            for (int k = 0; k < kFp64Sinks; ++k) {
                const int i = first + min(kFp64Sinks * g + k, ns - 1);
                L.px[k] = X[i];
                L.py[k] = Y[i];
                L.pz[k] = Z[i];
                L.ax[k] = L.ay[k] = L.az[k] = 0.0;
            }
            // the row's entries in batches of 32 (this lane's entry: particle
            // range), the next batch's loaded while the current one is used
            int64_t e0 = rb;
            int sip = 0, snp = 0, nip = 0, nnp = 0, incl = 0, total = 0, done = 0;
            auto load_batch = [&]() {
                nip = nnp = 0;
                if (e0 + lane < re) {
                    const LeafMeta *m = a.leaf + a.row_src[e0 + lane];
                    nip = m->ipart;
                    nnp = m->npart;
                }
            };
            // copies the row's next (up to chunk) sources into buf; returns their number
            auto fill = [&](double *buf) {
                int n = 0;
                while (n < chunk) {
                    if (done >= total) {
                        if (e0 >= re) break;
                        sip = nip;
                        snp = nnp;
                        e0 += 32;
                        load_batch();
                        incl = snp;
#pragma unroll
                        for (int off = 1; off < 32; off <<= 1) {
                            const int up = __shfl_up_sync(kFull, incl, off);
                            if (lane >= off) incl += up;
                        }
                        total = __shfl_sync(kFull, incl, 31);
                        done = 0;
                        continue;
                    }
                    const int take = min(min(32, chunk - n), total - done);
                    const int q = done + min(lane, take - 1);
                    int e = 0;  // the entry of source q: the first whose inclusive prefix exceeds it
#pragma unroll
                    for (int st = 16; st > 0; st >>= 1) {
                        const int probe = __shfl_sync(kFull, incl, e + st - 1);
                        if (probe <= q) e += st;
                    }
                    const int i = __shfl_sync(kFull, sip, e) +
                                  (q - (__shfl_sync(kFull, incl, e) - __shfl_sync(kFull, snp, e)));
                    if (lane < take) {
                        cp_async8(buf + n + lane, X + i);
                        cp_async8(buf + chunk + n + lane, Y + i);
                        cp_async8(buf + 2 * chunk + n + lane, Z + i);
                        if (MASSES) cp_async8(buf + 3 * chunk + n + lane, a.mass + i);
                    }
                    n += take;
                    done += take;
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                return n;
            };
            load_batch();
            int b = 0;
            int n = fill(wbase);
            while (n > 0) {
                const int next = fill(wbase + (b ^ 1) * 4 * chunk);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                __syncwarp();  // every lane's copies of this chunk have landed
                if (jl < J) {
                    // a 32-bit shared address: a generic pointer's was made anew for every source
                    const unsigned row = 8u * chunk, buf = wshared + 4u * row * b, end = buf + 8u * n;
#pragma unroll 1
                    for (unsigned at = buf + 8u * jl; at < end; at += 8u * J)
                        fp64_eval<SOFT, MASSES, NF>(load_shared(at), load_shared(at + row), load_shared(at + 2 * row),
                                                    MASSES ? load_shared(at + 3 * row) : 0.0, L, a, F);
                }
                __syncwarp();  // the chunk is read before the copies after next overwrite it
                n = next;
                b ^= 1;
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
            for (int k = 0; k < kFp64Sinks; ++k) {
                sums[(3 * k + 0) * 32 + lane] = L.ax[k];
                sums[(3 * k + 1) * 32 + lane] = L.ay[k];
                sums[(3 * k + 2) * 32 + lane] = L.az[k];
            }
            __syncthreads();
            for (int q = threadIdx.x; q < 3 * ns; q += blockDim.x) {
                const int c = q / ns, sk = q - c * ns;
                const int row = (3 * (sk % kFp64Sinks) + c) * 32 + sk / kFp64Sinks;
                double v = 0.0;
                for (int ww = 0; ww < W; ++ww) {
                    const double *ws = smem_d + ww * wdoubles + 4 * (size_t)cap + row;
                    for (int jj = 0; jj < J; ++jj) v += ws[jj * G];
                }
                double *o = a.acc + n3 * part + (size_t)c * a.npart + first + sk;
                v = MASSES ? v : v * a.mass_eq;
                *o = parts > 1 ? v : *o + v;
            }
            __syncthreads();  // the sums are read before the next slice writes its own
        }
    }
}

}  // namespace p2p
