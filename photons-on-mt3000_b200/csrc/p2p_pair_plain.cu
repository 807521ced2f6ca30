// Launcher of the FP64 drop-in pair kernels: pair_fp64_kernel where the pass
// has a fitted cutoff (PairLaunch::fit64), else pair_plain_kernel (no cutoff,
// or a cutoff or softening outside the fit's range).
#include "p2p_launch.h"
#include "p2p_pair_fp64.cuh"
#include "p2p_pair_kernels.cuh"

namespace p2p {
namespace {

template <int SOFT, bool MASSES, int NF>
PairLaunchResult launch_fp64(const PairLaunch &L, const PairArgs &a) {
    PairLaunchResult r;
    // (two chunks of up to 128 sources: a larger stage would only take shared memory)
    const int stage = L.stage < 256 ? L.stage : 256;
    const size_t smem = pair_smem_fp64(L.warps, stage);
    if (!persistent_blocks(L, pair_fp64_kernel<SOFT, MASSES, NF>, smem, r) || L.dry_run) return r;
    pair_fp64_kernel<SOFT, MASSES, NF><<<r.blocks, L.warps * 32, smem, L.stream>>>(a, *L.fit64, stage);
    r.cuda = cudaGetLastError();
    return r;
}

template <int SOFT, bool MASSES>
PairLaunchResult by_form(const PairLaunch &L, const PairArgs &a) {
    switch (L.fit64 ? L.fit64->nfar : 0) {
        case 17: return launch_fp64<SOFT, MASSES, 17>(L, a);
        case 19: return launch_fp64<SOFT, MASSES, 19>(L, a);
        case 22: return launch_fp64<SOFT, MASSES, 22>(L, a);
        case 25: return launch_fp64<SOFT, MASSES, 25>(L, a);
        default: return launch_persistent(L, pair_plain_kernel<SOFT, MASSES>, pair_smem_plain(L.warps, L.stage), a);
    }
}

template <int SOFT, bool MASSES>
cudaError_t allow_one() {
    const void *ks[] = {(const void *)pair_plain_kernel<SOFT, MASSES>,
                        (const void *)pair_fp64_kernel<SOFT, MASSES, 17>,
                        (const void *)pair_fp64_kernel<SOFT, MASSES, 19>,
                        (const void *)pair_fp64_kernel<SOFT, MASSES, 22>,
                        (const void *)pair_fp64_kernel<SOFT, MASSES, 25>};
    cudaError_t e = cudaSuccess;
    for (const void *k : ks) {
        // the opt-in limit covers static and dynamic shared memory together
        cudaFuncAttributes fa;
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     227 * 1024 - (int)fa.sharedSizeBytes);
    }
    return e;
}

}  // namespace

PairLaunchResult launch_pair_plain(const PairLaunch &L, const PairArgs &a) {
    if (L.soft_mode == SOFT_CLAMP)
        return L.masses ? by_form<SOFT_CLAMP, true>(L, a) : by_form<SOFT_CLAMP, false>(L, a);
    return L.masses ? by_form<SOFT_PLUMMER, true>(L, a) : by_form<SOFT_PLUMMER, false>(L, a);
}

cudaError_t allow_smem_plain() {
    cudaError_t e = allow_one<SOFT_CLAMP, false>();
    if (e == cudaSuccess) e = allow_one<SOFT_CLAMP, true>();
    if (e == cudaSuccess) e = allow_one<SOFT_PLUMMER, false>();
    if (e == cudaSuccess) e = allow_one<SOFT_PLUMMER, true>();
    return e;
}

}  // namespace p2p
