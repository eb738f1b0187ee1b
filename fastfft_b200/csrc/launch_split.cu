// Launcher of the batched fused correlation column pass on the split block FFT
// (xcorr_split_kernel in kernels_xcorr.cuh).
#include "kernels_xcorr.cuh"
#include "launch_common.cuh"

namespace ffb {

template <int N, class C, int G, int MIN_BLOCKS>
static cudaError_t xcorr_split_impl(const XcorrColArgs& a, cudaStream_t st) {
    static_assert(XcorrSplitSmem<N, C, G>::total(N) <= 227 * 1024, "fits for every template height");
    const int smem = XcorrSplitSmem<N, C, G>::total(a.L);
    static std::atomic<int> high_water[64];
    auto fn = xcorr_split_kernel<N, C, G, MIN_BLOCKS>;
    cudaError_t e = ensure_smem_at_least((const void*)fn, (size_t)smem, high_water);
    if (e != cudaSuccess) return e;
    return launch_dependent(fn, dim3(a.n_cols, (a.n_batch + a.tpb - 1) / a.tpb), SplitFft<N, C>::T * G, smem, st, a);
}

// Whether three blocks of the pair, its occupancy by registers, fit on an SM at template height L
// (228 KB of shared memory, 1 KB of it per block kept by the system).
template <int N, int G>
static bool pair_fits(int L) {
    return 3 * (XcorrSplitSmem<N, cpair, G>::total(L) + 1024) <= 228 * 1024;
}

// Blocks of G transform groups; registers for MIN_BLOCKS blocks per SM.  Measured on B200 (us per
// launch; "before": the radix-16 forms xcorr_cols_kernel / xcorr3_cols_kernel, which keep the
// other lengths):
//   length (template, window, templates)   before   single value   pair
//   1536 (384, 1024, 64)                     333    288 (2 x 4)    265 (2 x 3), 284 (3 x 2)
//   1536 (384, 1024, 12)                      85     65 (2 x 4)     67 (3 x 2)
//   1536 (384, 1024, 1)                     17.2   13.9 (1 x 8)   18.3 (1 x 6)
//   768  (256, 512, 64)                       90     80 (4 x 4)     80 (4 x 3)
//   384  (96, 256, 64)                      34.2   25.5 (4 x 8)   26.4 (4 x 6)
//   1024 (384, 512, 32)                     69.6   66.1 (2 x 4)   70.3 (2 x 3)
//   512  (150, 300, 32)                     25.4   20.6 (4 x 4)   23.4 (4 x 3)
//   256  (60, 128, 32)                      12.0    9.7 (8 x 5)    9.9 (8 x 3)
//   2048 (500, 1100, 16)                     159    136 (1 x 4)    129 (1 x 3)
// The single form at 128 registers (16 warps per SM) is the better one at most lengths (at 96 it
// spills: 382 us at 1536); at 2048, and at 1536 once a launch holds 16 templates, the pair is (168
// registers, 12 warps), while its staged columns leave room for three blocks: up to 448 template
// rows at 1536 and 1600 at 2048.  Above, two blocks (8 warps) are the slower form (us per launch, pair
// / single, same length and launch size, the window filling the length; both are flat on either
// side of the line):
//   1536, L = 448:  79.3 / 82.0 (16 templates)  151.9 / 154.2 (32)  277 / 294 (64)
//   1536, L = 449:  89.2 / 81.9                 167.4 / 154.8       316 / 295
//   1536, L = 1000: 89.5 / 86.0                 166.8 / 161.7       317 / 308
//   2048, L = 1000: 135.6 / 138.9 (16)          259 / 265 (32)
//   2048, L = 1590: 145.7 / 142.6               278 / 273
//   2048, L = 1610: 159.4 / 143.0               306 / 273
// Fewer than four templates take blocks of one group, so that no group
// idles.  At 1536 the pair's launch keeps the FP32 pipe 56 %, the shared-memory path 67 % and the
// issue slots 60 % busy at 3 warps per scheduler: bound by latency at that occupancy (before: 48,
// 75 and 71 %).  Spills per thread at 128 registers: 76 bytes at 1536 (2 x 4; 36 at 1 x 8), 32 at 2048,
// 20 at 768 (4 x 4); the pairs have none.  Both forms give the same bits (cpair.cuh), so the choice
// does not show in results.
cudaError_t launch_xcorr_split(int n, const XcorrColArgs& a0, cudaStream_t st) {
    XcorrColArgs a = a0;
    if (a.n_batch < 1 || a.n_batch > kMaxBatch || a.n_cols < 1 || a.L < 1 || a.L > n) return cudaErrorInvalidValue;
    if (a.tpb < 1 || a.tpb > a.n_batch) return cudaErrorInvalidValue;
    cudaError_t e = split_twiddles_for(n, &a.tw);
    if (e != cudaSuccess) return e;
    const bool few = a.n_batch < 4;
    switch (n) {
        case 256: return xcorr_split_impl<256, float2, 8, 5>(a, st);
        case 384: return xcorr_split_impl<384, float2, 4, 8>(a, st);
        case 512: return xcorr_split_impl<512, float2, 4, 4>(a, st);
        case 768:
            if (few) return xcorr_split_impl<768, float2, 1, 16>(a, st);
            return xcorr_split_impl<768, float2, 4, 4>(a, st);
        case 1024:
            if (few) return xcorr_split_impl<1024, float2, 1, 8>(a, st);
            return xcorr_split_impl<1024, float2, 2, 4>(a, st);
        case 1536:
            if (few) return xcorr_split_impl<1536, float2, 1, 8>(a, st);
            if (a.n_batch >= 16 && pair_fits<1536, 2>(a.L)) return xcorr_split_impl<1536, cpair, 2, 3>(a, st);
            return xcorr_split_impl<1536, float2, 2, 4>(a, st);
        case 2048:
            if (few || !pair_fits<2048, 1>(a.L)) return xcorr_split_impl<2048, float2, 1, 4>(a, st);
            return xcorr_split_impl<2048, cpair, 1, 3>(a, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ffb
