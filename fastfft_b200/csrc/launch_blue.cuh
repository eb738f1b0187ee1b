// Launchers of the chirp-z passes for one power-of-two length M, instantiated in launch_blue.cu
// (M up to 512), launch_blue_2k.cu (1024, 2048), launch_blue_4k.cu and launch_blue_8k.cu: separate
// translation units, because one holding all of them took far longest to compile.
#pragma once

#include "kernels_blue.cuh"
#include "launch_common.cuh"

namespace ffb {
namespace blue {

template <int M>
constexpr size_t blue_smem() {
    return (size_t)FftGroup<M, 1, true>::BYTES;
}

template <int M, class InT>
cudaError_t r2c_impl(const RowFwdArgs& a, const BlueArgs& b, cudaStream_t st) {
    static std::atomic<int> hw[64];
    auto fn = blue_r2c_rows_kernel<M, InT>;
    cudaError_t e = ensure_smem_at_least((const void*)fn, blue_smem<M>(), hw);
    if (e != cudaSuccess) return e;
    const int grid = (a.n_rows + 1) / 2;
    if (grid == 0) return cudaSuccess;
    return launch_dependent(fn, dim3(grid, a.n_batch), M / 16, blue_smem<M>(), st, a, b);
}

template <int M, class OutT>
cudaError_t c2r_impl(const RowInvArgs& a, const BlueArgs& b, cudaStream_t st) {
    static std::atomic<int> hw[64];
    auto fn = blue_c2r_rows_kernel<M, OutT>;
    cudaError_t e = ensure_smem_at_least((const void*)fn, blue_smem<M>(), hw);
    if (e != cudaSuccess) return e;
    const int grid = (a.n_rows + 1) / 2;
    if (grid == 0) return cudaSuccess;
    return launch_dependent(fn, dim3(grid, a.n_batch), M / 16, blue_smem<M>(), st, a, b);
}

template <int M, class InC>
cudaError_t c2c_fwd_impl(const RowFwdArgs& a, const BlueArgs& b, cudaStream_t st) {
    static std::atomic<int> hw[64];
    auto fn = blue_c2c_rows_fwd_kernel<M, InC>;
    cudaError_t e = ensure_smem_at_least((const void*)fn, blue_smem<M>(), hw);
    if (e != cudaSuccess) return e;
    if (a.n_rows == 0) return cudaSuccess;
    return launch_dependent(fn, dim3(a.n_rows, a.n_batch), M / 16, blue_smem<M>(), st, a, b);
}

template <int M, class OutC>
cudaError_t c2c_inv_impl(const RowInvArgs& a, const BlueArgs& b, cudaStream_t st) {
    static std::atomic<int> hw[64];
    auto fn = blue_c2c_rows_inv_kernel<M, OutC>;
    cudaError_t e = ensure_smem_at_least((const void*)fn, blue_smem<M>(), hw);
    if (e != cudaSuccess) return e;
    if (a.n_rows == 0) return cudaSuccess;
    return launch_dependent(fn, dim3(a.n_rows, a.n_batch), M / 16, blue_smem<M>(), st, a, b);
}

template <int M, int MODE, class InC, class ImgC, class OutC>
cudaError_t cols_impl(const ColArgs& a, const BlueArgs& b, cudaStream_t st) {
    static std::atomic<int> hw[64];
    auto fn = blue_cols_kernel<M, MODE, InC, ImgC, OutC>;
    cudaError_t e = ensure_smem_at_least((const void*)fn, blue_smem<M>(), hw);
    if (e != cudaSuccess) return e;
    if (a.n_cols == 0) return cudaSuccess;
    return launch_dependent(fn, dim3(a.n_cols, a.n_batch), M / 16, blue_smem<M>(), st, a, b);
}

template <int M>
cudaError_t r2c_m(int in_dtype, const RowFwdArgs& a, const BlueArgs& b, cudaStream_t st) {
    switch (in_dtype) {
        case 0: return r2c_impl<M, float>(a, b, st);
        case 1: return r2c_impl<M, __half>(a, b, st);
        case 2: return r2c_impl<M, __nv_bfloat16>(a, b, st);
        default: return cudaErrorInvalidValue;
    }
}
template <int M>
cudaError_t c2r_m(int out_dtype, const RowInvArgs& a, const BlueArgs& b, cudaStream_t st) {
    switch (out_dtype) {
        case 0: return c2r_impl<M, float>(a, b, st);
        case 1: return c2r_impl<M, __half>(a, b, st);
        case 2: return c2r_impl<M, __nv_bfloat16>(a, b, st);
        default: return cudaErrorInvalidValue;
    }
}
// complex storage: 3 float2, 4 __half2, 5 __nv_bfloat162
template <int M>
cudaError_t c2c_fwd_m(int in_dtype, const RowFwdArgs& a, const BlueArgs& b, cudaStream_t st) {
    switch (in_dtype) {
        case 3: return c2c_fwd_impl<M, float2>(a, b, st);
        case 4: return c2c_fwd_impl<M, __half2>(a, b, st);
        case 5: return c2c_fwd_impl<M, __nv_bfloat162>(a, b, st);
        default: return cudaErrorInvalidValue;
    }
}
template <int M>
cudaError_t c2c_inv_m(int out_dtype, const RowInvArgs& a, const BlueArgs& b, cudaStream_t st) {
    switch (out_dtype) {
        case 3: return c2c_inv_impl<M, float2>(a, b, st);
        case 4: return c2c_inv_impl<M, __half2>(a, b, st);
        case 5: return c2c_inv_impl<M, __nv_bfloat162>(a, b, st);
        default: return cudaErrorInvalidValue;
    }
}
// dtype: the output storage (FWD), the input storage (INV) or the image storage (XCORR), as the
// power-of-two column launchers take it
template <int M>
cudaError_t cols_m(int mode, int dtype, const ColArgs& a, const BlueArgs& b, cudaStream_t st) {
    if (mode == COL_FWD) {
        switch (dtype) {
            case 3: return cols_impl<M, COL_FWD, float2, float2, float2>(a, b, st);
            case 4: return cols_impl<M, COL_FWD, float2, float2, __half2>(a, b, st);
            case 5: return cols_impl<M, COL_FWD, float2, float2, __nv_bfloat162>(a, b, st);
            default: return cudaErrorInvalidValue;
        }
    }
    if (mode == COL_INV) {
        switch (dtype) {
            case 3: return cols_impl<M, COL_INV, float2, float2, float2>(a, b, st);
            case 4: return cols_impl<M, COL_INV, __half2, float2, float2>(a, b, st);
            case 5: return cols_impl<M, COL_INV, __nv_bfloat162, float2, float2>(a, b, st);
            default: return cudaErrorInvalidValue;
        }
    }
    switch (dtype) {
        case 3: return cols_impl<M, COL_XCORR, float2, float2, float2>(a, b, st);
        case 4: return cols_impl<M, COL_XCORR, float2, __half2, float2>(a, b, st);
        case 5: return cols_impl<M, COL_XCORR, float2, __nv_bfloat162, float2>(a, b, st);
        default: return cudaErrorInvalidValue;
    }
}


#define FFB_BLUE_LAUNCHERS(EXT, M)                                                                          \
    EXT template cudaError_t r2c_m<M>(int, const RowFwdArgs&, const BlueArgs&, cudaStream_t);               \
    EXT template cudaError_t c2r_m<M>(int, const RowInvArgs&, const BlueArgs&, cudaStream_t);               \
    EXT template cudaError_t c2c_fwd_m<M>(int, const RowFwdArgs&, const BlueArgs&, cudaStream_t);           \
    EXT template cudaError_t c2c_inv_m<M>(int, const RowInvArgs&, const BlueArgs&, cudaStream_t);           \
    EXT template cudaError_t cols_m<M>(int, int, const ColArgs&, const BlueArgs&, cudaStream_t);

}  // namespace blue
}  // namespace ffb
