// Row passes on the split block FFT (fft_split.cuh): the same arguments, layouts and results as
// r2c_rows_kernel / c2r_rows_kernel (kernels_2d.cuh), two real rows per complex transform.
//
// Both are bound by the shared-memory path (72 - 77 % busy at 1536 points as three 512-point
// FFTs and a radix-3 step: eight passes of the data in the C2R).  Here the C2R takes six: the
// gathered spectrum goes to shared memory at the position from which the sub-FFT threads read it
// (frequency s + E kp at row kp of a padded stride), one exchange inside the sub-FFTs, one across
// the transform, and the outputs leave from registers.  The R2C is the same in reverse.
#pragma once

#include "fft_split.cuh"
#include "kernels_2d.cuh"

namespace ffb {

template <int N, int FPB>
struct SplitRows {
    using F = SplitFft<N, float2>;
    static constexpr int T = F::T, E = F::E;
    // rows of E frequencies at a stride that keeps the reads at freq_index free of conflicts
    static constexpr int STEP = F::B >= 8 ? 2 : 16 / F::B;
    static constexpr int IS = F::B == 1 || (E / STEP) % 2 ? E : E + STEP;
    // buffers of consecutive transforms start 16 / FPB elements apart modulo a wavefront: the
    // gather and the split walk FPB transforms at each frequency
    static constexpr int NEED = F::BUF > F::P * IS ? F::BUF : F::P * IS;
    static constexpr int STRIDE = (NEED + 15) / 16 * 16 + (FPB >= 16 ? 1 : FPB > 1 ? 16 / FPB : 0);
    static constexpr int BYTES = FPB * STRIDE * 8;
    static constexpr int ITEMS = (N / 2 + 1 + T - 1) / T;   // frequencies per thread
    static __device__ __forceinline__ int pos(int k) { return k + (IS - E) * (k / E); }
    // position of freq_index(j, e), as base + constant
    static __device__ __forceinline__ int base(int j) { return (j % F::B) * IS + j / F::B; }
    static __device__ __forceinline__ int offset(int e) {
        const int m = e / F::A, u = (e % F::A) / F::B, k2 = e % F::B;
        return (F::B * u + F::A * k2) * IS + F::SPT * m;
    }
};

// barrier of the T threads of transform f (in-warp, named, or the block's)
template <int T, int FPB>
__device__ __forceinline__ void split_sync(int f) {
    if constexpr (T <= 32) {
        __syncwarp();
    } else if constexpr (FPB > 1) {
        asm volatile("bar.sync %0, %1;" ::"r"(f + 1), "n"(T) : "memory");
    } else {
        __syncthreads();
    }
}

template <int N, class InT, int FPB, int MIN_BLOCKS>
__global__ void __launch_bounds__(SplitRows<N, FPB>::T * FPB, MIN_BLOCKS)
r2c_split_rows_kernel(RowFwdArgs a) {
    grid_dependency();
    using SR = SplitRows<N, FPB>;
    using F = typename SR::F;
    constexpr int T = SR::T, E = SR::E;
    extern __shared__ __align__(128) float2 smem[];
    const int f = threadIdx.x / T, j = threadIdx.x % T;
    float2* const s = smem + f * SR::STRIDE;
    // batch entries in reverse order, as r2c_rows_kernel
    const int gb = gridDim.y - 1 - blockIdx.y;
    const int n_rows = a.rows_g[gb] > 0 ? a.rows_g[gb] : a.n_rows;
    const int L = a.L_g[gb] > 0 ? a.L_g[gb] : a.L;
    const long long in_pitch = a.pitch_g[gb] > 0 ? a.pitch_g[gb] : a.in_pitch;
    if (2 * blockIdx.x * FPB >= n_rows) return;   // (block-uniform) an uneven batch's shorter template
    const int ra = 2 * (blockIdx.x * FPB + f);
    const InT* in_g = static_cast<const InT*>(a.in[gb]);
    const InT* pa = in_g + input_row(ra, a.rows_y, a.rows_z) * in_pitch;
    const InT* pb = in_g + input_row(ra + 1, a.rows_y, a.rows_z) * in_pitch;
    const int La = ra < n_rows ? L : 0, Lb = ra + 1 < n_rows ? L : 0;
    const int qn = (L + T - 1) / T;
    float2 v[E];
#pragma unroll
    for (int q = 0; q < E; q++) {
        const int n = j + T * q;
        v[q] = make_float2(0.f, 0.f);
        if (q < qn) v[q] = make_float2(n < La ? ld_real<InT>(pa + n) : 0.f, n < Lb ? ld_real<InT>(pb + n) : 0.f);
    }
    if (a.scale != 1.f) {
#pragma unroll
        for (int q = 0; q < E; q++) v[q] = cscale(v[q], a.scale);
    }
    F::forward(v, s, j, a.tw, qn, [&]() { split_sync<T, FPB>(f); });
    split_sync<T, FPB>(f);   // the last exchange has been read
    {
        float2* const d = s + SR::base(j);
#pragma unroll
        for (int e = 0; e < E; e++) d[SR::offset(e)] = v[e];
    }
    __syncthreads();
    // split Z = A + iB: A[k] = (Z[k] + conj Z[N-k]) / 2, B[k] = -i (Z[k] - conj Z[N-k]) / 2;
    // item it of this thread: frequency k0 + T it of transform ff0
    const int ff0 = threadIdx.x % FPB, k0 = threadIdx.x / FPB;
    const float2* sf = smem + ff0 * SR::STRIDE;
    const int rr0 = 2 * (blockIdx.x * FPB + ff0);
    const bool two = rr0 + 1 < n_rows, one = rr0 < n_rows;
    float2* o = a.out + (long long)gb * a.out_batch_stride + (long long)k0 * a.out_pitch + rr0;
    const long long step = (long long)T * a.out_pitch;
#pragma unroll
    for (int it = 0; it < SR::ITEMS; it++, o += step) {
        const int k = k0 + T * it;
        if (k >= a.kmax) continue;
        const float2 z1 = sf[SR::pos(k)];
        const float2 z2 = sf[SR::pos(k == 0 ? 0 : N - k)];
        const float2 A = make_float2(0.5f * (z1.x + z2.x), 0.5f * (z1.y - z2.y));
        const float2 B = make_float2(0.5f * (z1.y + z2.y), 0.5f * (z2.x - z1.x));
        if (two) {
            *reinterpret_cast<float4*>(o) = make_float4(A.x, A.y, B.x, B.y);
        } else if (one) {
            *o = A;
        }
    }
}

// PLAIN: windows written at origin 0, no peak search, no projection.
template <int N, class OutT, int FPB, int MIN_BLOCKS, bool PLAIN>
__global__ void __launch_bounds__(SplitRows<N, FPB>::T * FPB, MIN_BLOCKS)
c2r_split_rows_kernel(RowInvArgs a) {
    grid_dependency();
    using SR = SplitRows<N, FPB>;
    using F = typename SR::F;
    constexpr int T = SR::T, E = SR::E, H = N / 2;
    extern __shared__ __align__(128) float2 smem[];
    const int f = threadIdx.x / T, j = threadIdx.x % T;
    float2* const s = smem + f * SR::STRIDE;
    // batch entries in reverse order, as c2r_rows_kernel
    const int gb = gridDim.y - 1 - blockIdx.y;
    // gather Z[k] = A[k] + i B[k] over the full circle from the two rows' half spectra (the
    // imaginary parts of the k = 0 and k = N/2 bins are dropped); all of a thread's loads are in
    // flight before the first is used
    {
        const int ff0 = threadIdx.x % FPB, k0 = threadIdx.x / FPB;
        float4 ld[SR::ITEMS];
        const int rr0 = 2 * (blockIdx.x * FPB + ff0);
        const bool two = rr0 + 1 < a.n_rows, one = rr0 < a.n_rows;
        const float2* p = a.in + (long long)gb * a.in_batch_stride + (long long)k0 * a.in_pitch + rr0;
        const long long step = (long long)T * a.in_pitch;
#pragma unroll
        for (int it = 0; it < SR::ITEMS; it++, p += step) {
            ld[it] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k0 + T * it <= H) {
                if (two) {
                    ld[it] = *reinterpret_cast<const float4*>(p);
                } else if (one) {
                    const float2 x = *p;
                    ld[it] = make_float4(x.x, x.y, 0.f, 0.f);
                }
            }
        }
        float2* const sf = smem + ff0 * SR::STRIDE;
#pragma unroll
        for (int it = 0; it < SR::ITEMS; it++) {
            const int k = k0 + T * it;
            if (k > H) continue;
            const float2 A = make_float2(ld[it].x, ld[it].y), B = make_float2(ld[it].z, ld[it].w);
            if (k == 0 || k == H) {
                sf[SR::pos(k)] = make_float2(A.x, B.x);
            } else {
                sf[SR::pos(k)] = make_float2(A.x - B.y, A.y + B.x);
                sf[SR::pos(N - k)] = make_float2(A.x + B.y, B.x - A.y);
            }
        }
    }
    __syncthreads();
    float2 v[E];
    {
        const float2* const d = s + SR::base(j);
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = d[SR::offset(e)];
    }
    split_sync<T, FPB>(f);   // the exchanges reuse the buffer
    F::inverse(v, s, j, a.tw, [&]() { split_sync<T, FPB>(f); });
    if (a.scale != 1.f) {
#pragma unroll
        for (int q = 0; q < E; q++) v[q] = cscale(v[q], a.scale);
    }
    const int ra = 2 * (blockIdx.x * FPB + f);
    OutT* oa = static_cast<OutT*>(a.out[gb]) + (long long)ra * a.out_pitch;
    OutT* ob = oa + a.out_pitch;
    const int Wa = ra < a.n_rows ? a.W : 0, Wb = ra + 1 < a.n_rows ? a.W : 0;
    if constexpr (PLAIN) {
#pragma unroll
        for (int q = 0; q < E; q++) {
            const int n = j + T * q;
            if (n < Wa) st_real<OutT>(oa + n, v[q].x);
            if (n < Wb) st_real<OutT>(ob + n, v[q].y);
        }
    } else {
        const bool write = !a.peaks_only;
        unsigned long long best = 0;
        const unsigned int tmpl = (unsigned)(a.mip_base + a.peak_slot[gb]);
        unsigned long long* ma = a.mip ? a.mip + (long long)ra * a.W : nullptr;
#pragma unroll
        for (int q = 0; q < E; q++) {
            const int n = j + T * q - a.X0;
            if (n < 0 || n >= Wa) continue;
            if (write) {
                st_real<OutT>(oa + n, v[q].x);
                if (n < Wb) st_real<OutT>(ob + n, v[q].y);
            }
            if (ma) {
                atomicMax(ma + n, peak_key(v[q].x, tmpl));
                if (n < Wb) atomicMax(ma + a.W + n, peak_key(v[q].y, tmpl));
            }
            if (a.peaks) {
                const unsigned long long ka = peak_key(v[q].x, (unsigned)(ra * a.W + n));
                best = ka > best ? ka : best;
                if (n < Wb) {
                    const unsigned long long kb = peak_key(v[q].y, (unsigned)((ra + 1) * a.W + n));
                    best = kb > best ? kb : best;
                }
            }
        }
        if (a.peaks) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
                best = other > best ? other : best;
            }
            if ((threadIdx.x & 31) == 0 && best != 0) atomicMax(a.peaks + a.peak_slot[gb], best);
        }
    }
}

}  // namespace ffb
