// Fused cross-correlation column pass, batched over templates (sm_100a), in two forms:
// xcorr_split_kernel (below) at the lengths of the split block FFT (256 ... 2048 and 384 ... 1536),
// where it replaced the first one, and xcorr_cols_kernel at the other powers of two (16 ... 128,
// 4096; the other R * 2^k lengths are in kernels_fft3.cuh).  In the latter, one block per spectrum
// column kx serves the templates of a group:
//   - the image-spectrum column (N values) and the template row-pass columns (L values
//     per template) are brought into shared memory by TMA bulk copies
//     (cp.async.bulk ... mbarrier::complete_tx) issued by one thread, so the image
//     column is read once per batch instead of once per template;
//   - each FFT group of the block then runs, per template, the zero-padded forward
//     column FFT, the conj(T) * I intra-op against the shared image column, and the
//     inverse FFT, and stores the first W outputs;
// Replaces block_fft_kernel_C2C_FWD_INCREASE_OP_INV_NONE (src/fastfft/FastFFT.cu:20-56),
// which reloads the image column per template and zero-pads explicitly.
//
// The mbarrier wait is bounded: if the copies have not landed after kWaitLimit polls,
// the block records kErrTimeout in *err and returns without touching the outputs.
#pragma once

#include "fft_split.cuh"
#include "kernels_2d.cuh"
#include "tma.cuh"

namespace ffb {

struct XcorrColArgs {
    const float2* t1;          // template g, column c: t1 + g * t1_batch + c * t1_pitch (L valid values)
    long long t1_pitch;
    long long t1_batch;
    int L;
    const void* img;           // image column c: img + c * img_stride (ImgC elements)
    long long img_stride;
    float2* out;               // template g, column c: out + g * out_batch + c * out_pitch (W values)
    long long out_pitch;
    long long out_batch;
    int W;
    int n_cols;
    int n_batch;
    int intra_kind;            // 0 NOOP, 2 CONJ_MUL, 3 CONJ_MUL_THEN_SCALE
    float intra_scale;
    const float2* tw;
    const float2* tw3;         // N = 3P: radix-3 pass twiddles (set by the launcher)
    int* err;
    int L_g[kMaxBatch];        // per-template valid rows of uneven batches (0: use L)
    int tpb;                   // templates per block: block (c, y) serves templates
                               // [y tpb, min((y + 1) tpb, n_batch)) of column c (grid.y blocks)
    int tc;                    // 1: the tensor-core form of the pass where it has one (length 1536,
                               // kernels_tc.cuh); otherwise the FP32 pass runs
};

// Shared-memory plan of the kernel (bytes), shared by the host launcher.
template <int N, class ImgC, int FPB>
struct XcorrSmem {
    static constexpr int kImgBytes = N * (int)sizeof(ImgC);
    static constexpr int kXchBytes = FftGroup<N, FPB, true>::BYTES;
    static __host__ __device__ constexpr int t1_col_elems(int L) { return (L + 1) & ~1; }  // 16-byte multiple
    static __host__ __device__ constexpr int img_off() { return 0; }
    static __host__ __device__ constexpr int xch_off() { return (kImgBytes + 127) & ~127; }
    static __host__ __device__ constexpr int t1_off() { return xch_off() + kXchBytes; }
    static __host__ __device__ constexpr int bar_off(int L, int nb) {
        return (t1_off() + nb * t1_col_elems(L) * 8 + 15) & ~15;
    }
    static __host__ __device__ constexpr int total(int L, int nb) { return bar_off(L, nb) + 16; }
};

// Block size of xcorr_cols_kernel: 128 threads (one FFT from N = 2048 up), with registers budgeted
// for 512 resident threads per SM.
constexpr int kXcorrBlockThreads = 128;
#ifndef FFB_XCORR_SM_THREADS
#define FFB_XCORR_SM_THREADS 512
#endif
constexpr int kXcorrSmThreads = FFB_XCORR_SM_THREADS;

// The intra-op is the conj-multiply (CONJ_MUL, or CONJ_MUL_THEN_SCALE: intra_kind 3): calls
// without it run at the plan's size.
template <int N, class ImgC, int FPB>
__global__ void __launch_bounds__(FftShape<N>::T * FPB,
                                  FftShape<N>::T * FPB < kXcorrSmThreads ? kXcorrSmThreads / (FftShape<N>::T * FPB) : 1)
xcorr_cols_kernel(XcorrColArgs a) {
    grid_dependency();
    using S = FftShape<N>;
    using SM = XcorrSmem<N, ImgC, FPB>;
    constexpr int T = S::T;
    extern __shared__ __align__(128) unsigned char sm_raw[];
    const ImgC* img_s = reinterpret_cast<const ImgC*>(sm_raw + SM::img_off());
    float2* xch = reinterpret_cast<float2*>(sm_raw + SM::xch_off());
    float2* t1_s = reinterpret_cast<float2*>(sm_raw + SM::t1_off());
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm_raw + SM::bar_off(a.L, a.tpb));
    const int g0 = blockIdx.y * a.tpb;                              // first template of the block
    const int nb = min(a.tpb, a.n_batch - g0);                      // templates of the block

    const int col = blockIdx.x;
    const int f = threadIdx.x / T;
    const int j = threadIdx.x - f * T;
    const int lcol = SM::t1_col_elems(a.L);

    __shared__ int ok_flag;
    uint32_t bytes = (uint32_t)SM::kImgBytes;
    for (int g = g0; g < g0 + nb; g++) bytes += (uint32_t)SM::t1_col_elems(a.L_g[g] > 0 ? a.L_g[g] : a.L) * 8;
    const bool staged = stage_block(bar, &ok_flag, bytes, a.err, [&]() {
        bulk_g2s(sm_raw + SM::img_off(), static_cast<const ImgC*>(a.img) + (long long)col * a.img_stride,
                 SM::kImgBytes, bar);
        for (int g = 0; g < nb; g++)
            bulk_g2s(t1_s + g * lcol, a.t1 + (g0 + g) * a.t1_batch + (long long)col * a.t1_pitch,
                     SM::t1_col_elems(a.L_g[g0 + g] > 0 ? a.L_g[g0 + g] : a.L) * 8, bar);
    });
    if (!staged) return;

    const float sc = a.intra_kind == 3 ? a.intra_scale : 1.f;
    const int rounds = (nb + FPB - 1) / FPB;
    FftGroup<N, FPB, true> grp(xch, f);
#pragma unroll 1
    for (int it = 0; it < rounds; it++) {
        const int gl = it * FPB + f;                 // template within the block
        const bool live = gl < nb;
        const int g = g0 + (live ? gl : 0);          // template within the launch
        const int Lg = (live && a.L_g[g] > 0) ? a.L_g[g] : a.L;
        // keep the next template's loads from being scheduled into this template's
        // transforms (that would hold twice the values live and spill)
        asm volatile("" ::: "memory");
        float2 v[16];
        const float2* src = t1_s + (live ? gl : 0) * lcol;
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const int n = j + T * q;
            v[q] = (live && n < Lg) ? src[n] : make_float2(0.f, 0.f);
        }
        BlockFft<N, false>::run(v, grp, j, a.tw, live ? leading_slots<T>(Lg, j) : 0);
        // CONJ_MUL (scale 1) skips the 32 multiplies of the scaling
        if (sc == 1.f) {
#pragma unroll
            for (int q = 0; q < 16; q++) v[q] = conj_mul(v[q], lds_cplx<ImgC>(img_s + j + T * q));
        } else {
#pragma unroll
            for (int q = 0; q < 16; q++) v[q] = cscale(conj_mul(v[q], lds_cplx<ImgC>(img_s + j + T * q)), sc);
        }
        // output pruning: only X[j + T q] < W are kept
        BlockFft<N, true>::run(v, grp, j, a.tw, 16, leading_slots<T>(a.W, j));
        if (live) {
            float2* o = a.out + (long long)g * a.out_batch + (long long)col * a.out_pitch;
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const int n = j + T * q;
                if (n < a.W) o[n] = v[q];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// The same pass on the split block FFT (fft_split.cuh), two templates per transform group
// ---------------------------------------------------------------------------
// 16- and 8-byte asynchronous copies global -> shared (the thread waits for its own)
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// element (both templates of a pair) from its two values, and back
template <class C> __device__ __forceinline__ C c_join(float2 a, float2 b);
template <> __device__ __forceinline__ float2 c_join<float2>(float2 a, float2) { return a; }
template <> __device__ __forceinline__ cpair c_join<cpair>(float2 a, float2 b) {
    return cmake<cpair>(make_float2(a.x, b.x), make_float2(a.y, b.y));
}
__device__ __forceinline__ float2 c_part(float2 v, int) { return v; }
__device__ __forceinline__ float2 c_part(cpair v, int w) {
    return w == 0 ? make_float2(v.x.x, v.y.x) : make_float2(v.x.y, v.y.y);
}

// Shared memory of a block: the image column, stored as P rows of E values (frequency s + E kp
// at row kp) of a stride that keeps the reads at freq_index free of bank conflicts, the exchange
// buffers of the G groups, and the input columns that each group works on next, thread by thread.
template <int N, class C, int G>
struct XcorrSplitSmem {
    using F = SplitFft<N, C>;
    static constexpr int W = (int)sizeof(C) / 8;   // templates per group
    static constexpr int IMG_STEP = F::B >= 8 ? 2 : 16 / F::B;
    static constexpr int IS = (F::E / IMG_STEP) % 2 ? F::E : F::B == 1 ? F::E : F::E + IMG_STEP;
    static constexpr int kImgBytes = F::P * IS * 8;
    static constexpr int kBufBytes = F::BUF * (int)sizeof(C);
    static __host__ __device__ constexpr int buf_off() { return (kImgBytes + 127) & ~127; }
    static __host__ __device__ constexpr int in_off() { return buf_off() + G * kBufBytes; }
    static __host__ __device__ constexpr int total(int L) { return in_off() + G * W * L * 8; }
};

template <int N, class C, int G, int MIN_BLOCKS>
__global__ void __launch_bounds__(SplitFft<N, C>::T * G, MIN_BLOCKS)
xcorr_split_kernel(XcorrColArgs a) {
    grid_dependency();
    using F = SplitFft<N, C>;
    using SM = XcorrSplitSmem<N, C, G>;
    constexpr int T = F::T, E = F::E, W = SM::W;
    extern __shared__ __align__(128) unsigned char sm_raw[];
    const int f = threadIdx.x / T, j = threadIdx.x % T;
    const int col = blockIdx.x;
    const int g0 = blockIdx.y * a.tpb;
    const int nb = min(a.tpb, a.n_batch - g0);
    float2* const img_s = reinterpret_cast<float2*>(sm_raw);
    C* const buf = reinterpret_cast<C*>(sm_raw + SM::buf_off()) + f * F::BUF;
    float2* const in_s = reinterpret_cast<float2*>(sm_raw + SM::in_off()) + f * W * a.L;

    auto sync = [&]() {
        if constexpr (T <= 32) {
            __syncwarp();
        } else if constexpr (G > 1) {
            asm volatile("bar.sync %0, %1;" ::"r"(f + 1), "n"(T) : "memory");
        } else {
            __syncthreads();
        }
    };
    // templates of this group in round `it`: first g, valid rows of each (0: none)
    auto rows = [&](int it, int w) {
        const int gl = (it * G + f) * W + w;
        if (gl >= nb) return 0;
        const int Lg = a.L_g[g0 + gl];
        return Lg > 0 ? Lg : a.L;
    };
    // each thread copies the elements it will read itself
    auto fetch = [&](int it) {
#pragma unroll
        for (int w = 0; w < W; w++) {
            const int Lw = rows(it, w);
            const float2* src =
                a.t1 + (long long)(g0 + (it * G + f) * W + w) * a.t1_batch + (long long)col * a.t1_pitch;
            for (int n = j; n < Lw; n += T) cp_async8(in_s + w * a.L + n, src + n);
        }
        cp_async_commit();
    };
    // the first templates before the image column, which only the product after the first forward
    // transform waits for
    fetch(0);
    {
        const float2* src = static_cast<const float2*>(a.img) + (long long)col * a.img_stride;
        for (int c = threadIdx.x; c < N / 2; c += T * G) {
            const int kp = c / (E / 2), s = 2 * (c % (E / 2));
            cp_async16(img_s + kp * SM::IS + s, src + 2 * c);
        }
    }
    cp_async_commit();

    const float sc = a.intra_kind == 3 ? a.intra_scale : 1.f;
    const float2* const img_t = img_s + (j % F::B) * SM::IS + j / F::B;
    const int rounds = (nb + G * W - 1) / (G * W);
#pragma unroll 1
    for (int it = 0; it < rounds; it++) {
        const int L0 = rows(it, 0), L1 = W > 1 ? rows(it, 1) : 0;
        const int qn = (max(L0, L1) + T - 1) / T;
        C v[E];
        if (it == 0)
            cp_async_wait<1>();
        else
            cp_async_wait<0>();
#pragma unroll
        for (int q = 0; q < E; q++) {
            const int n = j + T * q;
            float2 x0 = make_float2(0.f, 0.f), x1 = x0;
            if (q < qn) {
                if (n < L0) x0 = in_s[n];
                if (W > 1 && n < L1) x1 = in_s[a.L + n];
            }
            v[q] = c_join<C>(x0, x1);
        }
        F::forward(v, buf, j, a.tw, qn, sync);
        if (it == 0) {
            cp_async_wait<0>();
            __syncthreads();   // every thread's part of the image column is there
        }
        if (it + 1 < rounds) fetch(it + 1);
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int m = e / F::A, u = (e % F::A) / F::B, k2 = e % F::B;
            v[e] = pconj_mul(v[e], lds_cplx<float2>(img_t + (F::B * u + F::A * k2) * SM::IS + F::SPT * m));
        }
        if (sc != 1.f) {   // CONJ_MUL_THEN_SCALE
#pragma unroll
            for (int e = 0; e < E; e++) v[e] = pscale(v[e], sc);
        }
        F::inverse(v, buf, j, a.tw, sync);
#pragma unroll
        for (int w = 0; w < W; w++) {
            const int gl = (it * G + f) * W + w;
            if (gl < nb) {
                float2* o = a.out + (long long)(g0 + gl) * a.out_batch + (long long)col * a.out_pitch + j;
#pragma unroll
                for (int q = 0; q < E; q++)
                    if (j + T * q < a.W) o[T * q] = c_part(v[q], w);
            }
        }
    }
}

}  // namespace ffb
