// Split block FFT: N = E P with E values per thread (E = 16 or 24), the outer DFT_E in registers
// and P-point sub-FFTs of a few neighbouring threads.
//
// T = P threads run one transform.  With n = b + P q and k = s + E kp (q, s < E; b, kp < P):
//   forward (decimation in frequency)
//     y_s[b] = W_N^(b s) sum_q W_E^(q s) x[b + P q]           thread b, in registers
//     X[s + E kp] = sum_b W_P^(b kp) y_s[b]                   sub-FFT s
//   inverse (decimation in time): the same steps conjugated, in reverse order.
// A sub-FFT is P = A B: B neighbouring threads (of one warp) hold A values each, a DFT_A, the
// twiddle W_P^(i k1), an exchange among those B threads, and DFT_Bs; thread (jh, i) = (j / B,
// j mod B) serves the sub-FFTs s = jh + (T / B) m, m < E / A.  Time-domain values are in natural
// order (slot q = x[j + T q]); the spectrum stays where the sub-FFT leaves it (freq_index), which
// is where a pointwise product is applied and where the inverse starts.
//
// What this split is for: a forward and inverse transform together take two block-wide
// exchanges (four barriers of T threads) and two exchanges within a few threads of a warp,
// whose synchronisation is __syncwarp().  Length 1536 as 24 x 64 moves 8 x N values through
// shared memory per forward-inverse pair and reads its input once; as three 512-point FFTs of
// 16-value threads and a radix-3 step it moved 10 x N and read the input three times, and the
// shared-memory path (75 % busy, 333 us per 64-template launch against 265) was what bound the
// pass.
//
// C = float2 runs one transform, C = cpair two at a time (cpair.cuh).
#pragma once

#include "cpair.cuh"
#include "fft_core.cuh"

namespace ffb {

template <int N>
struct SplitShape;
#define FFB_SPLIT_SHAPE(N_, E_, A_, B_) \
    template <>                         \
    struct SplitShape<N_> {             \
        static constexpr int E = E_, A = A_, B = B_; \
    };
FFB_SPLIT_SHAPE(256, 16, 16, 1)
FFB_SPLIT_SHAPE(384, 24, 8, 2)
FFB_SPLIT_SHAPE(512, 16, 8, 4)
FFB_SPLIT_SHAPE(768, 24, 8, 4)
FFB_SPLIT_SHAPE(1024, 16, 8, 8)
FFB_SPLIT_SHAPE(1536, 24, 8, 8)
FFB_SPLIT_SHAPE(2048, 16, 16, 8)
#undef FFB_SPLIT_SHAPE

// Lengths with a split form, in table order.
constexpr int kSplitCount = 7;
__host__ __device__ constexpr int split_size(int i) { return (i % 2 ? 384 : 256) << (i / 2); }  // 256, 384, 512, ... 2048
__host__ __device__ constexpr bool is_split_size(int n) {
    return n == 256 || n == 384 || n == 512 || n == 768 || n == 1024 || n == 1536 || n == 2048;
}
// Twiddle table of length N: W_N^(s b) at s P + b (s < E, b < P), then W_P^(i k1) at k1 B + i
// (k1 < A, i < B): N + P entries.
__host__ __device__ constexpr int split_e(int n) { return n % 3 == 0 ? 24 : 16; }
__host__ __device__ constexpr int split_b(int n) {
    return n == 256 ? 1 : n == 384 ? 2 : n <= 768 ? 4 : 8;
}
__host__ __device__ constexpr int tws_size_of(int n) { return n + n / split_e(n); }
__host__ __device__ constexpr int tws_base(int n) {
    int off = 0;
    for (int i = 0; i < kSplitCount && split_size(i) < n; i++) off += tws_size_of(split_size(i));
    return off;
}
constexpr int kTwsTotal = tws_base(2048) + tws_size_of(2048);

// Shared-memory layout of one transform's exchange buffer: one region of RS elements per
// sub-FFT; nat(b, p) holds element b of the sub-FFT's time side, ex(k1, i, p) the exchange
// inside it; p = parity of jh.  The element at which a wavefront's lanes (8 of 16 bytes, 16 of 8
// bytes) meet must differ modulo that many elements: by an exclusive or where the lanes of a
// wavefront are whole sub-FFTs or parts of one, else by padding.
template <int A, int B, int BYTES>
struct SplitLayout {
    static constexpr int P = A * B;
    static constexpr int LANES = 128 / BYTES;                    // elements per wavefront
    static constexpr bool SWIZZLE = B >= 8;                      // i ^ row
    static constexpr int PS = SWIZZLE || B == 1 ? B : B + 1;     // stride of k1 in the exchange
    static constexpr int NEED = A * PS > P ? A * PS : P;
    // padded regions of consecutive sub-FFTs start B elements apart modulo a wavefront
    static constexpr int RS = SWIZZLE ? P : NEED + ((B - NEED) % LANES + LANES) % LANES;
    static constexpr int MASK = (B < LANES ? B : LANES) - 1;
    // the parity of the sub-FFT moves it to the other half of a wavefront
    static constexpr int PAR = SWIZZLE && B < LANES ? B : 0;
    static __device__ __forceinline__ int nat(int b, int p) { return PAR ? b ^ (p ? PAR : 0) : b; }
    static __device__ __forceinline__ int ex(int k1, int i, int p) {
        if constexpr (SWIZZLE) return (k1 * B + (i ^ (k1 & MASK))) ^ (PAR && p ? PAR : 0);
        else return k1 * PS + i;
    }
};

template <int N, class C>
struct SplitFft {
    using S = SplitShape<N>;
    static constexpr int E = S::E, A = S::A, B = S::B;
    static constexpr int P = A * B;
    static constexpr int T = P;                   // threads per transform
    static constexpr int M = E / A;               // sub-FFTs per thread
    static constexpr int U = A / B;               // DFT_Bs per sub-FFT and thread
    static constexpr int SPT = T / B;             // stride of a thread's sub-FFTs
    static_assert(N == E * P && E % A == 0 && A % B == 0 && SPT * M == E && 32 % B == 0, "shape");
    using L = SplitLayout<A, B, (int)sizeof(C)>;
    static constexpr int BUF = E * L::RS;         // elements of the exchange buffer
    static constexpr int parity(int s) { return (s % SPT) & 1; }

    // natural index of slot e = m A + u B + k2 of thread j after forward()
    static __device__ __forceinline__ int freq_index(int j, int e) {
        const int m = e / A, u = (e % A) / B, k2 = e % B;
        return (j / B + SPT * m) + E * ((j % B) + B * u + A * k2);
    }

    // Outer twiddles v[s] *= W_N^(s b), s < E, from the table values W^1, W^2, W^4, W^8 and (E = 24)
    // W^16; t = table + b.  In the order r, r + 8, r + 16, so that few of the products are
    // held at a time (all of them at once cost registers, and spills at 128).
    template <bool INV>
    static __device__ __forceinline__ void twiddle(C (&v)[E], const float2* __restrict__ t) {
        const float2 w1 = ld_tw(t + P), w2 = ld_tw(t + 2 * P), w4 = ld_tw(t + 4 * P), w8 = ld_tw(t + 8 * P);
        const float2 w16 = E > 16 ? ld_tw(t + (E > 16 ? 16 : 0) * P) : w8;
        float2 w3 = w1;
        v[8] = pmul<INV>(v[8], w8);
        if constexpr (E > 16) v[16] = pmul<INV>(v[16], w16);
#pragma unroll
        for (int r = 1; r < 8; r++) {
            const float2 w = r == 1 ? w1 : r == 2 ? w2 : r == 4 ? w4
                           : r == 3 ? wmul(w1, w2) : r == 5 ? wmul(w1, w4) : r == 6 ? wmul(w2, w4) : wmul(w3, w4);
            if (r == 3) w3 = w;
            v[r] = pmul<INV>(v[r], w);
            v[r + 8] = pmul<INV>(v[r + 8], wmul(w, w8));
            if constexpr (E > 16) v[r + 16] = pmul<INV>(v[r + 16], wmul(w, w16));
        }
    }

    template <bool INV, int MM>
    static __device__ __forceinline__ void sub_first(C (&v)[E]) {
        if constexpr (MM < M) {
            pdft<INV, A, MM * A>(v);
            sub_first<INV, MM + 1>(v);
        }
    }
    template <bool INV, int I>
    static __device__ __forceinline__ void sub_last(C (&v)[E]) {
        if constexpr (B > 1 && I < M * U) {
            pdft<INV, B, I * B>(v);
            sub_last<INV, I + 1>(v);
        }
    }
    template <bool INV, int MM>
    static __device__ __forceinline__ void sub_twiddle(C (&v)[E], const float2 (&w)[A]) {
        if constexpr (MM < M) {
#pragma unroll
            for (int k1 = 1; k1 < A; k1++) v[MM * A + k1] = pmul<INV>(v[MM * A + k1], w[k1]);
            sub_twiddle<INV, MM + 1>(v, w);
        }
    }
    // W_P^(i k1), k1 < A, one set for all of the thread's sub-FFTs
    static __device__ __forceinline__ void sub_weights(float2 (&w)[A], const float2* __restrict__ t, int i) {
#pragma unroll
        for (int k = 1; k < A; k++) {
            const int top = k >= 8 ? 8 : k >= 4 ? 4 : k >= 2 ? 2 : 1;
            w[k] = k == top ? ld_tw(t + k * B + i) : wmul(w[k - top], w[top]);
        }
    }

    // v[q] = x[j + T q] in, spectrum out (freq_index).  Only the slots q < qn are read.  buf: this
    // transform's exchange buffer; sync(): barrier of its T threads.
    template <class Sync>
    static __device__ __forceinline__ void forward(C (&v)[E], C* buf, int j, const float2* __restrict__ tws, int qn,
                                                   Sync sync) {
        const int jh = j / B, i = j % B, p = jh & 1;
        pdft_fwd_head<E>(v, qn);
        twiddle<false>(v, tws + j);
        sync();   // earlier readers of the buffer are done
#pragma unroll
        for (int s = 0; s < E; s++) buf[s * L::RS + L::nat(j, parity(s))] = v[s];
        sync();
        C* const sub = buf + jh * L::RS;
#pragma unroll
        for (int m = 0; m < M; m++)
#pragma unroll
            for (int r = 0; r < A; r++) v[m * A + r] = sub[m * SPT * L::RS + L::nat(i + B * r, p)];
        sub_first<false, 0>(v);
        if constexpr (B > 1) {
            float2 w[A];
            sub_weights(w, tws + N, i);
            sub_twiddle<false, 0>(v, w);
            __syncwarp();   // the sub-FFT's threads have read its region
#pragma unroll
            for (int m = 0; m < M; m++)
#pragma unroll
                for (int k1 = 0; k1 < A; k1++) sub[m * SPT * L::RS + L::ex(k1, i, p)] = v[m * A + k1];
            __syncwarp();
#pragma unroll
            for (int m = 0; m < M; m++)
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int b = 0; b < B; b++)
                        v[m * A + u * B + b] = sub[m * SPT * L::RS + L::ex(i + B * u, b, p)];
            sub_last<false, 0>(v);
        }
    }

    // Spectrum in (freq_index), v[q] = x[j + T q] out (unnormalised).  Follows a forward() on the
    // same buffer and threads.
    template <class Sync>
    static __device__ __forceinline__ void inverse(C (&v)[E], C* buf, int j, const float2* __restrict__ tws, Sync sync) {
        const int jh = j / B, i = j % B, p = jh & 1;
        C* const sub = buf + jh * L::RS;
        if constexpr (B > 1) {
            sub_last<true, 0>(v);
            __syncwarp();   // the forward exchange has been read
#pragma unroll
            for (int m = 0; m < M; m++)
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int b = 0; b < B; b++)
                        sub[m * SPT * L::RS + L::ex(i + B * u, b, p)] = v[m * A + u * B + b];
            __syncwarp();
#pragma unroll
            for (int m = 0; m < M; m++)
#pragma unroll
                for (int k1 = 0; k1 < A; k1++) v[m * A + k1] = sub[m * SPT * L::RS + L::ex(k1, i, p)];
            float2 w[A];
            sub_weights(w, tws + N, i);
            sub_twiddle<true, 0>(v, w);
        }
        sub_first<true, 0>(v);
        if constexpr (B > 1) __syncwarp();
#pragma unroll
        for (int m = 0; m < M; m++)
#pragma unroll
            for (int r = 0; r < A; r++) sub[m * SPT * L::RS + L::nat(i + B * r, p)] = v[m * A + r];
        sync();
#pragma unroll
        for (int s = 0; s < E; s++) v[s] = buf[s * L::RS + L::nat(j, parity(s))];
        twiddle<true>(v, tws + j);
        pdft<true, E, 0>(v);
    }
};

}  // namespace ffb
