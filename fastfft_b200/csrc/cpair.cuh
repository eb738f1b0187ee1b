// Arithmetic shared by single complex values (float2) and pairs of them (cpair): the split
// block FFT (fft_split.cuh) is written once and runs one transform or two at a time.
//
// A cpair holds the same element of two independent transforms, component-wise: x = the two
// real parts, y = the two imaginary parts.  No operation needs an exchange between the halves: a
// rotation by i is a renaming of registers, as for a single value.  (Packing the two components of
// one value instead needs register moves for every rotation and twiddle, and measured slower.)  Sums
// and differences are written as one sm_100 paired FP32 instruction (add.f32x2); products, whose
// second factor is one value for both halves, as two scalar ones: a paired product would first copy
// that factor into both halves of a register pair (288 against 282 us for a 64-template pass).  A paired
// instruction takes two cycles of the FP32 pipe but one issue slot, so the pair leaves the other
// slots to the shared-memory exchanges and addresses, and one twiddle, image value and address
// serves two transforms.  Measured on B200: a radix-16 pass with its twiddles takes 303
// cycles per warp and sub-partition as scalar code, 263 per transform as a pair.
//
// Products are rounded on their own (no contraction across these functions), so the two forms
// give bit-identical results.
#pragma once

#include <cuda_runtime.h>

namespace ffb {

struct __align__(16) cpair {
    float2 x, y;
};

__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float rsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float rmul(float a, float w) { return __fmul_rn(a, w); }
__device__ __forceinline__ float rfma(float a, float w, float c) { return __fmaf_rn(a, w, c); }
__device__ __forceinline__ float2 radd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 rsub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 rmul(float2 a, float w) { return make_float2(__fmul_rn(a.x, w), __fmul_rn(a.y, w)); }
__device__ __forceinline__ float2 rfma(float2 a, float w, float2 c) {
    return make_float2(__fmaf_rn(a.x, w, c.x), __fmaf_rn(a.y, w, c.y));
}

template <class C, class S>
__device__ __forceinline__ C cmake(S x, S y) {
    C c;
    c.x = x;
    c.y = y;
    return c;
}

template <class C>
__device__ __forceinline__ C padd(C a, C b) {
    return cmake<C>(radd(a.x, b.x), radd(a.y, b.y));
}
template <class C>
__device__ __forceinline__ C psub(C a, C b) {
    return cmake<C>(rsub(a.x, b.x), rsub(a.y, b.y));
}
// a + i b, a - i b
template <class C>
__device__ __forceinline__ C padd_i(C a, C b) {
    return cmake<C>(rsub(a.x, b.y), radd(a.y, b.x));
}
template <class C>
__device__ __forceinline__ C psub_i(C a, C b) {
    return cmake<C>(radd(a.x, b.y), rsub(a.y, b.x));
}
template <class C>
__device__ __forceinline__ C pscale(C a, float s) {
    return cmake<C>(rmul(a.x, s), rmul(a.y, s));
}
// a w (INV: a conj(w)): the twiddle w is one value for both transforms of a pair
template <bool INV, class C>
__device__ __forceinline__ C pmul(C a, float2 w) {
    const float wy = INV ? -w.y : w.y;
    return cmake<C>(rfma(a.x, w.x, rmul(a.y, -wy)), rfma(a.x, wy, rmul(a.y, w.x)));
}
// conj(a) b: the CONJ_MUL intra-op
template <class C>
__device__ __forceinline__ C pconj_mul(C a, float2 b) {
    return cmake<C>(rfma(a.x, b.x, rmul(a.y, b.y)), rfma(a.x, b.y, rmul(a.y, -b.x)));
}
// the twiddle product itself (one value)
__device__ __forceinline__ float2 wmul(float2 a, float2 b) {
    return make_float2(rfma(a.x, b.x, rmul(a.y, -b.y)), rfma(a.x, b.y, rmul(a.y, b.x)));
}

// ---------------------------------------------------------------------------
// Small DFTs, natural order in and out, in place on v[O .. O + n)
// ---------------------------------------------------------------------------
constexpr float kPC1 = 0.923879532511286756128f;  // cos(pi/8)
constexpr float kPS1 = 0.382683432365089771728f;  // sin(pi/8)
constexpr float kPR2 = 0.707106781186547524401f;  // sqrt(2)/2
constexpr float kPH3 = 0.866025403784438646764f;  // sqrt(3)/2

// a W8 and a W8^3 (INV: conjugates), W8 = exp(-2 pi i / 8)
template <bool INV, class C>
__device__ __forceinline__ C mul_w8_1(C a) {
    return INV ? cmake<C>(rmul(rsub(a.x, a.y), kPR2), rmul(radd(a.x, a.y), kPR2))
               : cmake<C>(rmul(radd(a.x, a.y), kPR2), rmul(rsub(a.y, a.x), kPR2));
}
template <bool INV, class C>
__device__ __forceinline__ C mul_w8_3(C a) {
    return INV ? cmake<C>(rmul(radd(a.x, a.y), -kPR2), rmul(rsub(a.x, a.y), kPR2))
               : cmake<C>(rmul(rsub(a.y, a.x), kPR2), rmul(radd(a.x, a.y), -kPR2));
}
// a + (-i) b and a - (-i) b (INV: +i): the quarter turn of a DFT4's odd outputs
template <bool INV, class C>
__device__ __forceinline__ C add_turn(C a, C b) {
    return INV ? padd_i(a, b) : psub_i(a, b);
}
template <bool INV, class C>
__device__ __forceinline__ C sub_turn(C a, C b) {
    return INV ? psub_i(a, b) : padd_i(a, b);
}

template <class C>
__device__ __forceinline__ void pdft2(C& a0, C& a1) {
    const C t = psub(a0, a1);
    a0 = padd(a0, a1);
    a1 = t;
}
// TURN2: the third input enters times -i (INV: +i), a twiddle folded into the first sums
template <bool INV, bool TURN2 = false, class C>
__device__ __forceinline__ void pdft4(C& a0, C& a1, C& a2, C& a3) {
    const C s0 = TURN2 ? add_turn<INV>(a0, a2) : padd(a0, a2);
    const C e = TURN2 ? sub_turn<INV>(a0, a2) : psub(a0, a2);
    const C s1 = padd(a1, a3), d = psub(a1, a3);
    a0 = padd(s0, s1);
    a2 = psub(s0, s1);
    a1 = add_turn<INV>(e, d);
    a3 = sub_turn<INV>(e, d);
}
// outputs of DFT8 from the DFT4s of its even (e) and odd (o) inputs
template <bool INV, class C>
__device__ __forceinline__ void pdft8_join(C& e0, C& o0, C& e1, C& o1, C& e2, C& o2, C& e3, C& o3) {
    const C t1 = mul_w8_1<INV>(o1), t3 = mul_w8_3<INV>(o3);
    const C x0 = padd(e0, o0), x4 = psub(e0, o0), x1 = padd(e1, t1), x5 = psub(e1, t1);
    const C x2 = add_turn<INV>(e2, o2), x6 = sub_turn<INV>(e2, o2), x3 = padd(e3, t3), x7 = psub(e3, t3);
    e0 = x0; o0 = x1; e1 = x2; o1 = x3; e2 = x4; o2 = x5; e3 = x6; o3 = x7;
}
template <bool INV, class C>
__device__ __forceinline__ void pdft8(C& a0, C& a1, C& a2, C& a3, C& a4, C& a5, C& a6, C& a7) {
    pdft4<INV>(a0, a2, a4, a6);
    pdft4<INV>(a1, a3, a5, a7);
    pdft8_join<INV>(a0, a1, a2, a3, a4, a5, a6, a7);
}
// forward DFT8 with a2 = a5 = 0 (their values are not read; all eight outputs are formed)
template <class C>
__device__ __forceinline__ void pdft8_fwd_no25(C& a0, C& a1, C& a2, C& a3, C& a4, C& a5, C& a6, C& a7) {
    const C s = padd(a0, a4), e = psub(a0, a4);
    a0 = padd(s, a6);
    a4 = psub(s, a6);
    a2 = padd_i(e, a6);
    a6 = psub_i(e, a6);
    const C t = padd(a3, a7), d = psub(a3, a7), o = a1;
    a1 = padd(o, t);
    a5 = psub(o, t);
    a3 = psub_i(o, d);
    a7 = padd_i(o, d);
    pdft8_join<false>(a0, a1, a2, a3, a4, a5, a6, a7);
}

// second half of DFT16 after its first DFT4s, a[n1 + 4 k1]: constant twiddles and DFT4s over n1
template <bool INV, int O, int E, class C>
__device__ __forceinline__ void pdft16_join(C (&v)[E]) {
    const float2 c1 = make_float2(kPC1, -kPS1), c3 = make_float2(kPS1, -kPC1), c9 = make_float2(-kPC1, kPS1);
    v[O + 5] = pmul<INV>(v[O + 5], c1);
    v[O + 9] = mul_w8_1<INV>(v[O + 9]);
    v[O + 13] = pmul<INV>(v[O + 13], c3);
    v[O + 6] = mul_w8_1<INV>(v[O + 6]);
    v[O + 14] = mul_w8_3<INV>(v[O + 14]);
    v[O + 7] = pmul<INV>(v[O + 7], c3);
    v[O + 11] = mul_w8_3<INV>(v[O + 11]);
    v[O + 15] = pmul<INV>(v[O + 15], c9);
    pdft4<INV>(v[O], v[O + 1], v[O + 2], v[O + 3]);
    pdft4<INV>(v[O + 4], v[O + 5], v[O + 6], v[O + 7]);
    pdft4<INV, true>(v[O + 8], v[O + 9], v[O + 10], v[O + 11]);
    pdft4<INV>(v[O + 12], v[O + 13], v[O + 14], v[O + 15]);
    C t[16];
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++)
#pragma unroll
        for (int k2 = 0; k2 < 4; k2++) t[k1 + 4 * k2] = v[O + 4 * k1 + k2];
#pragma unroll
    for (int k = 0; k < 16; k++) v[O + k] = t[k];
}

// DFT24 as 3 x 8 without twiddles (Good's prime-factor order: input n = 8 n3 + 3 n8 mod 24,
// output k with k mod 3 = k3, k mod 8 = k8)
template <bool INV, class C>
__device__ __forceinline__ void pdft3(C& a0, C& a1, C& a2) {
    const C s = padd(a1, a2), d = psub(a1, a2);
    const C m = cmake<C>(rfma(s.x, -0.5f, a0.x), rfma(s.y, -0.5f, a0.y));
    const float h = INV ? kPH3 : -kPH3;   // a1: m + i h d
    a0 = padd(a0, s);
    a1 = cmake<C>(rfma(d.y, -h, m.x), rfma(d.x, h, m.y));
    a2 = cmake<C>(rfma(d.y, h, m.x), rfma(d.x, -h, m.y));
}
constexpr int pfa_in(int n3, int n8) { return (8 * n3 + 3 * n8) % 24; }
constexpr int pfa_out(int k3, int k8) { return (16 * k3 + 9 * k8) % 24; }  // 16 = (1, 0), 9 = (0, 1) mod (3, 8)

template <bool INV, class C>
__device__ __forceinline__ void pdft24_eights(C (&v)[24]) {
#pragma unroll
    for (int a = 0; a < 3; a++)
        pdft8<INV>(v[pfa_in(a, 0)], v[pfa_in(a, 1)], v[pfa_in(a, 2)], v[pfa_in(a, 3)], v[pfa_in(a, 4)],
                   v[pfa_in(a, 5)], v[pfa_in(a, 6)], v[pfa_in(a, 7)]);
}
template <bool INV, class C>
__device__ __forceinline__ void pdft24_threes(C (&v)[24]) {
#pragma unroll
    for (int b = 0; b < 8; b++) pdft3<INV>(v[pfa_in(0, b)], v[pfa_in(1, b)], v[pfa_in(2, b)]);
}
// The forward DFT24 takes the DFT3s first, as its short head below does, so that both give the
// same bits where the short one applies: which of the two a pair takes depends on both its templates.
template <bool INV, class C>
__device__ __forceinline__ void pdft24(C (&v)[24]) {
    if constexpr (INV) {
        pdft24_eights<INV>(v);
        pdft24_threes<INV>(v);
    } else {
        pdft24_threes<INV>(v);
        pdft24_eights<INV>(v);
    }
    C t[24];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 8; b++) t[pfa_out(a, b)] = v[pfa_in(a, b)];
#pragma unroll
    for (int k = 0; k < 24; k++) v[k] = t[k];
}
// a W3 and a W3^2 (forward), a being the only non-zero input n3 = 1 (R = 1) or 2 (R = 2) of a DFT3
template <int R, class C>
__device__ __forceinline__ void pdft3_one(C a, C& y1, C& y2) {
    const C m = cmake<C>(rmul(a.x, -0.5f), rmul(a.y, -0.5f));
    const float h = R == 1 ? -kPH3 : kPH3;
    y1 = cmake<C>(rfma(a.y, -h, m.x), rfma(a.x, h, m.y));
    y2 = cmake<C>(rfma(a.y, h, m.x), rfma(a.x, -h, m.y));
}
// forward DFT24 whose inputs v[6 .. 24) are zero (and not read): inputs 0 .. 5 are (n3, n8) =
// (0,0) (2,3) (1,6) (0,1) (2,4) (1,7), one per DFT3, and the DFT8s lack n8 = 2 and 5
template <class C>
__device__ __forceinline__ void pdft24_fwd_head6(C (&v)[24]) {
    C y[3][8];
    y[0][0] = y[1][0] = y[2][0] = v[0];
    y[0][1] = y[1][1] = y[2][1] = v[3];
    y[0][3] = v[1];
    pdft3_one<2>(v[1], y[1][3], y[2][3]);
    y[0][6] = v[2];
    pdft3_one<1>(v[2], y[1][6], y[2][6]);
    y[0][4] = v[4];
    pdft3_one<2>(v[4], y[1][4], y[2][4]);
    y[0][7] = v[5];
    pdft3_one<1>(v[5], y[1][7], y[2][7]);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        pdft8_fwd_no25(y[a][0], y[a][1], y[a][2], y[a][3], y[a][4], y[a][5], y[a][6], y[a][7]);
#pragma unroll
        for (int b = 0; b < 8; b++) v[pfa_out(a, b)] = y[a][b];
    }
}

// DFT of length R in place on v[O .. O + R)
template <bool INV, int R, int O, int E, class C>
__device__ __forceinline__ void pdft(C (&v)[E]) {
    if constexpr (R == 2) {
        pdft2(v[O], v[O + 1]);
    } else if constexpr (R == 4) {
        pdft4<INV>(v[O], v[O + 1], v[O + 2], v[O + 3]);
    } else if constexpr (R == 8) {
        pdft8<INV>(v[O], v[O + 1], v[O + 2], v[O + 3], v[O + 4], v[O + 5], v[O + 6], v[O + 7]);
    } else if constexpr (R == 16) {
        pdft4<INV>(v[O], v[O + 4], v[O + 8], v[O + 12]);
        pdft4<INV>(v[O + 1], v[O + 5], v[O + 9], v[O + 13]);
        pdft4<INV>(v[O + 2], v[O + 6], v[O + 10], v[O + 14]);
        pdft4<INV>(v[O + 3], v[O + 7], v[O + 11], v[O + 15]);
        pdft16_join<INV, O>(v);
    } else {
        static_assert(R == 24 && O == 0 && E == 24, "radix 2, 4, 8, 16 or 24");
        pdft24<INV>(v);
    }
}

// forward DFT of length E whose inputs v[qn .. E) are zero: the first stages of the shorter
// heads are specialised (size increase: the padding is neither loaded nor transformed)
template <int E, class C>
__device__ __forceinline__ void pdft_fwd_head(C (&v)[E], int qn) {
    if constexpr (E == 24) {
        if (qn <= 6)
            pdft24_fwd_head6(v);
        else
            pdft24<false>(v);
    } else {
        static_assert(E == 16, "16 or 24 values per thread");
        if (qn <= 4) {
#pragma unroll
            for (int n = 0; n < 4; n++) v[n + 4] = v[n + 8] = v[n + 12] = v[n];
        } else if (qn <= 8) {
#pragma unroll
            for (int n = 0; n < 4; n++) {
                const C a = v[n], b = v[n + 4];
                v[n] = padd(a, b);
                v[n + 4] = psub_i(a, b);
                v[n + 8] = psub(a, b);
                v[n + 12] = padd_i(a, b);
            }
        } else {
            pdft4<false>(v[0], v[4], v[8], v[12]);
            pdft4<false>(v[1], v[5], v[9], v[13]);
            pdft4<false>(v[2], v[6], v[10], v[14]);
            pdft4<false>(v[3], v[7], v[11], v[15]);
        }
        pdft16_join<false, 0>(v);
    }
}

}  // namespace ffb
