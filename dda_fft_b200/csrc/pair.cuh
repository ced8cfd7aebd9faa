// Two complex numbers per register quadruple and the packed FP32 instructions of sm_100
// (add / mul / fma .f32x2: the flops of two scalar instructions in one issue slot; measured
// 1.8-1.95 of them per SM and clock against 3.8 scalar ones, so the FP32 rate is the same and
// half the issue slots are left to loads, stores and addresses).
//
// The matvec's pairs are the two parity halves of the padded z axis: bins 2k and 2k + 1 of a
// 2n-point line go through the same transforms with the same twiddles, so every butterfly is
// one packed instruction per real and imaginary part, and a pair is one 16-byte access.
#pragma once
#include "common.cuh"

struct P2 {
    float2 r, i;   // (Re a, Re b), (Im a, Im b)
};

DDA_DEV float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
DDA_DEV float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
DDA_DEV float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
DDA_DEV float2 sub2(float2 a, float2 b)
{
    float2 d;
    asm("{ .reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; sub.rn.f32x2 z, x, y; mov.b64 {%0, %1}, z; }"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
DDA_DEV float2 dup2(float x) { return make_float2(x, x); }

DDA_DEV P2 padd(P2 a, P2 b) { return {add2(a.r, b.r), add2(a.i, b.i)}; }
DDA_DEV P2 psub(P2 a, P2 b) { return {sub2(a.r, b.r), sub2(a.i, b.i)}; }
DDA_DEV P2 pzero() { return {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }
// both numbers times w (cmul's operations and roundings)
DDA_DEV P2 pmul(P2 a, float2 w)
{
    return {fma2(a.r, dup2(w.x), mul2(a.i, dup2(-w.y))), fma2(a.r, dup2(w.y), mul2(a.i, dup2(w.x)))};
}
DDA_DEV P2 pmulc(P2 a, float2 w) { return pmul(a, make_float2(w.x, -w.y)); }   // times conj(w)
DDA_DEV P2 ppack(float2 a, float2 b) { return {make_float2(a.x, b.x), make_float2(a.y, b.y)}; }
DDA_DEV float2 pfirst(P2 p) { return make_float2(p.r.x, p.i.x); }
DDA_DEV float2 psecond(P2 p) { return make_float2(p.r.y, p.i.y); }

DDA_DEV P2 p_of(float4 q) { return {make_float2(q.x, q.y), make_float2(q.z, q.w)}; }
DDA_DEV float4 f4_of(P2 p) { return make_float4(p.r.x, p.r.y, p.i.x, p.i.y); }

// a pair as two columns of the work buffer
DDA_DEV float4 columns_of(P2 p) { return make_float4(p.r.x, p.i.x, p.r.y, p.i.y); }
DDA_DEV P2 of_columns(float4 q) { return {make_float2(q.x, q.z), make_float2(q.y, q.w)}; }

// a -+ i b: the times -i (forward) or +i (inverse) of a butterfly as a choice of add and sub
template <bool INV>
DDA_DEV P2 padd_rot(P2 a, P2 b)   // a + (INV ? i : -i) b
{
    return INV ? P2{sub2(a.r, b.i), add2(a.i, b.r)} : P2{add2(a.r, b.i), sub2(a.i, b.r)};
}
template <bool INV>
DDA_DEV P2 psub_rot(P2 a, P2 b)   // a - (INV ? i : -i) b
{
    return padd_rot<!INV>(a, b);
}
// a + w b and a - w b for w = exp(-+ i pi / 4) (ODD 0) or its cube (ODD 1): two adds and four
// fused multiply-adds
template <bool INV, int ODD>
DDA_DEV void pbfly8(P2 a, P2 b, P2 &x, P2 &y)
{
    const float2 h = dup2(0.70710678118654752440f), n = dup2(-0.70710678118654752440f);
    const float2 s = INV ? sub2(b.r, b.i) : add2(b.r, b.i), d = INV ? add2(b.i, b.r) : sub2(b.i, b.r);
    if (ODD == 0) {
        x = {fma2(h, s, a.r), fma2(h, d, a.i)};
        y = {fma2(n, s, a.r), fma2(n, d, a.i)};
    } else if (INV) {
        x = {fma2(n, d, a.r), fma2(h, s, a.i)};
        y = {fma2(h, d, a.r), fma2(n, s, a.i)};
    } else {
        x = {fma2(h, d, a.r), fma2(n, s, a.i)};
        y = {fma2(n, d, a.r), fma2(h, s, a.i)};
    }
}

// In-register DFT of R points (2..16) of pairs, natural order in and out.
template <bool INV>
DDA_DEV void dft4p(P2 &a0, P2 &a1, P2 &a2, P2 &a3)
{
    const P2 t0 = padd(a0, a2), t1 = psub(a0, a2), t2 = padd(a1, a3), t3 = psub(a1, a3);
    a0 = padd(t0, t2);
    a2 = psub(t0, t2);
    a1 = padd_rot<INV>(t1, t3);
    a3 = psub_rot<INV>(t1, t3);
}

template <bool INV>
DDA_DEV void dft8p(P2 &a0, P2 &a1, P2 &a2, P2 &a3, P2 &a4, P2 &a5, P2 &a6, P2 &a7)
{
    dft4p<INV>(a0, a2, a4, a6);   // even part: bins 0..3 in a0 a2 a4 a6
    dft4p<INV>(a1, a3, a5, a7);   // odd part in a1 a3 a5 a7
    const P2 e0 = a0, e1 = a2, e2 = a4, e3 = a6, o0 = a1, o1 = a3, o2 = a5, o3 = a7;
    a0 = padd(e0, o0);
    a4 = psub(e0, o0);
    pbfly8<INV, 0>(e1, o1, a1, a5);
    a2 = padd_rot<INV>(e2, o2);
    a6 = psub_rot<INV>(e2, o2);
    pbfly8<INV, 1>(e3, o3, a3, a7);
}

template <int R, bool INV>
DDA_DEV void dftp(P2 (&v)[R])
{
    static_assert(R == 1 || R == 2 || R == 4 || R == 8 || R == 16, "register DFT size");
    if constexpr (R == 2) {
        const P2 a = v[0], b = v[1];
        v[0] = padd(a, b);
        v[1] = psub(a, b);
    } else if constexpr (R == 4) {
        dft4p<INV>(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        dft8p<INV>(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
    } else if constexpr (R == 16) {
        dft8p<INV>(v[0], v[2], v[4], v[6], v[8], v[10], v[12], v[14]);
        dft8p<INV>(v[1], v[3], v[5], v[7], v[9], v[11], v[13], v[15]);
        P2 e[8], o[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            e[k] = v[2 * k];
            o[k] = v[2 * k + 1];
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (k == 0) {
                v[0] = padd(e[0], o[0]);
                v[8] = psub(e[0], o[0]);
            } else if (k == 4) {
                v[4] = padd_rot<INV>(e[4], o[4]);
                v[12] = psub_rot<INV>(e[4], o[4]);
            } else if (k == 2) {
                pbfly8<INV, 0>(e[2], o[2], v[2], v[10]);
            } else if (k == 6) {
                pbfly8<INV, 1>(e[6], o[6], v[6], v[14]);
            } else {
                float2 w = w16(k);
                if (INV) w.y = -w.y;
                const P2 t = pmul(o[k], w);
                v[k] = padd(e[k], t);
                v[k + 8] = psub(e[k], t);
            }
        }
    }
}

// n = R1 R2 of the matvec's lines: two steps at every edge (R1 = R2 or 2 R2)
template <int N>
struct line_split {
    static constexpr int R1 = fft_split<N>::R1, R2 = fft_split<N>::R2;
};
template <> struct line_split<4> { static constexpr int R1 = 2, R2 = 2; };
template <> struct line_split<8> { static constexpr int R1 = 4, R2 = 2; };
static_assert(line_split<16>::R2 == 4 && line_split<32>::R2 == 4 && line_split<64>::R2 == 8 && line_split<128>::R2 == 8,
              "the host's twiddle tables follow these splits (line_r2)");
