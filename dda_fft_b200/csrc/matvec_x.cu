// x pass of the matvec for lattice edges 4..128: forward along i, symmetric 3x3 product with the
// Green tensor, inverse along i, in place on the work buffer of matvec_yz.cu, whose rows are 2 nl
// complex columns (column 2 zpos + h holds the z bin 2 kl + h).
//
// Every n-point line uses n = R1 R2: a thread (sub, column), consecutive lanes on consecutive
// columns, holds R1 elements of a line for step A and R2 elements for step B, and the steps
// exchange data through shared memory.  An even / odd pair of transforms covers the padded
// line: bins 2 k + h are DFT_n(x W_2n^(h j)), and the inverse keeps the first n outputs.
//
// What bounds it: the L1 data path, where every 128-byte line that an access touches costs a cycle.
// Per right-hand side at 64^3 the pass brings 25 MB of columns and 100 MB of Green tensor in,
// 25 MB out and moves 200 MB through shared memory; counters at the packed pair form: 74% of the
// path's cycles busy, FP32 43%, DRAM a third.  Hence whole lines per access, 16-byte pairs and,
// for polarisation pairs, one load of the Green tensor for both.
// Compiled once per x edge (X_NI).
#include <cuda.h>   // CUtensorMap (the type only; maps are encoded in ddagpu.cu)

#include <type_traits>

#include "internal.h"
#include "pair.cuh"
#include "zorder.cuh"

namespace ddagpu {

namespace {

template <int N>
struct Sx {
    static constexpr int R1 = line_split<N>::R1, R2 = line_split<N>::R2, RM = R1;
    static_assert(R2 > 1 && (R1 == R2 || R1 == 2 * R2), "two-step lines only");
};

template <bool INV>
DDA_DEV float2 twid(const float2 *__restrict__ tw, int k)
{
    float2 w = __ldg(&tw[k]);
    if (INV) w.y = -w.y;
    return w;
}

// grid order of the x pass: right-hand side fastest where the Green octant outgrows L2, so that
// CTAs that run together read the same of its columns (128^3: 18.8 -> 18.4 ms per 42
// right-hand sides); smaller octants stay in L2, and there the spectral row first is faster
__host__ __device__ constexpr bool k2_rhs_fastest(int NI) { return NI >= 128; }

// ---- bulk asynchronous copies (the copy engine moves global rows into shared memory and
// signals an mbarrier; no multicast)
DDA_DEV unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

DDA_DEV void mbar_init(unsigned long long *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

DDA_DEV void mbar_expect_tx(unsigned long long *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

DDA_DEV void bulk_g2s(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
                     "r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// One tile of a 5-D tensor map (TMA, no multicast): the box at coordinates (x0 .. x4)
// into shared memory, completing on the mbarrier.  x0 is the innermost coordinate; its
// byte offset (x0 x 8) must be a multiple of 16, which the callers' column tiles keep.
DDA_DEV void tma_load_5d(void *dst, const CUtensorMap *map, int x0, int x1, int x2, int x3, int x4,
                         unsigned long long *bar)
{
    asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(smem_addr(dst)),
                 "l"(reinterpret_cast<unsigned long long>(map)), "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(x4),
                 "r"(smem_addr(bar))
                 : "memory");
}

// Waits for the barrier's phase `parity` to complete, at most `polls` polls; false if it did
// not (the caller reports it through the error flag instead of hanging).
DDA_DEV bool mbar_wait(unsigned long long *bar, unsigned parity, int polls = 1 << 22)
{
    const unsigned a = smem_addr(bar);
    for (int it = 0; it < polls; it++) {
        unsigned done;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(done)
                     : "r"(a), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}

// ---- packed form: a block takes 8 neighbouring zpos (a pair of z bins each: pair.cuh) of one
// spectral row, all components; threads (sub, t).  The pairs share every twiddle, so the
// transforms are packed instructions and shared-memory accesses are 16 bytes; rows are read and
// written as whole 128-byte lines.
constexpr int XC = 8;   // zpos per block

// one component's inputs (elements t2 + R2 k) through forward step A into shared memory
template <int NI>
DDA_DEV void pair_step_a(float4 *B, int c, P2 (&v)[Sx<NI>::R1], int sub, int t, const float2 *tw, const float2 *hw)
{
    using S = Sx<NI>;
    constexpr int R1 = S::R1, R2 = S::R2;
    auto put = [&](int h, int t2, P2(&u)[R1]) {
        dftp<R1, false>(u);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) {
            if (k1) u[k1] = pmul(u[k1], __ldg(&tw[t2 * k1]));
            B[((c * 2 + h) * NI + t2 + R2 * k1) * XC + t] = f4_of(u[k1]);
        }
    };
    if constexpr (R1 > R2) {   // each x half on its own lanes
        const int h = sub / R2, t2 = sub % R2;
        if (h) {
#pragma unroll
            for (int k = 0; k < R1; k++) v[k] = pmul(v[k], __ldg(&hw[t2 + R2 * k]));
        }
        put(h, t2, v);
    } else {
        P2 w[R1];
#pragma unroll
        for (int k = 0; k < R1; k++) w[k] = pmul(v[k], __ldg(&hw[sub + R2 * k]));
        put(0, sub, v);
        put(1, sub, w);
    }
}

// sum of three products of pairs; sg = -1 (G) or +1 (conj(G)) on the products of imaginary parts
DDA_DEV P2 dot3p(P2 a, P2 x, P2 b, P2 y, P2 c, P2 z, float2 sg, float2 ng)
{
    const float2 p = fma2(c.r, z.r, fma2(b.r, y.r, mul2(a.r, x.r)));
    const float2 q = fma2(c.i, z.i, fma2(b.i, y.i, mul2(a.i, x.i)));
    const float2 s = fma2(c.r, z.i, fma2(b.r, y.i, mul2(a.r, x.i)));
    const float2 t = fma2(c.i, z.r, fma2(b.i, y.r, mul2(a.i, x.r)));
    return {fma2(sg, q, p), fma2(ng, t, s)};
}

DDA_DEV float2 flip2(float2 v, unsigned m)   // sign flip by a mask of 0 or the sign bit
{
    return make_float2(__uint_as_float(__float_as_uint(v.x) ^ m), __uint_as_float(__float_as_uint(v.y) ^ m));
}

// Inverse step B of pairs whose step-A outputs u of lane k1 lie at R2 k1 + u (load(c, h, pos)):
// lane `sub`'s outputs, both x halves combined, to put(c, i, pair)
template <int NI, class Load, class Put>
DDA_DEV void pair_step_b(Load load, int sub, const float2 *hw, Put put)
{
    using S = Sx<NI>;
    constexpr int R1 = S::R1, R2 = S::R2;
    if constexpr (R1 > R2) {
        // lane (k1p, hb): outputs k2 = 2 m + hb, an R1/2-point inverse DFT of
        // y[n] = (x[n] + (-1)^hb x[n + R1/2]) exp(2 pi i n hb / R1)
        constexpr int H = R1 / 2;
        const int k1p = sub % R2, hb = sub / R2;
#pragma unroll 1
        for (int c = 0; c < 3; c++) {
            P2 e[H], o[H];
#pragma unroll
            for (int n = 0; n < H; n++) {
                const P2 e0 = load(c, 0, R2 * n + k1p), e1 = load(c, 0, R2 * (n + H) + k1p);
                const P2 o0 = load(c, 1, R2 * n + k1p), o1 = load(c, 1, R2 * (n + H) + k1p);
                if (hb) {
                    const float2 w = w16(n * (16 / R1));
                    e[n] = n ? pmulc(psub(e0, e1), w) : psub(e0, e1);
                    o[n] = n ? pmulc(psub(o0, o1), w) : psub(o0, o1);
                } else {
                    e[n] = padd(e0, e1);
                    o[n] = padd(o0, o1);
                }
            }
            dftp<H, true>(e);
            dftp<H, true>(o);
#pragma unroll
            for (int m = 0; m < H; m++) {
                const int i = k1p + R2 * (2 * m + hb);
                put(c, i, padd(e[m], pmulc(o[m], __ldg(&hw[i]))));
            }
        }
    } else {
#pragma unroll 1
        for (int c = 0; c < 3; c++) {
            P2 e[R1], o[R1];
#pragma unroll
            for (int q = 0; q < R1; q++) {
                e[q] = load(c, 0, R2 * q + sub);
                o[q] = load(c, 1, R2 * q + sub);
            }
            dftp<R1, true>(e);
            dftp<R1, true>(o);
#pragma unroll
            for (int k2 = 0; k2 < R1; k2++) {
                const int i = sub + R2 * k2;
                put(c, i, padd(e[k2], pmulc(o[k2], __ldg(&hw[i]))));
            }
        }
    }
}

// A block whose wait for its inputs ran out leaves its columns not a number, which the inverse
// spreads over the whole product: a caller that does not ask for the error flag sees it too.
// (A function of its own: inlined, its loop changes the kernels around it.)
__device__ __noinline__ void gave_up(float4 *col, size_t step, int n)
{
    const float nan = __int_as_float(0x7fffffff);
    for (int k = 0; k < n; k++) col[k * step] = make_float4(nan, nan, nan, nan);
}

template <int NI>
constexpr int pair_min_blocks() { return NI >= 128 ? 2 : NI >= 64 ? 4 : NI >= 32 ? 7 : 12; }

template <int NI, int LD>
__global__ void __launch_bounds__(Sx<NI>::RM * XC, pair_min_blocks<NI>())
k2q(MatvecArgs a, const __grid_constant__ CUtensorMap tmap)
{
    using S = Sx<NI>;
    constexpr int R1 = S::R1, R2 = S::R2;
    extern __shared__ __align__(128) float4 Bq[];   // [3][2][NI][XC]
    constexpr bool rhs_fast = k2_rhs_fastest(NI);
    const int js = rhs_fast ? blockIdx.z : blockIdx.x, rhs = rhs_fast ? blockIdx.x : blockIdx.z;
    chain_enter();
    if (a.rhs_active && !a.rhs_active[rhs]) return;
    const int nj = a.L.nj, nl = a.L.nl, z0 = blockIdx.y * XC;
    const int t = threadIdx.x % XC, sub = threadIdx.x / XC, col = z0 + t;
    const bool ok = col < nl;
    const size_t plane = (size_t)(2 * nj) * nl, cstr = (size_t)NI * plane;
    float4 *base = reinterpret_cast<float4 *>(a.work + (size_t)rhs * a.wstride) + (size_t)js * nl + col;
    const float2 *tw = a.L.tw_i, *hw = a.L.tw_i + NI;
    const int t2 = R1 > R2 ? sub % R2 : sub;
    auto at = [&](int c, int h, int pos) -> float4 & { return Bq[((c * 2 + h) * NI + pos) * XC + t]; };

    // ---- forward step A
    if constexpr (LD == 0) {
        P2 v[3][R1];
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int k = 0; k < R1; k++)
                v[c][k] = ok ? of_columns(base[c * cstr + (size_t)(t2 + R2 * k) * plane]) : pzero();
#pragma unroll
        for (int c = 0; c < 3; c++) pair_step_a<NI>(Bq, c, v[c], sub, t, tw, hw);
    } else {
        // the rows land as [i][t] in the half-0 slots; step A works in place
        __shared__ __align__(8) unsigned long long bar;
        const int w = nl - z0 < XC ? nl - z0 : XC;
        if (threadIdx.x == 0) {
            mbar_init(&bar, 1);
            mbar_expect_tx(&bar, 3u * NI * w * (unsigned)sizeof(float4));
        }
        __syncthreads();
        if constexpr (LD == 2) {
            if (threadIdx.x == 0)
#pragma unroll
                for (int c = 0; c < 3; c++) tma_load_5d(Bq + c * 2 * NI * XC, &tmap, 2 * z0, js, 0, c, rhs, &bar);
        } else {
            for (int q = threadIdx.x; q < 3 * NI; q += blockDim.x) {
                const int c = q / NI, i = q - c * NI;
                bulk_g2s(Bq + (c * 2 * NI + i) * XC, base - t + c * cstr + (size_t)i * plane,
                         w * (unsigned)sizeof(float4), &bar);
            }
        }
        // (self-test: after the copies, wait briefly for the next phase, which nothing completes)
        bool got = mbar_wait(&bar, 0);
        if (got && a.wait_selftest) got = mbar_wait(&bar, 1, 1 << 10);
        if (!__syncthreads_and(got)) {   // the same decision for every thread
            if (ok) gave_up(base + (size_t)sub * plane, (size_t)R1 * plane, 3 * NI / R1);
            if (threadIdx.x == 0 && a.err) atomicExch(a.err, 1);
            mbar_wait(&bar, 0);           // one more bounded wait for the copies in flight
            return;
        }
#pragma unroll 1
        for (int c = 0; c < 3; c++) {
            P2 v[R1];
#pragma unroll
            for (int k = 0; k < R1; k++) v[k] = ok ? of_columns(at(c, 0, t2 + R2 * k)) : pzero();
            __syncthreads();   // component c is read before its slots are rewritten
            pair_step_a<NI>(Bq, c, v, sub, t, tw, hw);
        }
    }
    __syncthreads();

    // ---- forward step B, product, inverse step A in place
    const int hj = js >= nj, jp = 2 * (js - hj * nj) + hj;
    const bool by = jp > nj;
    const int lp = ok ? z_bin(2 * col, nl, a.zs) : 0;
    // (at the bins lp = nl and kx = NI, where the mirrored halves meet, the odd components vanish)
    const bool bz = lp >= nl;
    const unsigned sign = 0x80000000u, my = by ? sign : 0u, mz = bz ? sign : 0u;
    const size_t sp = z_entries(nl, a.zs), sy = 3 * sp, sxo = (size_t)(nj + 1) * sy;
    const float4 *G0 = a.ahat + (size_t)(by ? 2 * nj - jp : jp) * sy;
    const int e0 = z_order(bz ? 2 * nl - lp : lp, nl, a.zs, z_parity_split(NI)), e1 = z_order(bz ? 2 * nl - lp - 1 : lp + 1, nl, a.zs, z_parity_split(NI));
    const float2 sg = dup2(a.conj ? 1.f : -1.f), ng = dup2(a.conj ? -1.f : 1.f);
    const int k1 = sub;
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
        P2 X[3][R2];
#pragma unroll
        for (int c = 0; c < 3; c++) {
#pragma unroll
            for (int q = 0; q < R2; q++) X[c][q] = p_of(at(c, h, R2 * k1 + q));
            dftp<R2, false>(X[c]);
        }
#pragma unroll
        for (int q = 0; q < R2; q++) {
            const int kx = 2 * (k1 + R1 * q) + h;
            const bool bx = 2 * q >= R2;
            const unsigned mx = bx ? sign : 0u;
            const float4 *G = G0 + (size_t)(bx ? 2 * NI - kx : kx) * sxo;
            P2 g[6];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const float4 u = __ldg(G + k * sp + e0), w = __ldg(G + k * sp + e1);
                g[2 * k] = {make_float2(u.x, w.x), make_float2(u.y, w.y)};
                g[2 * k + 1] = {make_float2(u.z, w.z), make_float2(u.w, w.w)};
            }
            g[1] = {flip2(g[1].r, mx ^ my), flip2(g[1].i, mx ^ my)};
            g[2] = {flip2(g[2].r, mx ^ mz), flip2(g[2].i, mx ^ mz)};
            g[4] = {flip2(g[4].r, my ^ mz), flip2(g[4].i, my ^ mz)};
            const P2 x = X[0][q], y = X[1][q], z = X[2][q];
            X[0][q] = dot3p(g[0], x, g[1], y, g[2], z, sg, ng);
            X[1][q] = dot3p(g[1], x, g[3], y, g[4], z, sg, ng);
            X[2][q] = dot3p(g[2], x, g[4], y, g[5], z, sg, ng);
        }
        // transposed split: lane k1's outputs u stay where it read
#pragma unroll
        for (int c = 0; c < 3; c++) {
            dftp<R2, true>(X[c]);
#pragma unroll
            for (int u = 0; u < R2; u++) {
                if (u) X[c][u] = pmulc(X[c][u], __ldg(&tw[k1 * u]));
                at(c, h, R2 * k1 + u) = f4_of(X[c][u]);
            }
        }
    }
    __syncthreads();

    // ---- inverse step B, combine, store
    pair_step_b<NI>([&](int c, int h, int pos) { return p_of(at(c, h, pos)); }, sub, hw, [&](int c, int i, P2 v) {
        if (ok) base[c * cstr + i * plane] = columns_of(v);
    });
}

// ---- unpacked form, edge 64: a block takes TL neighbouring columns, one complex number per
// access.  16.4 M warp instructions per right-hand side against 10.9 M packed ones, but twice the
// warps (16 per SM, 128 registers): 18.4 against 21 us at 24 right-hand sides.
template <int NI, int TL>
__global__ void __launch_bounds__(Sx<NI>::RM * TL, 512 / (Sx<NI>::RM * TL)) k2f(MatvecArgs a)
{
    using S = Sx<NI>;
    constexpr int R1 = S::R1, R2 = S::R2;
    static_assert(R1 == R2, "square line splits");
    extern __shared__ __align__(128) float2 B[];   // [6][NI][TL]
    const int js = blockIdx.x, rhs = blockIdx.z;
    chain_enter();
    if (a.rhs_active && !a.rhs_active[rhs]) return;
    const int nj = a.L.nj, nl = a.L.nl;
    const int l0 = blockIdx.y * TL;
    const int t = threadIdx.x % TL, sub = threadIdx.x / TL;
    const size_t plane = (size_t)(2 * nj) * (2 * nl), cstr = (size_t)NI * plane;
    float2 *base = a.work + (size_t)rhs * a.wstride + (size_t)js * (2 * nl) + l0 + t;
    const float2 *tw = a.L.tw_i, *hw = a.L.tw_i + NI;
    auto Bat = [&](int c, int h, int pos) -> float2 & { return B[((c * 2 + h) * NI + pos) * TL + t]; };

    // ---- forward step A (both halves from one load)
    {
        // step A of one component from its R1 loaded values
        auto step_a = [&](int c, float2 (&v)[R1]) {
            float2 w[R1];
#pragma unroll
            for (int r = 0; r < R1; r++) w[r] = cmul(v[r], __ldg(&hw[sub + R2 * r]));
            dft_reg<R1, false>(v);
            dft_reg<R1, false>(w);
#pragma unroll
            for (int k1 = 0; k1 < R1; k1++) {
                const float2 tk = k1 ? twid<false>(tw, sub * k1) : make_float2(1.f, 0.f);
                Bat(c, 0, sub + R2 * k1) = k1 ? cmul(v[k1], tk) : v[k1];
                Bat(c, 1, sub + R2 * k1) = k1 ? cmul(w[k1], tk) : w[k1];
            }
        };
        {
            // all three components' loads in flight before any arithmetic
            float2 v0[R1], v1[R1], v2[R1];
#pragma unroll
            for (int r = 0; r < R1; r++) {
                const size_t o = (size_t)(sub + R2 * r) * plane;
                v0[r] = base[o];
                v1[r] = base[cstr + o];
                v2[r] = base[2 * cstr + o];
            }
            step_a(0, v0);
            step_a(1, v1);
            step_a(2, v2);
        }
    }
    __syncthreads();

    // ---- forward step B, product with the Green tensor, inverse step A
    const int hj = js >= nj, kj = js - hj * nj, jp = 2 * kj + hj;
    const int my = jp > nj, oy = my ? 2 * nj - jp : jp;
    const int lp = z_bin(l0 + t, nl, a.zs), mz = lp > nl, oz = mz ? 2 * nl - lp : lp;
    // [ox][oy][3][z_order(oz)], two components per float4
    const size_t sp = z_entries(nl, a.zs), sy = 3 * sp, sxo = (size_t)(nj + 1) * sy;
    const float4 *Ayz = a.ahat + (size_t)oy * sy + z_order(oz, nl, a.zs, z_parity_split(NI));
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
        float2 X[3][R2];
        const int k1 = sub;
#pragma unroll
        for (int c = 0; c < 3; c++) {
#pragma unroll
            for (int q = 0; q < R2; q++) X[c][q] = Bat(c, h, R2 * k1 + q);
            dft_reg<R2, false>(X[c]);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < R2; q++) {
            const int kx = 2 * (k1 + R1 * q) + h, mx = kx > NI, ox = mx ? 2 * NI - kx : kx;
            const float4 *A = Ayz + (size_t)ox * sxo;
            const float4 a01 = __ldg(A), a23 = __ldg(A + sp), a45 = __ldg(A + 2 * sp);
            float2 g0 = make_float2(a01.x, a01.y), g1 = make_float2(a01.z, a01.w),
                   g2 = make_float2(a23.x, a23.y), g3 = make_float2(a23.z, a23.w),
                   g4 = make_float2(a45.x, a45.y), g5 = make_float2(a45.z, a45.w);
            if (mx ^ my) g1 = cscale(g1, -1.f);
            if (mx ^ mz) g2 = cscale(g2, -1.f);
            if (my ^ mz) g4 = cscale(g4, -1.f);
            if (a.conj) {
                g0 = cconj(g0); g1 = cconj(g1); g2 = cconj(g2);
                g3 = cconj(g3); g4 = cconj(g4); g5 = cconj(g5);
            }
            const float2 vx = X[0][q], vy = X[1][q], vz = X[2][q];
            X[0][q] = cadd(cadd(cmul(g0, vx), cmul(g1, vy)), cmul(g2, vz));
            X[1][q] = cadd(cadd(cmul(g1, vx), cmul(g3, vy)), cmul(g4, vz));
            X[2][q] = cadd(cadd(cmul(g2, vx), cmul(g4, vy)), cmul(g5, vz));
        }
        // inverse step A with the transposed split: lane k1 owns positions k1 + R1 q
#pragma unroll
        for (int c = 0; c < 3; c++) {
            dft_reg<R2, true>(X[c]);
#pragma unroll
            for (int u = 0; u < R2; u++) {
                const float2 y = u ? cmul(X[c][u], twid<true>(tw, k1 * u)) : X[c][u];
                Bat(c, h, k1 + R1 * u) = y;
            }
        }
        __syncthreads();
    }

    // ---- inverse step B (transposed split: R2 lanes of R1 elements), combine, store
    {
        const int k1p = sub;
#pragma unroll 1
        for (int c = 0; c < 3; c++) {
            float2 e[R1], o[R1];
#pragma unroll
            for (int q = 0; q < R1; q++) {
                e[q] = Bat(c, 0, R1 * k1p + q);
                o[q] = Bat(c, 1, R1 * k1p + q);
            }
            dft_reg<R1, true>(e);
            dft_reg<R1, true>(o);
#pragma unroll
            for (int k2 = 0; k2 < R1; k2++) {
                const int i = k1p + R2 * k2;
                base[c * cstr + i * plane] = cadd(e[k2], cmulc(o[k2], __ldg(&hw[i])));
            }
        }
    }
}

// Pair form of the x pass (MatvecArgs::pair, step 0): CTA (spectral row js, TL spectral columns,
// polarisation pair k).  The forward transform of phi (component slot 0 of right-hand side
// 2k) is done once, its two x halves as one packed pair, and stays in registers; then both
// polarisations' spectra G (E_q phi) go through the product and the inverse transforms as
// packed pairs, so a Green entry is loaded once for the two, and are written to the three
// component slots of right-hand sides 2k and 2k + 1.
// Bound by the L1 data path (74% of its wavefronts: the packed exchange of the inverse, then
// Green and the stores); 64^3, 128 right-hand sides: 1700 us, 1909 with one polarisation at a time.
template <int NI, int TL>
__global__ void __launch_bounds__(Sx<NI>::RM * TL, pair_min_blocks<NI>() * XC / TL) k2r(MatvecArgs a)
{
    using S = Sx<NI>;
    constexpr int R1 = S::R1, R2 = S::R2;
    extern __shared__ __align__(128) float4 Bq[];   // [3][2][NI][TL]
    constexpr bool rhs_fast = k2_rhs_fastest(NI);
    const int js = rhs_fast ? blockIdx.z : blockIdx.x, rhs0 = 2 * (rhs_fast ? blockIdx.x : blockIdx.z);
    chain_enter();
    if (a.rhs_active && !a.rhs_active[rhs0]) return;
    const int nj = a.L.nj, nl = a.L.nl, t = threadIdx.x % TL, sub = threadIdx.x / TL, col = blockIdx.y * TL + t;
    const size_t plane = (size_t)(2 * nj) * (2 * nl), cstr = (size_t)NI * plane, off = (size_t)js * (2 * nl) + col;
    const float2 *tw = a.L.tw_i, *hw = a.L.tw_i + NI;
    auto at = [&](int c, int h, int pos) -> float4 & { return Bq[((c * 2 + h) * NI + pos) * TL + t]; };

    // ---- phi forward, pair = (x half 0, x half 1)
    if (sub < R2) {
        const float2 *src = a.work + (size_t)rhs0 * a.wstride + off;
        float2 v[R1];
        P2 u[R1];
#pragma unroll
        for (int k = 0; k < R1; k++) v[k] = src[(size_t)(sub + R2 * k) * plane];
#pragma unroll
        for (int k = 0; k < R1; k++) u[k] = ppack(v[k], cmul(v[k], __ldg(&hw[sub + R2 * k])));
        dftp<R1, false>(u);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) {
            if (k1) u[k1] = pmul(u[k1], __ldg(&tw[sub * k1]));
            at(0, 0, sub + R2 * k1) = f4_of(u[k1]);
        }
    }
    __syncthreads();
    P2 F[R2];   // bins 2 (k1 + R1 q) + h
#pragma unroll
    for (int q = 0; q < R2; q++) F[q] = p_of(at(0, 0, R2 * sub + q));
    dftp<R2, false>(F);
    __syncthreads();

    // ---- products, inverse step A (transposed split); pair = (polarisation 0, polarisation 1)
    const int hj = js >= nj, jp = 2 * (js - hj * nj) + hj;
    const bool by = jp > nj;
    const int lp = z_bin(col, nl, a.zs);
    const bool bz = lp > nl;
    const unsigned sign = 0x80000000u, my = by ? sign : 0u, mz = bz ? sign : 0u;
    const size_t sp = z_entries(nl, a.zs), sy = 3 * sp, sxo = (size_t)(nj + 1) * sy;
    const float4 *G0 = a.ahat + (size_t)(by ? 2 * nj - jp : jp) * sy + z_order(bz ? 2 * nl - lp : lp, nl, a.zs, z_parity_split(NI));
    const double *E0 = a.einc + 6 * rhs0, *E1 = E0 + 6;
    P2 E[3];
#pragma unroll
    for (int c = 0; c < 3; c++)
        E[c] = {make_float2((float)E0[2 * c], (float)E1[2 * c]), make_float2((float)E0[2 * c + 1], (float)E1[2 * c + 1])};
    // real incident fields (every rotated x or y polarisation): G E with real weights, then one
    // complex product per component; the branch is taken once, outside the unrolled loops
    bool real = true;
#pragma unroll
    for (int c = 0; c < 3; c++) real = real && E[c].i.x == 0.f && E[c].i.y == 0.f;
    const int k1 = sub;
    auto product = [&](auto real_tag) {
        constexpr bool REAL = decltype(real_tag)::value;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            P2 X[3][R2];
#pragma unroll
            for (int q = 0; q < R2; q++) {
                const int kx = 2 * (k1 + R1 * q) + h;
                const bool bx = 2 * q >= R2;   // (at kx = NI the odd components vanish)
                const unsigned mx = bx ? sign : 0u;
                const float4 *G = G0 + (size_t)(bx ? 2 * NI - kx : kx) * sxo;
                const float4 a01 = __ldg(G), a23 = __ldg(G + sp), a45 = __ldg(G + 2 * sp);
                const float2 g0 = make_float2(a01.x, a01.y), g1 = flip2(make_float2(a01.z, a01.w), mx ^ my),
                             g2 = flip2(make_float2(a23.x, a23.y), mx ^ mz), g3 = make_float2(a23.z, a23.w),
                             g4 = flip2(make_float2(a45.x, a45.y), my ^ mz), g5 = make_float2(a45.z, a45.w);
                const float2 f = h ? psecond(F[q]) : pfirst(F[q]);
                auto row = [&](float2 ga, float2 gb, float2 gc) {
                    P2 u;
                    if constexpr (REAL) {
                        u = {fma2(dup2(ga.x), E[0].r, fma2(dup2(gb.x), E[1].r, mul2(dup2(gc.x), E[2].r))),
                             fma2(dup2(ga.y), E[0].r, fma2(dup2(gb.y), E[1].r, mul2(dup2(gc.y), E[2].r)))};
                    } else {
                        u = padd(padd(pmul(E[0], ga), pmul(E[1], gb)), pmul(E[2], gc));
                    }
                    return pmul(u, f);
                };
                X[0][q] = row(g0, g1, g2);
                X[1][q] = row(g1, g3, g4);
                X[2][q] = row(g2, g4, g5);
            }
#pragma unroll
            for (int c = 0; c < 3; c++) {
                dftp<R2, true>(X[c]);
#pragma unroll
                for (int u = 0; u < R2; u++) {
                    if (u) X[c][u] = pmulc(X[c][u], __ldg(&tw[k1 * u]));
                    at(c, h, R2 * k1 + u) = f4_of(X[c][u]);
                }
            }
        }
    };
    if (real) product(std::true_type{});
    else product(std::false_type{});
    __syncthreads();

    // ---- inverse step B, combine, store
    float2 *b0 = a.work + (size_t)rhs0 * a.wstride + off, *b1 = b0 + a.wstride;
    auto store = [&](int c, int i, P2 v) {
        b0[c * cstr + i * plane] = pfirst(v);
        b1[c * cstr + i * plane] = psecond(v);
    };
    pair_step_b<NI>([&](int c, int h, int pos) { return p_of(at(c, h, pos)); }, sub, hw, store);
}

// ---- launches
template <int NI, int LD>
cudaError_t launch_packed(const MatvecArgs &a, cudaStream_t st)
{
    const unsigned ct = (unsigned)((a.L.nl + XC - 1) / XC), js = 2 * a.L.nj;
    static const CUtensorMap none{};
    const CUtensorMap &map = LD == 2 ? *static_cast<const CUtensorMap *>(a.tmaps) : none;
    return launch_chained(a.chained, k2q<NI, LD>, k2_rhs_fastest(NI) ? dim3(a.nrhs, ct, js) : dim3(js, ct, a.nrhs),
                          Sx<NI>::RM * XC, 6 * NI * XC * sizeof(float4), st, 1, a, map);
}

template <int TL>
cudaError_t launch_unpacked(const MatvecArgs &a, cudaStream_t st)
{
    return launch_chained(a.chained, k2f<64, TL>, dim3(2 * a.L.nj, 2 * a.L.nl / TL, a.nrhs), Sx<64>::RM * TL,
                          (size_t)6 * 64 * TL * sizeof(float2), st, 1, a);
}

// columns per CTA of the pair form: whole 128-byte lines where two CTAs of that size fit an SM's
// registers (edges up to 32: 229 against 247 us at 32^3 x 128), 8 at 64 and 128 (1.80 against
// 1.87 and 1.98 against 2.20 ms)
template <int NI>
constexpr int pair_columns() { return NI <= 32 ? 16 : 8; }

template <int NI, int TL>
cudaError_t launch_pair(const MatvecArgs &a, cudaStream_t st)
{
    const unsigned ct = 2 * a.L.nl / TL, js = 2 * a.L.nj, np = a.nrhs / 2;
    return launch_chained(a.chained, k2r<NI, TL>, k2_rhs_fastest(NI) ? dim3(np, ct, js) : dim3(js, ct, np),
                          Sx<NI>::RM * TL, (size_t)6 * NI * TL * sizeof(float4), st, 1, a);
}

// x variants: 0..2 the unpacked form with 32 / 16 / 8 columns at edge 64 (packed with register
// loads elsewhere); the packed form with bulk copies of the rows (3..5), register loads (6..8)
// or one TMA tensor tile per component (9..11; register loads where a row is shorter)
template <int NI>
cudaError_t launch_x(const MatvecArgs &a, cudaStream_t st)
{
    if (a.inc && a.pair) {
        if (2 * a.L.nl >= pair_columns<NI>()) return launch_pair<NI, pair_columns<NI>()>(a, st);
        return launch_pair<NI, 8>(a, st);
    }
    if constexpr (NI == 64) {
        if (a.fx < 3) {
            // the widest tile of the variant that the row holds
            const int tl = 32 >> a.fx;
            if (tl >= 32 && 2 * a.L.nl >= 32) return launch_unpacked<32>(a, st);
            if (tl >= 16 && 2 * a.L.nl >= 16) return launch_unpacked<16>(a, st);
            return launch_unpacked<8>(a, st);
        }
    }
    if (a.fx >= 9 && a.L.nl >= XC) return launch_packed<NI, 2>(a, st);
    if (a.fx >= 3 && a.fx < 6) return launch_packed<NI, 1>(a, st);
    return launch_packed<NI, 0>(a, st);
}

// the kernel that launch_x takes for the same arguments
template <int NI>
cudaError_t prep_x(int nl, int fx, int form)
{
    auto set = [](const void *k, size_t bytes) { return raise_smem_limit(k, (int)bytes); };
    if (form == 2) {
        constexpr int PC = pair_columns<NI>();
        if (2 * nl >= PC) return set((const void *)k2r<NI, PC>, (size_t)6 * NI * PC * sizeof(float4));
        return set((const void *)k2r<NI, 8>, (size_t)6 * NI * 8 * sizeof(float4));
    }
    if constexpr (NI == 64) {
        constexpr size_t C = (size_t)6 * 64 * sizeof(float2);
        if (fx == 0 && 2 * nl >= 32) return set((const void *)k2f<64, 32>, 32 * C);
        if (fx < 2 && 2 * nl >= 16) return set((const void *)k2f<64, 16>, 16 * C);
        if (fx < 3) return set((const void *)k2f<64, 8>, 8 * C);
    }
    constexpr size_t P = (size_t)6 * NI * XC * sizeof(float4);
    if (fx >= 9 && nl >= XC) return set((const void *)k2q<NI, 2>, P);
    if (fx >= 3 && fx < 6) return set((const void *)k2q<NI, 1>, P);
    return set((const void *)k2q<NI, 0>, P);
}

}  // namespace

template <>
cudaError_t x_prepare<X_NI>(int nl, int fx, int form) { return prep_x<X_NI>(nl, fx, form); }

template <>
cudaError_t x_launch<X_NI>(const MatvecArgs &a, cudaStream_t st)
{
    return launch_x<X_NI>(a, st);
}

}  // namespace ddagpu
