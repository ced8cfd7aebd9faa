// x pass of the matvec for lattice edges 4..128: forward along i, symmetric 3x3 product with the
// Green tensor, inverse along i, in place on the work buffer of matvec_yz.cu, whose rows are 2 nl
// complex columns (column 2 zpos + h holds the z bin 2 kl + h).
//
// Every n-point line uses n = R1 R2: a thread (sub, col), consecutive lanes on consecutive
// columns, holds R1 elements of a line for step A and R2 elements for step B, and the steps
// exchange data through shared memory.  An even / odd pair of transforms covers the padded
// line: bins 2 k + h are DFT_n(x W_2n^(h j)), and the inverse keeps the first n outputs.
//
// What bounds it: bytes through the L1 data path -- at 64^3 and per right-hand side 50 MB of
// columns and 100 MB of Green tensor in (64 bytes per SM and clock from L2), 50 MB out and
// 200 MB through shared memory, 16 us in all; FP32 is 9 us and DRAM 8 us of it.
// Compiled once per x edge (X_NI).
#include <cuda.h>   // CUtensorMap (the type only; maps are encoded in ddagpu.cu)

#include <type_traits>

#include "internal.h"
#include "pair.cuh"
#include "zorder.cuh"

namespace ddagpu {

namespace {

// The x pass's line factorisation N = R1 R2: ALT 0 is line_split<N>; ALT 1 the second
// schedule the autotuner may pick -- the two factors swapped, or for a square split
// 2 R1 x R2 / 2 (16: 8 x 2, 32: 4 x 8, 64: 16 x 4, 128: 8 x 16).  The reference chooses
// among radix-8/4/2 stage sequences per length the same way (fft_kernel.hpp:210-263).
template <int N, int ALT>
struct Sx {
    static constexpr int A1 = line_split<N>::R1, A2 = line_split<N>::R2;
    static constexpr bool SW = ALT != 0 && N > 4;
    static constexpr int R1 = !SW ? A1 : (A1 == A2 ? 2 * A1 : A2);
    static constexpr int R2 = !SW ? A2 : (A1 == A2 ? A2 / 2 : A1);
    static constexpr int RM = R1 > R2 ? R1 : R2;
    static_assert(R1 * R2 == N && R1 <= 16 && R2 <= 16, "bad line factorisation");
};

template <bool INV>
DDA_DEV float2 twid(const float2 *__restrict__ tw, int k)
{
    float2 w = __ldg(&tw[k]);
    if (INV) w.y = -w.y;
    return w;
}

// ------------------------------------------------------------------------------ K2
// CTA (spectral row js, TL spectral columns): forward x (both halves), 3x3 product,
// inverse x, in place.  Shared B[c][h][pos][t].
// grid order of the x pass: right-hand side fastest where the Green octant outgrows L2
__host__ __device__ constexpr bool k2_rhs_fastest(int NI) { return NI >= 128; }

// at least this many CTAs per SM: about 128 registers a thread (80 for the 16-point lines)
constexpr int k2_min_blocks(int NI, int threads)
{
    return NI <= 16 ? (6 * 128 / threads < 16 ? 6 * 128 / threads : 16) : (512 / threads > 0 ? 512 / threads : 1);
}

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

// LD: how the input columns reach the CTA -- 0 register loads, 1 one bulk copy per row,
// 2 one TMA tensor tile per component (tmap: the work buffer as [rhs][c][i][js][ls] with
// the box TL x 1 x NI; unused otherwise)
template <int NI, int TL, int LD, int ALT>
__global__ void __launch_bounds__(Sx<NI, ALT>::RM * TL, k2_min_blocks(NI, Sx<NI, ALT>::RM * TL))
k2f(MatvecArgs a, const __grid_constant__ CUtensorMap tmap)
{
    using S = Sx<NI, ALT>;
    constexpr bool BULK = LD != 0;
    static_assert(!BULK || ALT == 0, "bulk copies with the default factorisation only");
    constexpr int R1 = S::R1, R2 = S::R2, RM = S::RM;
    extern __shared__ __align__(128) float2 B[];   // [6][NI][TL]
    // at edge 128 the right-hand side is the fastest grid index: CTAs that run together
    // read the same Green-tensor columns, which then come from L2 (that octant, 103 MB,
    // does not stay resident while a whole right-hand side streams through; 18.8 -> 18.4 ms
    // per 42-RHS matvec).  Smaller octants stay in L2, and there the spectral row first
    // is faster (64^3, 128 RHS: 2.42 vs 2.63 ms for this pass)
    constexpr bool rhs_fast = k2_rhs_fastest(NI);
    const int js = rhs_fast ? blockIdx.z : blockIdx.x, rhs = rhs_fast ? blockIdx.x : blockIdx.z;
    if (a.rhs_active && !a.rhs_active[rhs]) return;
    const int nj = a.L.nj, nl = a.L.nl;
    const int l0 = blockIdx.y * TL;
    const int t = threadIdx.x % TL, sub = threadIdx.x / TL;
    const size_t plane = (size_t)(2 * nj) * (2 * nl), cstr = (size_t)NI * plane;
    float2 *base = a.work + (size_t)rhs * a.wstride + (size_t)js * (2 * nl) + l0 + t;
    const float2 *tw = a.L.tw_i, *hw = a.L.tw_i + NI;
    auto Bat = [&](int c, int h, int pos) -> float2 & { return B[((c * 2 + h) * NI + pos) * TL + t]; };

    // ---- bulk variant: the 3 x NI input rows of TL columns arrive in the half-0 planes of B
    // by asynchronous bulk copies (one per row, 16-byte aligned: l0 and TL are multiples
    // of 4 float2); step A then reads them from shared memory and works in place
    if constexpr (BULK) {
        __shared__ __align__(8) unsigned long long bar;
        if (threadIdx.x == 0) {
            mbar_init(&bar, 1);
            mbar_expect_tx(&bar, 3u * NI * TL * (unsigned)sizeof(float2));
        }
        __syncthreads();
        if constexpr (LD == 2) {
            // three tensor tiles: component c's NI x TL columns land as [i][t] in half 0
            if (threadIdx.x == 0)
#pragma unroll
                for (int c = 0; c < 3; c++) tma_load_5d(&B[(c * 2) * NI * TL], &tmap, l0, js, 0, c, rhs, &bar);
        } else {
            const float2 *row0 = a.work + (size_t)rhs * a.wstride + (size_t)js * (2 * nl) + l0;
            for (int q = threadIdx.x; q < 3 * NI; q += blockDim.x) {
                const int c = q / NI, i = q - c * NI;
                bulk_g2s(&B[((c * 2) * NI + i) * TL], row0 + c * cstr + (size_t)i * plane,
                         TL * (unsigned)sizeof(float2), &bar);
            }
        }
        // (self-test: after the copies, wait briefly for the next phase, which nothing completes)
        bool got = mbar_wait(&bar, 0);
        if (got && a.wait_selftest) got = mbar_wait(&bar, 1, 1 << 10);
        if (!__syncthreads_and(got)) {   // the same decision for every thread
            if (threadIdx.x == 0 && a.err) atomicExch(a.err, 1);
            mbar_wait(&bar, 0);           // one more bounded wait for the copies in flight
            return;
        }
        if constexpr (R1 == 2 * R2) {
            // R1 = 2 R2 (edges 32, 128): every lane works -- lane (t2, hb) transforms half hb
            // (hb = 1: the input times W_2NI^m) of the lines t2 + R2 r
            const int t2 = sub % R2, hb = sub / R2;
#pragma unroll 1
            for (int c = 0; c < 3; c++) {
                float2 v[R1];
#pragma unroll
                for (int r = 0; r < R1; r++) {
                    v[r] = Bat(c, 0, t2 + R2 * r);
                    if (hb) v[r] = cmul(v[r], __ldg(&hw[t2 + R2 * r]));
                }
                __syncthreads();   // half 0 of component c is read by both lane halves before it is rewritten
                dft_reg<R1, false>(v);
#pragma unroll
                for (int k1 = 0; k1 < R1; k1++) {
                    const float2 tk = k1 ? twid<false>(tw, t2 * k1) : make_float2(1.f, 0.f);
                    Bat(c, hb, t2 + R2 * k1) = k1 ? cmul(v[k1], tk) : v[k1];
                }
            }
        } else if (sub < R2) {
            auto step_a_smem = [&](int c) {
                float2 v[R1], w[R1];
#pragma unroll
                for (int r = 0; r < R1; r++) {
                    v[r] = Bat(c, 0, sub + R2 * r);
                    w[r] = cmul(v[r], __ldg(&hw[sub + R2 * r]));
                }
                dft_reg<R1, false>(v);
                dft_reg<R1, false>(w);
#pragma unroll
                for (int k1 = 0; k1 < R1; k1++) {
                    const float2 tk = k1 ? twid<false>(tw, sub * k1) : make_float2(1.f, 0.f);
                    Bat(c, 0, sub + R2 * k1) = k1 ? cmul(v[k1], tk) : v[k1];
                    Bat(c, 1, sub + R2 * k1) = k1 ? cmul(w[k1], tk) : w[k1];
                }
            };
#pragma unroll 1
            for (int c = 0; c < 3; c++) step_a_smem(c);
        }
    } else
    // ---- forward step A (both halves from one load)
    if (sub < R2) {
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
        if constexpr (BULK) {
            // unreachable: the bulk variant loads below, before this branch
        } else if constexpr (3 * R1 <= 24) {
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
        } else {
#pragma unroll 1
            for (int c = 0; c < 3; c++) {
                float2 v[R1];
#pragma unroll
                for (int r = 0; r < R1; r++) v[r] = base[c * cstr + (size_t)(sub + R2 * r) * plane];
                step_a(c, v);
            }
        }
    }
    __syncthreads();

    // ---- forward step B, product with the Green tensor, inverse step A
    const int hj = js >= nj, kj = js - hj * nj, jp = 2 * kj + hj;
    const int my = jp > nj, oy = my ? 2 * nj - jp : jp;
    const int lp = z_bin(l0 + t, nl, a.zs), mz = lp > nl, oz = mz ? 2 * nl - lp : lp;
    // [ox][oy][3][z_order(oz)], two components per float4: the lanes of each parity read runs
    // of consecutive float4s
    const size_t sp = z_entries(nl, a.zs), sy = 3 * sp, sxo = (size_t)(nj + 1) * sy;
    const float4 *Ayz = a.aq + (size_t)oy * sy + z_order(oz, nl, a.zs);
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
        float2 X[3][R2];
        const bool act = sub < R1;
        const int k1 = sub;
        if (act) {
#pragma unroll
            for (int c = 0; c < 3; c++) {
#pragma unroll
                for (int q = 0; q < R2; q++) X[c][q] = Bat(c, h, R2 * k1 + q);
                dft_reg<R2, false>(X[c]);
            }
        }
        __syncthreads();
        if (act) {
            {
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
            }
        }
        __syncthreads();
    }

    // ---- inverse step B (transposed split: R2 lanes of R1 elements), combine, store
    if constexpr (R1 == 2 * R2) {
        // every lane works: lane (k1p, hb) produces the outputs k2 = 2 m + hb of its lines,
        // an R1/2-point inverse DFT of y[n] = (x[n] + (-1)^hb x[n + R1/2]) exp(2 pi i n hb / R1)
        const int k1p = sub % R2, hb = sub / R2;
        constexpr int H = R1 / 2;
#pragma unroll 1
        for (int c = 0; c < 3; c++) {
            float2 e[H], o[H];
#pragma unroll
            for (int n = 0; n < H; n++) {
                const float2 e0 = Bat(c, 0, R1 * k1p + n), e1 = Bat(c, 0, R1 * k1p + n + H);
                const float2 o0 = Bat(c, 1, R1 * k1p + n), o1 = Bat(c, 1, R1 * k1p + n + H);
                if (hb) {
                    const float2 wn = cconj(w16(n * (16 / R1)));
                    e[n] = n ? cmul(csub(e0, e1), wn) : csub(e0, e1);
                    o[n] = n ? cmul(csub(o0, o1), wn) : csub(o0, o1);
                } else {
                    e[n] = cadd(e0, e1);
                    o[n] = cadd(o0, o1);
                }
            }
            dft_reg<H, true>(e);
            dft_reg<H, true>(o);
#pragma unroll
            for (int m = 0; m < H; m++) {
                const int i = k1p + R2 * (2 * m + hb);
                base[c * cstr + i * plane] = cadd(e[m], cmulc(o[m], __ldg(&hw[i])));
            }
        }
    } else if (sub < R2) {
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

// Pair form of the x pass (MatvecArgs::pair, step 0): CTA (spectral row js, TL spectral
// columns, polarisation pair k).  The forward transform of phi (component slot 0 of
// right-hand side 2k) is done once; then for each polarisation q the spectrum G (E_q phi)
// is formed -- the product of the single form with v = E_q phi -- inverse-transformed and
// written to the three component slots of right-hand side 2k + q.  Shared B[c][h][pos][t]
// with c = 0..2 the output components and c = 3 the spectrum of phi.
template <int NI, int TL>
__global__ void __launch_bounds__(Sx<NI, 0>::RM * TL, k2_min_blocks(NI, Sx<NI, 0>::RM * TL)) k2p(MatvecArgs a)
{
    using S = Sx<NI, 0>;
    constexpr int R1 = S::R1, R2 = S::R2;
    extern __shared__ __align__(128) float2 B[];   // [4][2][NI][TL]
    constexpr bool rhs_fast = k2_rhs_fastest(NI);
    const int js = rhs_fast ? blockIdx.z : blockIdx.x, pr = rhs_fast ? blockIdx.x : blockIdx.z;
    const int rhs0 = 2 * pr;
    if (a.rhs_active && !a.rhs_active[rhs0]) return;
    const int nj = a.L.nj, nl = a.L.nl;
    const int l0 = blockIdx.y * TL;
    const int t = threadIdx.x % TL, sub = threadIdx.x / TL;
    const size_t plane = (size_t)(2 * nj) * (2 * nl), cstr = (size_t)NI * plane;
    const size_t col = (size_t)js * (2 * nl) + l0 + t;
    const float2 *tw = a.L.tw_i, *hw = a.L.tw_i + NI;
    auto Bat = [&](int c, int h, int pos) -> float2 & { return B[((c * 2 + h) * NI + pos) * TL + t]; };

    // ---- forward step A of phi, both halves from one load
    if (sub < R2) {
        const float2 *src = a.work + (size_t)rhs0 * a.wstride + col;
        float2 v[R1], w[R1];
#pragma unroll
        for (int r = 0; r < R1; r++) v[r] = src[(size_t)(sub + R2 * r) * plane];
#pragma unroll
        for (int r = 0; r < R1; r++) w[r] = cmul(v[r], __ldg(&hw[sub + R2 * r]));
        dft_reg<R1, false>(v);
        dft_reg<R1, false>(w);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) {
            const float2 tk = k1 ? twid<false>(tw, sub * k1) : make_float2(1.f, 0.f);
            Bat(3, 0, sub + R2 * k1) = k1 ? cmul(v[k1], tk) : v[k1];
            Bat(3, 1, sub + R2 * k1) = k1 ? cmul(w[k1], tk) : w[k1];
        }
    }
    __syncthreads();
    // ---- forward step B of phi, in place: lane k1 keeps frequencies k1 + R1 q at R2 k1 + q
    if (sub < R1) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float2 X[R2];
#pragma unroll
            for (int q = 0; q < R2; q++) X[q] = Bat(3, h, R2 * sub + q);
            dft_reg<R2, false>(X);
#pragma unroll
            for (int q = 0; q < R2; q++) Bat(3, h, R2 * sub + q) = X[q];
        }
    }
    __syncthreads();

    const int hj = js >= nj, kj = js - hj * nj, jp = 2 * kj + hj;
    const int my = jp > nj, oy = my ? 2 * nj - jp : jp;
    const int lp = z_bin(l0 + t, nl, a.zs), mz = lp > nl, oz = mz ? 2 * nl - lp : lp;
    const size_t sp = z_entries(nl, a.zs), sy = 3 * sp, sxo = (size_t)(nj + 1) * sy;
    const float4 *Ayz = a.aq + (size_t)oy * sy + z_order(oz, nl, a.zs);
#pragma unroll 1
    for (int pol = 0; pol < 2; pol++) {
        const double *E = a.einc + 6 * (rhs0 + pol);
        const float2 Ex = make_float2((float)E[0], (float)E[1]), Ey = make_float2((float)E[2], (float)E[3]),
                     Ez = make_float2((float)E[4], (float)E[5]);
        // a real incident field (every rotated x or y polarisation): u = G E with real
        // weights (fused multiply-adds on the components), then u psi -- 30 instead of 54
        // floating-point instructions per frequency
        const bool Ereal = Ex.y == 0.f && Ey.y == 0.f && Ez.y == 0.f;
        // ---- product with the Green tensor, inverse step A (transposed split); the branch
        // on a real field is taken once per polarisation, outside the unrolled loops
        auto product = [&](auto real_tag) {
            constexpr bool REAL = decltype(real_tag)::value;
            const int k1 = sub;
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                float2 X[3][R2];
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
                    const float2 ps = Bat(3, h, R2 * k1 + q);
                    if constexpr (REAL) {
                        const float ex = Ex.x, ey = Ey.x, ez = Ez.x;
                        auto dot = [&](float2 ga, float2 gb, float2 gc) {
                            return make_float2(fmaf(ga.x, ex, fmaf(gb.x, ey, gc.x * ez)),
                                               fmaf(ga.y, ex, fmaf(gb.y, ey, gc.y * ez)));
                        };
                        X[0][q] = cmul(dot(g0, g1, g2), ps);
                        X[1][q] = cmul(dot(g1, g3, g4), ps);
                        X[2][q] = cmul(dot(g2, g4, g5), ps);
                    } else {
                        const float2 vx = cmul(Ex, ps), vy = cmul(Ey, ps), vz = cmul(Ez, ps);
                        X[0][q] = cadd(cadd(cmul(g0, vx), cmul(g1, vy)), cmul(g2, vz));
                        X[1][q] = cadd(cadd(cmul(g1, vx), cmul(g3, vy)), cmul(g4, vz));
                        X[2][q] = cadd(cadd(cmul(g2, vx), cmul(g4, vy)), cmul(g5, vz));
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    dft_reg<R2, true>(X[c]);
#pragma unroll
                    for (int u = 0; u < R2; u++) {
                        const float2 y = u ? cmul(X[c][u], twid<true>(tw, k1 * u)) : X[c][u];
                        Bat(c, h, k1 + R1 * u) = y;
                    }
                }
            }
        };
        if (sub < R1) {
            if (Ereal) product(std::true_type{});
            else product(std::false_type{});
        }
        __syncthreads();
        // ---- inverse step B, combine the halves, store to right-hand side 2k + pol
        float2 *base = a.work + (size_t)(rhs0 + pol) * a.wstride + col;
        if constexpr (R1 == 2 * R2) {
            const int k1p = sub % R2, hb = sub / R2;
            constexpr int H = R1 / 2;
#pragma unroll 1
            for (int c = 0; c < 3; c++) {
                float2 e[H], o[H];
#pragma unroll
                for (int n = 0; n < H; n++) {
                    const float2 e0 = Bat(c, 0, R1 * k1p + n), e1 = Bat(c, 0, R1 * k1p + n + H);
                    const float2 o0 = Bat(c, 1, R1 * k1p + n), o1 = Bat(c, 1, R1 * k1p + n + H);
                    if (hb) {
                        const float2 wn = cconj(w16(n * (16 / R1)));
                        e[n] = n ? cmul(csub(e0, e1), wn) : csub(e0, e1);
                        o[n] = n ? cmul(csub(o0, o1), wn) : csub(o0, o1);
                    } else {
                        e[n] = cadd(e0, e1);
                        o[n] = cadd(o0, o1);
                    }
                }
                dft_reg<H, true>(e);
                dft_reg<H, true>(o);
#pragma unroll
                for (int m = 0; m < H; m++) {
                    const int i = k1p + R2 * (2 * m + hb);
                    base[c * cstr + i * plane] = cadd(e[m], cmulc(o[m], __ldg(&hw[i])));
                }
            }
        } else if (sub < R2) {
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
        __syncthreads();
    }
}

template <int NI>
constexpr int x_tile(int v)
{
    // variant 0: 32 columns per CTA (16 at NI = 128); variants 1, 2: a half, a quarter
    const int t0 = NI <= 64 ? 32 : 16;
    return t0 >> v;
}

// x variants 0..2: register loads with 32 / 16 / 8 columns (16 / 8 / 4 at edge 128);
// 3..5: the same tiles fed by bulk asynchronous copies; 6..8: register loads with the
// second line factorisation (Sx<N, 1>)
// 9..11: the same tiles as 0..2 fed by one TMA tensor tile per component
template <int V>
constexpr int x_load(int) { return (V >= 3 && V < 6) ? 1 : (V >= 9 ? 2 : 0); }

template <int NI, int V>
void launch_x_v(const MatvecArgs &a, cudaStream_t st)
{
    constexpr int TL = x_tile<NI>(V % 3), ALT = (V >= 6 && V < 9) ? 1 : 0, LD = x_load<V>(0);
    const int ncol = 2 * a.L.nl;
    const size_t smem = (size_t)6 * NI * TL * sizeof(float2);
    const dim3 grid = k2_rhs_fastest(NI) ? dim3(a.nrhs, ncol / TL, 2 * a.L.nj)
                                         : dim3(2 * a.L.nj, ncol / TL, a.nrhs);
    static const CUtensorMap none{};
    const CUtensorMap &map = LD == 2 ? static_cast<const CUtensorMap *>(a.tmaps)[V % 3] : none;
    k2f<NI, TL, LD, ALT><<<grid, Sx<NI, ALT>::RM * TL, smem, st>>>(a, map);
}

// the pair form of the x pass (step 0 of polarisation pairs), same column tiles
template <int NI, int V>
void launch_x_pair_v(const MatvecArgs &a, cudaStream_t st)
{
    constexpr int TL = x_tile<NI>(V);
    const int ncol = 2 * a.L.nl, np = a.nrhs / 2;
    const size_t smem = (size_t)8 * NI * TL * sizeof(float2);
    const dim3 grid = k2_rhs_fastest(NI) ? dim3(np, ncol / TL, 2 * a.L.nj) : dim3(2 * a.L.nj, ncol / TL, np);
    k2p<NI, TL><<<grid, Sx<NI, 0>::RM * TL, smem, st>>>(a);
}

template <int NI>
void launch_x(const MatvecArgs &a, cudaStream_t st)
{
    // the widest tile of the variant that the row holds
    int t = a.fx % 3;
    while (t < 2 && (x_tile<NI>(0) >> t) > 2 * a.L.nl) t++;
    if (a.inc && a.pair) {
        if (t == 2) launch_x_pair_v<NI, 2>(a, st);
        else if (t == 1) launch_x_pair_v<NI, 1>(a, st);
        else launch_x_pair_v<NI, 0>(a, st);
        return;
    }
    switch (a.fx - a.fx % 3 + t) {
    case 11: launch_x_v<NI, 11>(a, st); break;
    case 10: launch_x_v<NI, 10>(a, st); break;
    case 9: launch_x_v<NI, 9>(a, st); break;
    case 8: launch_x_v<NI, 8>(a, st); break;
    case 7: launch_x_v<NI, 7>(a, st); break;
    case 6: launch_x_v<NI, 6>(a, st); break;
    case 5: launch_x_v<NI, 5>(a, st); break;
    case 4: launch_x_v<NI, 4>(a, st); break;
    case 3: launch_x_v<NI, 3>(a, st); break;
    case 2: launch_x_v<NI, 2>(a, st); break;
    case 1: launch_x_v<NI, 1>(a, st); break;
    default: launch_x_v<NI, 0>(a, st); break;
    }
}

template <int NI, int V>
cudaError_t prep_x_v()
{
    constexpr int TL = x_tile<NI>(V % 3), ALT = (V >= 6 && V < 9) ? 1 : 0, LD = x_load<V>(0);
    cudaError_t e = cudaFuncSetAttribute(k2f<NI, TL, LD, ALT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(6 * NI * TL * sizeof(float2)));
    if (e == cudaSuccess && V < 3)
        e = cudaFuncSetAttribute(k2p<NI, TL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(8 * NI * TL * sizeof(float2)));
    return e;
}

template <int NI>
cudaError_t prep_x()
{
    cudaError_t e = prep_x_v<NI, 0>();
    if (e == cudaSuccess) e = prep_x_v<NI, 1>();
    if (e == cudaSuccess) e = prep_x_v<NI, 2>();
    if (e == cudaSuccess) e = prep_x_v<NI, 3>();
    if (e == cudaSuccess) e = prep_x_v<NI, 4>();
    if (e == cudaSuccess) e = prep_x_v<NI, 5>();
    if (e == cudaSuccess) e = prep_x_v<NI, 6>();
    if (e == cudaSuccess) e = prep_x_v<NI, 7>();
    if (e == cudaSuccess) e = prep_x_v<NI, 8>();
    if (e == cudaSuccess) e = prep_x_v<NI, 9>();
    if (e == cudaSuccess) e = prep_x_v<NI, 10>();
    return e == cudaSuccess ? prep_x_v<NI, 11>() : e;
}

}  // namespace

template <>
cudaError_t x_prepare<X_NI>() { return prep_x<X_NI>(); }

template <>
cudaError_t x_launch<X_NI>(const MatvecArgs &a, cudaStream_t st)
{
    launch_x<X_NI>(a, st);
    return cudaGetLastError();
}

}  // namespace ddagpu
