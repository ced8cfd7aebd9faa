// Forward and inverse y/z passes of the matvec for lattice edges 4..128, every size a
// compile-time constant (matvec_x.cu: the x pass between them).
//
// A plane (component, lattice plane i) of a field is NJ x NL; its zero-padded spectrum along
// z is kept as pairs: bins 2 kl and 2 kl + 1 of the 2 NL-point line are the two halves of one
// float4 (pair.cuh), so both go through every transform together, the field is read once and
// no second CTA has to combine the halves.  A plane of pairs is at most 64 KB of shared
// memory: where NJ x NL is larger, ZS = 2 or 4 CTAs take the bins kl = r (mod ZS) -- a line of
// ML = NL / ZS points each, after (forward) or before (inverse) one butterfly over the ZS
// parts of the row -- and the inverse pass sums the ranks' shares through distributed shared
// memory.  Work buffer: [rhs][c][i][js][zpos] float4, js = hy NJ + ky (bin 2 ky + hy),
// zpos = r ML + m (kl = ZS m + r); there a pair is two complex columns, bins 2 kl and 2 kl + 1.
//
// An n-point line is n = R1 R2 (line_split): R2 register DFTs of R1 points, twiddles, an exchange
// through shared memory and R1 DFTs of R2 points.  z lines (rows of the plane) belong to R1
// consecutive lanes; y lines (columns) to a group of 8 columns x R1 lanes, whose accesses are
// whole 128-byte lines (a line costs the L1 data path a cycle however little of it is used:
// with 2 or 4 columns per warp the passes took 20-30% longer) and whose barrier is its own.
//
// What bounds it: 24 n^3 bytes read and 96 n^3 written (forward), the reverse for the inverse
// pass, and the L1 data path (65-75% of its wavefronts); 2.5 M warp instructions of FP32 at 64^3
// are a third of that time.  64^3 x 24: forward 208 -> 153 us, inverse 290 -> 160 us against a CTA
// per z half with scalar arithmetic, whose halves met through a cluster.
// Compiled once per y edge (YZ_NJ).
#include <cooperative_groups.h>

#include "internal.h"
#include "pair.cuh"

namespace cg = cooperative_groups;

namespace ddagpu {

namespace {

template <int N>
struct Split {
    static constexpr int R1 = line_split<N>::R1, R2 = line_split<N>::R2;
    static_assert(R2 > 1 && (R1 == R2 || R1 == 2 * R2), "two-step lines only");
};

template <int NJ, int NL, int NT, int MB>
struct Yz {
    static constexpr int ZS = matvec_z_split(NJ, NL);
    static constexpr int ML = NL / ZS;                      // z line of one CTA
    using SZ = Split<ML>;
    using SY = Split<NJ>;
    static constexpr int RG = SZ::R1 / SZ::R2;              // rows a lane group starts together
    static constexpr int ROWS = NT / SZ::R1 * RG;           // rows per pass of the block
    // A warp loads whole rows (forward) where the R2 elements of a lane group are 32-byte runs of the
    // field, eight lines per warp access; with that, without the next rows' prefetch where it
    // spilled (ZS 4) and with at()'s row term k1p takes 321 instead of 398 us (128^3 x 4) and 70
    // instead of 74 (32 x 128 x 64 x 6).  (At 128 x 128 the incident-field forms spill still, 20 and 12
    // bytes a thread.)  Longer runs (ML 64) gain nothing from the extra hop.
    static constexpr bool WIDE = ZS > 1 && ML == 32;
    static constexpr int CW = 8;                            // columns of a lane group: 128-byte runs
    static constexpr int GT = CW * SY::R1;                  // its threads (1, 2 or 4 warps)
    static constexpr int GROUPS = NT / GT;
    static_assert(GROUPS >= 1 && (GT <= 32 || GROUPS <= 15), "one named barrier per group");
    static constexpr bool PAIRED = SY::R1 == 2 * SY::R2;    // half the lanes take each y half
    static constexpr size_t PLANE = (size_t)NJ * ML * sizeof(float4);
    // odd y half's exchange of a warp's columns
    static constexpr size_t SCRATCH = PAIRED ? (size_t)GROUPS * NJ * CW * sizeof(float4) : 0;
    static constexpr size_t SMEM = PLANE + SCRATCH;
    static constexpr int FIT = (int)(227 * 1024 / (SMEM + 1024));
    static constexpr int WANT = MB;
    static constexpr int MINB = FIT < WANT ? (FIT < 1 ? 1 : FIT) : WANT;

    // Position of bin p of row `row`: within an aligned run of eight pairs (128 bytes) the order is
    // permuted by p >> 3, as a row's lanes read runs of stride R2, and by the row where eight
    // lanes access R2 < 8 pairs each of consecutive rows.
    __device__ static int at(int row, int p)
    {
        constexpr int RR = SZ::R2 < 8 ? 8 / SZ::R2 : 1;
        return row * ML + (ML >= 8 ? p ^ (((p >> 3) ^ (row % RR * SZ::R2)) & 7) : p);
    }
    // barrier of one column group
    __device__ static void sync(int group)
    {
        if (GT <= 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(GT) : "memory");
    }
};

// One element's inputs x[b] (element l + ML b of the row) -> element l of the pair line of rank
// r: bins s = 2 r, 2 r + 1 (mod 2 ZS), v_s = W^(s l) sum_b W^(s ML b) x_b.
template <int NL, int ZS>
DDA_DEV P2 fold(const float2 (&x)[ZS], int r, int l, const float2 *__restrict__ fz)
{
    constexpr int ML = NL / ZS;
    float2 h0, h1;
    if constexpr (ZS == 1) {
        h0 = x[0];
        h1 = x[0];
    } else if constexpr (ZS == 2) {
        // W^ML = -i
        const float2 a = x[0], b = x[1];
        h0 = r ? csub(a, b) : cadd(a, b);
        h1 = r ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, a.y - b.x);
    } else {
        // W^ML = exp(-i pi / 4)
        const float2 s = cadd(x[0], x[2]), d = csub(x[0], x[2]);
        const float2 q = cadd(x[1], x[3]), n = csub(x[1], x[3]);
        const float sg = r & 2 ? -1.f : 1.f;
        if (r & 1) h0 = make_float2(fmaf(sg, n.y, d.x), fmaf(-sg, n.x, d.y));   // d - sg i n
        else h0 = make_float2(fmaf(sg, q.x, s.x), fmaf(sg, q.y, s.y));
        // odd bin s = 2 r + 1: x0 -+ i x2 + w (x1 -+' i x3) with w = exp(-i pi s / 4)
        const float sr = r & 1 ? -1.f : 1.f;   // (-1)^r: W^(2 s ML) = -i (-1)^r
        const float2 a = make_float2(fmaf(sr, x[2].y, x[0].x), fmaf(-sr, x[2].x, x[0].y));
        const float2 b = make_float2(fmaf(sr, x[3].y, x[1].x), fmaf(-sr, x[3].x, x[1].y));
        const float2 w = __ldg(&fz[(2 * r + 1) * NL + ML]);
        const float2 t = cmul(b, w);
        h1 = cadd(a, t);
    }
    if (ZS > 1 && r) h0 = cmul(h0, __ldg(&fz[2 * r * NL + l]));
    h1 = cmul(h1, __ldg(&fz[(2 * r + 1) * NL + l]));
    return ppack(h0, h1);
}

// ------------------------------------------------------------------------------ K1
// CTA (i, r; component; right-hand side): z forward of the plane's rows, then y forward of the
// CTA's columns for both y halves.  IM 1: the input is the incident field, computed here and
// stored (each rank stores its part of the rows); IM 2: incident field of a polarisation pair
// (MatvecArgs::pair) -- phi = alpha_m exp(i k.(r - c)) into component slot 0 of right-hand side
// 2k, and p = phi E_q of both polarisations stored.
template <int NJ, int NL, int NT, int MB, int IM>
__global__ void __launch_bounds__(NT, Yz<NJ, NL, NT, MB>::MINB) k1p(MatvecArgs a)
{
    using Y = Yz<NJ, NL, NT, MB>;
    constexpr int ZS = Y::ZS, ML = Y::ML;
    extern __shared__ float4 S[];
    const int r = ZS > 1 ? blockIdx.x % ZS : 0, i = blockIdx.x / ZS, c = blockIdx.y;
    const int rhs = IM == 2 ? 2 * (int)blockIdx.z : (int)blockIdx.z;
    chain_enter();
    if (a.rhs_active && !a.rhs_active[rhs]) return;
    const int ni = a.L.ni;
    // twiddles in the order the lanes read them: tz[k1 R2 + t2] = W_ML^(t2 k1), ty likewise for
    // the y lines, fz[s NL + l] = W_2NL^(s l); at a stride of k1 a warp's load took a wavefront
    // per lane
    const float2 *tz = a.L.tz, *fz = a.L.fz;

    // ---- z: rows
    {
        constexpr int R1 = Y::SZ::R1, R2 = Y::SZ::R2, RG = Y::RG;
        const int sub = threadIdx.x % R1, g = threadIdx.x / R1, ar = sub / R2, t2 = sub % R2;
        // what load number k of a pass fetches: element t2 + R2 k of the lane's row, or, WIDE, element
        // `lane` of row k of the warp's R1 rows (which it hands over through the plane)
        static_assert(!Y::WIDE || (32 / R1 * RG == R1 && NJ % Y::ROWS == 0), "a warp's rows of a pass");
        auto row_of = [&](int r0, int k) { return Y::WIDE ? r0 + (int)threadIdx.x / 32 * R1 + k : r0 + g * RG + ar; };
        auto elem = [&](int k) { return Y::WIDE ? (int)threadIdx.x % 32 : t2 + R2 * k; };
        const float2 *src = a.src + (size_t)rhs * a.fstride + ((size_t)c * ni + i) * (NJ * NL);
        // incident field: ((x phase * y phase) * z phase) * alpha_m * E_c, the products of the
        // separate pass in its order (FirstApproximation, dda_func.cpp:654-689)
        const Epilogue &ep = a.ep;
        const float2 *pt = IM ? a.inc_tab + (size_t)rhs * (NJ + NL + ni) : nullptr;
        const float2 tx = IM ? pt[NJ + NL + i] : czero();
        const double *E = IM ? a.einc + 6 * rhs : nullptr;
        float2 Ef = czero(), Ep[2][3];
        if (IM == 1) Ef = make_float2((float)E[2 * c], (float)E[2 * c + 1]);
        if (IM == 2) {
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int k = 0; k < 3; k++)
                    Ep[q][k] = make_float2((float)E[6 * q + 2 * k], (float)E[6 * q + 2 * k + 1]);
        }
        const signed char *ob = IM ? ep.occ + (size_t)rhs * ep.occ_stride + (size_t)i * NJ * NL : nullptr;
        const float2 *al = IM ? ep.alpha + (size_t)rhs * ep.nmat1 : nullptr;
        const bool rt = IM && ep.nmat1 <= 2;   // up to two materials from registers
        const bool mv0 = IM && ep.mv[0] != 0, mv1 = IM && ep.nmat1 > 1 && ep.mv[1] != 0;
        const float2 al0 = IM ? al[0] : czero(), al1 = IM && ep.nmat1 > 1 ? al[1] : czero();
        float2 *pout = IM ? a.inc_out + (size_t)rhs * a.fstride + ((size_t)c * ni + i) * (NJ * NL) : nullptr;
        auto load = [&](int r0, float2 (&x)[R1][ZS], int (&o)[R1][ZS]) {
            if (row_of(r0, 0) >= NJ) return;   // (a warp's rows are in the plane or all past it)
#pragma unroll
            for (int k = 0; k < R1; k++)
#pragma unroll
                for (int b = 0; b < ZS; b++) {
                    const int e = row_of(r0, k) * NL + elem(k) + ML * b;
                    if (IM) o[k][b] = ob[e];
                    else x[k][b] = src[e];
                }
        };
        float2 x[R1][ZS], xn[R1][ZS];
        int o[R1][ZS], on[R1][ZS];
        constexpr bool AHEAD = ZS < 4;   // (with four parts of a row both sets do not fit the registers)
        if (AHEAD) load(0, x, o);
#pragma unroll 1
        for (int r0 = 0; r0 < NJ; r0 += Y::ROWS) {
            const int row0 = r0 + g * RG, row = row0 + ar;
            const bool ok = row < NJ;
            if (!AHEAD) load(r0, x, o);
            // the next pass's row is loaded while this one is transformed
            if (AHEAD && r0 + Y::ROWS < NJ) load(r0 + Y::ROWS, xn, on);
            if (ok) {
                if constexpr (IM != 0) {
#pragma unroll
                    for (int k = 0; k < R1; k++) {
                        const int rk = row_of(r0, k);
                        const float2 txy = cmul(tx, pt[rk]);
#pragma unroll
                        for (int b = 0; b < ZS; b++) {
                            const int l = elem(k) + ML * b, m = o[k][b];
                            const bool act = rt ? ((m & 1) ? mv1 : mv0) : ep.mv[m] != 0;
                            float2 val = czero();
                            if (act) {
                                val = cmul(cmul(txy, pt[NJ + l]), rt ? ((m & 1) ? al1 : al0) : al[m]);
                                if (IM == 1) val = cmul(val, Ef);
                            }
                            if (b == r) {
                                const size_t q = (size_t)rk * NL + l;
                                if (IM == 1) {
                                    pout[q] = val;
                                } else {
#pragma unroll
                                    for (int p = 0; p < 2; p++)
#pragma unroll
                                        for (int d = 0; d < 3; d++)
                                            pout[p * a.fstride + (size_t)d * ni * (NJ * NL) + q] = cmul(val, Ep[p][d]);
                                }
                            }
                            x[k][b] = val;
                        }
                    }
                }
                P2 v[R1];
#pragma unroll
                for (int k = 0; k < R1; k++) v[k] = fold<NL, ZS>(x[k], r, elem(k), fz);
                if constexpr (Y::WIDE) {
#pragma unroll
                    for (int k = 0; k < R1; k++) S[Y::at(row_of(r0, k), elem(k))] = f4_of(v[k]);
                    __syncwarp();
#pragma unroll
                    for (int k = 0; k < R1; k++) v[k] = p_of(S[Y::at(row, t2 + R2 * k)]);
                }
                dftp<R1, false>(v);
#pragma unroll
                for (int k1 = 0; k1 < R1; k1++) {
                    if (k1) v[k1] = pmul(v[k1], __ldg(&tz[k1 * R2 + t2]));
                    S[Y::at(row, t2 + R2 * k1)] = f4_of(v[k1]);
                }
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < RG; q++) {
                const int rw = row0 + q;
                P2 u[R2];
                if (rw < NJ) {
#pragma unroll
                    for (int t = 0; t < R2; t++) u[t] = p_of(S[Y::at(rw, R2 * sub + t)]);
                    dftp<R2, false>(u);
                }
                __syncwarp();
                if (rw < NJ) {
#pragma unroll
                    for (int k2 = 0; k2 < R2; k2++) S[Y::at(rw, sub + R1 * k2)] = f4_of(u[k2]);
                }
            }
            if (AHEAD)
#pragma unroll
                for (int k = 0; k < R1; k++)
#pragma unroll
                    for (int b = 0; b < ZS; b++) {
                        x[k][b] = xn[k][b];
                        o[k][b] = on[k][b];
                    }
        }
    }
    __syncthreads();

    // ---- y: columns, both halves from the same registers
    {
        constexpr int R1 = Y::SY::R1, R2 = Y::SY::R2, CW = Y::CW;
        const int group = threadIdx.x / Y::GT, t = threadIdx.x % CW, sub = threadIdx.x % Y::GT / CW;
        const float2 *tw = a.L.ty, *hw = a.L.tw_j + NJ;
        float4 *dst = reinterpret_cast<float4 *>(a.work + (size_t)rhs * a.wstride) +
                      ((size_t)c * ni + i) * (2 * NJ) * NL + r * ML;
        float4 *X = S + NJ * ML + (size_t)group * NJ * CW;   // PAIRED
#pragma unroll 1
        for (int c0 = 0; c0 < ML; c0 += Y::GROUPS * CW) {   // uniform over the block
            const int col = c0 + group * CW + t;
            const bool ok = col < ML;
            if constexpr (Y::PAIRED) {
                const int hy = sub / R2, t2 = sub % R2;
                P2 v[R1];
                if (ok) {
#pragma unroll
                    for (int k = 0; k < R1; k++) {
                        v[k] = p_of(S[Y::at(t2 + R2 * k, col)]);
                        if (hy) v[k] = pmul(v[k], __ldg(&hw[t2 + R2 * k]));
                    }
                    dftp<R1, false>(v);
#pragma unroll
                    for (int k1 = 1; k1 < R1; k1++) v[k1] = pmul(v[k1], __ldg(&tw[k1 * R2 + t2]));
                }
                Y::sync(group);
                if (ok) {
#pragma unroll
                    for (int k1 = 0; k1 < R1; k1++) {
                        if (hy) X[(t2 + R2 * k1) * CW + t] = f4_of(v[k1]);
                        else S[Y::at(t2 + R2 * k1, col)] = f4_of(v[k1]);
                    }
                }
                Y::sync(group);
                if (ok) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        P2 u[R2];
#pragma unroll
                        for (int q = 0; q < R2; q++)
                            u[q] = p_of(h ? X[(R2 * sub + q) * CW + t] : S[Y::at(R2 * sub + q, col)]);
                        dftp<R2, false>(u);
#pragma unroll
                        for (int k2 = 0; k2 < R2; k2++)
                            dst[(size_t)(h * NJ + sub + R1 * k2) * NL + col] = columns_of(u[k2]);
                    }
                }
                Y::sync(group);
            } else {
                P2 v[R1];
                if (ok) {
#pragma unroll
                    for (int k = 0; k < R1; k++) v[k] = p_of(S[Y::at(sub + R2 * k, col)]);
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    P2 u[R1];
                    if (ok) {
#pragma unroll
                        for (int k = 0; k < R1; k++) u[k] = h ? pmul(v[k], __ldg(&hw[sub + R2 * k])) : v[k];
                        dftp<R1, false>(u);
#pragma unroll
                        for (int k1 = 1; k1 < R1; k1++) u[k1] = pmul(u[k1], __ldg(&tw[k1 * R2 + sub]));
                    }
                    Y::sync(group);   // the column's elements are read before they are replaced
                    if (ok) {
#pragma unroll
                        for (int k1 = 0; k1 < R1; k1++) S[Y::at(sub + R2 * k1, col)] = f4_of(u[k1]);
                    }
                    Y::sync(group);
                    if (ok) {
                        P2 y[R2];
#pragma unroll
                        for (int q = 0; q < R2; q++) y[q] = p_of(S[Y::at(R2 * sub + q, col)]);
                        dftp<R2, false>(y);
#pragma unroll
                        for (int k2 = 0; k2 < R2; k2++)
                            dst[(size_t)(h * NJ + sub + R1 * k2) * NL + col] = columns_of(y[k2]);
                    }
                }
                Y::sync(group);
            }
        }
    }
}

// ------------------------------------------------------------------------------ K3
// CTA (i, r; component; right-hand side): y inverse of the CTA's columns (both y halves), z
// inverse of the plane's rows, then out = conv, or the solver epilogue sv v - alpha_m conv.
template <int NJ, int NL, int NT, int MB>
__global__ void __launch_bounds__(NT, Yz<NJ, NL, NT, MB>::MINB) k3p(MatvecArgs a)
{
    using Y = Yz<NJ, NL, NT, MB>;
    constexpr int ZS = Y::ZS, ML = Y::ML;
    extern __shared__ float4 S[];
    const int r = ZS > 1 ? blockIdx.x % ZS : 0, i = blockIdx.x / ZS, c = blockIdx.y, rhs = blockIdx.z;
    chain_enter();
    if (a.rhs_active && !a.rhs_active[rhs]) return;   // uniform over a cluster
    const int ni = a.L.ni;
    // twiddles in the order the lanes read them: tz[k1 R2 + t2] = W_ML^(t2 k1), ty likewise for
    // the y lines, fz[s NL + l] = W_2NL^(s l); at a stride of k1 a warp's load took a wavefront
    // per lane
    const float2 *tz = a.L.tz, *fz = a.L.fz;

    // ---- y inverse: x[j] = IDFT(even)[j] + W^-j IDFT(odd)[j]
    {
        constexpr int R1 = Y::SY::R1, R2 = Y::SY::R2, CW = Y::CW;
        const int group = threadIdx.x / Y::GT, t = threadIdx.x % CW, sub = threadIdx.x % Y::GT / CW;
        const float2 *tw = a.L.ty, *hw = a.L.tw_j + NJ;
        const float4 *src = reinterpret_cast<const float4 *>(a.work + (size_t)rhs * a.wstride) +
                            ((size_t)c * ni + i) * (2 * NJ) * NL + r * ML;
        float4 *X = S + NJ * ML + (size_t)group * NJ * CW;   // PAIRED
#pragma unroll 1
        for (int c0 = 0; c0 < ML; c0 += Y::GROUPS * CW) {   // uniform over the block
            const int col = c0 + group * CW + t;
            const bool ok = col < ML;
            P2 y[R2];
            if constexpr (Y::PAIRED) {
                const int hy = sub / R2, t2 = sub % R2;
                if (ok) {
                    P2 v[R1];
#pragma unroll
                    for (int k = 0; k < R1; k++) v[k] = of_columns(src[(size_t)(hy * NJ + t2 + R2 * k) * NL + col]);
                    dftp<R1, true>(v);
#pragma unroll
                    for (int k1 = 0; k1 < R1; k1++) {
                        if (k1) v[k1] = pmulc(v[k1], __ldg(&tw[k1 * R2 + t2]));
                        if (hy) X[(t2 + R2 * k1) * CW + t] = f4_of(v[k1]);
                        else S[Y::at(t2 + R2 * k1, col)] = f4_of(v[k1]);
                    }
                }
                Y::sync(group);
                if (ok) {
                    P2 u[R2];
#pragma unroll
                    for (int q = 0; q < R2; q++) {
                        y[q] = p_of(S[Y::at(R2 * sub + q, col)]);
                        u[q] = p_of(X[(R2 * sub + q) * CW + t]);
                    }
                    dftp<R2, true>(y);
                    dftp<R2, true>(u);
#pragma unroll
                    for (int k2 = 0; k2 < R2; k2++) y[k2] = padd(y[k2], pmulc(u[k2], __ldg(&hw[sub + R1 * k2])));
                }
            } else {
                P2 v[2][R1];
                if (ok) {
                    // both halves' loads in flight before the first transform
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int k = 0; k < R1; k++) v[h][k] = of_columns(src[(size_t)(h * NJ + sub + R2 * k) * NL + col]);
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    if (ok) {
                        dftp<R1, true>(v[h]);
#pragma unroll
                        for (int k1 = 0; k1 < R1; k1++) {
                            if (k1) v[h][k1] = pmulc(v[h][k1], __ldg(&tw[k1 * R2 + sub]));
                            S[Y::at(sub + R2 * k1, col)] = f4_of(v[h][k1]);
                        }
                    }
                    Y::sync(group);
                    if (ok) {
                        P2 u[R2];
#pragma unroll
                        for (int q = 0; q < R2; q++) u[q] = p_of(S[Y::at(R2 * sub + q, col)]);
                        dftp<R2, true>(u);
#pragma unroll
                        for (int k2 = 0; k2 < R2; k2++)
                            y[k2] = h ? padd(y[k2], pmulc(u[k2], __ldg(&hw[sub + R1 * k2]))) : u[k2];
                    }
                    Y::sync(group);
                }
            }
            Y::sync(group);
            if (ok) {
#pragma unroll
                for (int k2 = 0; k2 < R2; k2++) S[Y::at(sub + R1 * k2, col)] = f4_of(y[k2]);
            }
            if (Y::PAIRED) Y::sync(group);
        }
    }
    __syncthreads();

    // ---- epilogue of one output cell
    const size_t N = a.L.N;
    const Epilogue &ep = a.ep;
    const size_t obase = (size_t)rhs * a.fstride + (size_t)c * N + (size_t)i * NJ * NL;
    const signed char *ob = ep.occ + (size_t)rhs * ep.occ_stride + (size_t)i * NJ * NL;
    const bool solver = ep.mode == 1, regtab = solver && ep.nmat1 <= 2, withv = solver && ep.sv != 0.f;
    bool act0 = false, act1 = false;
    float2 al0 = czero(), al1 = czero();
    if (regtab) {
        act0 = ep.mv[0] != 0;
        al0 = ep.alpha[(size_t)rhs * ep.nmat1];
        if (ep.nmat1 > 1) {
            act1 = ep.mv[1] != 0;
            al1 = ep.alpha[(size_t)rhs * ep.nmat1 + 1];
        }
        if (ep.conj) {
            al0 = cconj(al0);
            al1 = cconj(al1);
        }
    }
    auto emit = [&](int e, float2 conv, int m, float2 v) {
        float2 res = conv;
        if (solver) {
            const bool act = regtab ? ((m & 1) ? act1 : act0) : ep.mv[m] != 0;
            if (!act) {
                res = czero();
            } else {
                float2 al;
                if (regtab) {
                    al = (m & 1) ? al1 : al0;
                } else {
                    al = ep.alpha[(size_t)rhs * ep.nmat1 + m];
                    if (ep.conj) al = cconj(al);
                }
                res = csub(cscale(v, ep.sv), cmul(al, conv));
            }
        }
        a.out[obase + e] = res;
    };

    // ---- z inverse of the rows
    {
        constexpr int R1 = Y::SZ::R1, R2 = Y::SZ::R2, RG = Y::RG;
        const int sub = threadIdx.x % R1, g = threadIdx.x / R1, ar = sub / R2, t2 = sub % R2;
#pragma unroll 1
        for (int r0 = 0; r0 < NJ; r0 += Y::ROWS) {
            const int row0 = r0 + g * RG, row = row0 + ar;
            // the outputs' materials and v are loaded before the transform
            int m[RG][R2];
            float2 vv[RG][R2];
            if (ZS == 1 && solver) {
#pragma unroll
                for (int q = 0; q < RG; q++)
                    if (row0 + q < NJ) {
#pragma unroll
                        for (int k2 = 0; k2 < R2; k2++) {
                            const int e = (row0 + q) * NL + sub + R1 * k2;
                            m[q][k2] = ob[e];
                            vv[q][k2] = withv ? ep.v[obase + e] : czero();
                        }
                    }
            }
            P2 v[R1];
            if (row < NJ) {
#pragma unroll
                for (int k = 0; k < R1; k++) v[k] = p_of(S[Y::at(row, t2 + R2 * k)]);
                dftp<R1, true>(v);
            }
            __syncwarp();
            if (row < NJ) {
#pragma unroll
                for (int k1 = 0; k1 < R1; k1++) {
                    if (k1) v[k1] = pmulc(v[k1], __ldg(&tz[k1 * R2 + t2]));
                    S[Y::at(row, t2 + R2 * k1)] = f4_of(v[k1]);
                }
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < RG; q++) {
                const int rw = row0 + q;
                P2 u[R2];
                if (rw < NJ) {
#pragma unroll
                    for (int t = 0; t < R2; t++) u[t] = p_of(S[Y::at(rw, R2 * sub + t)]);
                    dftp<R2, true>(u);
                }
                if constexpr (ZS == 1) {
                    if (rw < NJ) {
#pragma unroll
                        for (int k2 = 0; k2 < R2; k2++) {
                            const int l = sub + R1 * k2;
                            emit(rw * NL + l, cadd(pfirst(u[k2]), cmulc(psecond(u[k2]), __ldg(&fz[NL + l]))), m[q][k2], vv[q][k2]);
                        }
                    }
                } else {
                    __syncwarp();
                    if (rw < NJ) {
#pragma unroll
                        for (int k2 = 0; k2 < R2; k2++) S[Y::at(rw, sub + R1 * k2)] = f4_of(u[k2]);
                    }
                }
            }
            if (ZS > 1) __syncwarp();
        }
    }
    if constexpr (ZS > 1) {
        // ---- the ranks' shares: rank r sums rows [r NJ / ZS, (r + 1) NJ / ZS).  Bin class
        // s = 2 rank + half of element l' contributes conj(W^(s (l' + ML b))) u_s to part b.
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        constexpr int HR = NJ / ZS, CELLS = HR * ML;
        for (int e = threadIdx.x; e < CELLS; e += NT) {
            const int row = r * HR + e / ML, lp = e % ML;
            int m[ZS];
            float2 vv[ZS];
            if (solver) {
#pragma unroll
                for (int b = 0; b < ZS; b++) {
                    const int o = row * NL + lp + ML * b;
                    m[b] = ob[o];
                    vv[b] = withv ? ep.v[obase + o] : czero();
                }
            }
            float2 t[2 * ZS];
#pragma unroll
            for (int k = 0; k < ZS; k++) {
                const float4 *R = cl.map_shared_rank(S, k);
                const P2 u = p_of(R[Y::at(row, lp)]);
                t[2 * k] = k ? cmulc(pfirst(u), __ldg(&fz[2 * k * NL + lp])) : pfirst(u);
                t[2 * k + 1] = cmulc(psecond(u), __ldg(&fz[(2 * k + 1) * NL + lp]));
            }
            dft_reg<2 * ZS, true>(t);   // the parts are its first ZS outputs
#pragma unroll
            for (int b = 0; b < ZS; b++) emit(row * NL + lp + ML * b, t[b], m[b], vv[b]);
        }
        cl.sync();   // no rank leaves while its plane is read
    }
}

// block sizes of the launch variants
constexpr int yz_threads(int v) { return v == 1 ? 128 : 256; }
constexpr int yz_blocks(int v) { return v == 1 ? 4 : 2; }   // per SM where shared memory allows

template <int NJ, int NL, int V>
cudaError_t launch_yz_v(const MatvecArgs &a, int fwd, cudaStream_t st)
{
    constexpr int NT = yz_threads(V), MB = yz_blocks(V);
    using Y = Yz<NJ, NL, NT, MB>;
    const unsigned gx = Y::ZS * a.L.ni;
    const dim3 g3(gx, 3, a.nrhs), g1(gx, 1, a.nrhs / 2);
    if (fwd && a.inc && a.pair) return launch_chained(a.chained, k1p<NJ, NL, NT, MB, 2>, g1, NT, Y::SMEM, st, 1, a);
    if (fwd && a.inc) return launch_chained(a.chained, k1p<NJ, NL, NT, MB, 1>, g3, NT, Y::SMEM, st, 1, a);
    if (fwd) return launch_chained(a.chained, k1p<NJ, NL, NT, MB, 0>, g3, NT, Y::SMEM, st, 1, a);
    return launch_chained(a.chained, k3p<NJ, NL, NT, MB>, g3, NT, Y::SMEM, st, Y::ZS, a);
}

template <int NJ, int NL, int V>
cudaError_t prep_yz_v(int form)
{
    constexpr int NT = yz_threads(V), MB = yz_blocks(V), B = (int)Yz<NJ, NL, NT, MB>::SMEM;
    const void *k1[3] = {(const void *)k1p<NJ, NL, NT, MB, 0>, (const void *)k1p<NJ, NL, NT, MB, 1>,
                         (const void *)k1p<NJ, NL, NT, MB, 2>};
    const cudaError_t e = raise_smem_limit(k1[form], B);
    return e == cudaSuccess ? raise_smem_limit((const void *)k3p<NJ, NL, NT, MB>, B) : e;
}

template <class F>
cudaError_t with_nl(int nl, F f)
{
    switch (nl) {
    case 4: return f(std::integral_constant<int, 4>{});
    case 8: return f(std::integral_constant<int, 8>{});
    case 16: return f(std::integral_constant<int, 16>{});
    case 32: return f(std::integral_constant<int, 32>{});
    case 64: return f(std::integral_constant<int, 64>{});
    case 128: return f(std::integral_constant<int, 128>{});
    }
    return cudaErrorInvalidValue;
}

}  // namespace

template <>
cudaError_t yz_prepare<YZ_NJ>(int nl, int fyz, int form)
{
    return with_nl(nl, [&](auto l) {
        constexpr int NL = decltype(l)::value;
        return fyz == 1 ? prep_yz_v<YZ_NJ, NL, 1>(form) : prep_yz_v<YZ_NJ, NL, 0>(form);
    });
}

template <>
cudaError_t yz_launch<YZ_NJ>(const MatvecArgs &a, int fwd, cudaStream_t st)
{
    return with_nl(a.L.nl, [&](auto l) {
        constexpr int NL = decltype(l)::value;
        return a.fyz == 1 ? launch_yz_v<YZ_NJ, NL, 1>(a, fwd, st) : launch_yz_v<YZ_NJ, NL, 0>(a, fwd, st);
    });
}

}  // namespace ddagpu
