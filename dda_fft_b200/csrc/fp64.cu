// FP64 solve of one polarisation: the reference's DDA_FFT (dda_func.cpp:1075-1570) with every
// field, transform, product and scalar in double -- the reference's FP64 build
// (complex.hpp:10 with `typedef double real`) run on the GPU.  It is the oracle solve of the
// precision pattern: the error of a float solve (with or without FP64-residual refinement)
// is measured against it, on lattices where a CPU FP64 solve would take hours.
//
// The convolution runs as five passes over a work buffer [3][ni][2nj][2nl] (only the i < ni
// planes of the padded grid exist, as in the float passes), with the Green tensor's FP64
// octant [6][ni+1][nj+1][nl+1] (green.cu) unfolded by its parities:
//   Z  forward along l of every lattice row (c, i, j < nj)
//   Y  forward along j of tiles of spectral columns (c, i, kz)
//   X  forward along i, the symmetric 3x3 product, inverse along i (i < ni kept), per
//      tile of (ky, kz) columns with all 3 components
//   YI inverse along j (j < nj kept)
//   ZI inverse along l (l < nl kept) with the solver epilogue out = sv v - alpha_m conv
// Every transform is an n-point FFT: the even and odd bins of a zero-padded 2n-point line
// are DFT_n(x) and DFT_n(x W_2n^j), and of the inverse only the first n outputs are kept,
// IDFT_n(even) + W_2n^-j IDFT_n(odd).  An n-point line is two register DFTs (n = R1 R2)
// with one exchange through shared memory, its sizes compile-time constants.
//
// What bounds it: the passes move 1248 n^3 bytes at least (48 + 96, 96 + 192, 192 + 192,
// 192 + 96, 96 + 48), from L2 while the work buffer fits there, and do about 450 n^3
// double multiply-adds; the first form (iterative radix-2 stages over padded 2n-point lines
// in shared memory) moved every line through shared memory 2 log2(2n) times.
#include <cuda_runtime.h>

#include <cmath>
#include <complex>
#include <cstring>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "fp64.h"

namespace ddagpu {

namespace {

constexpr int kT = 256;      // threads per block of the field passes
constexpr int kF = 128;      // threads per block of the transform passes

__device__ __forceinline__ double2 dadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 dsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 dmul(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 dconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 dzero() { return make_double2(0.0, 0.0); }

// exp(-2 pi i m / 16), m = 0..7
__device__ __forceinline__ double2 w16d(int m)
{
    const double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173, h = 0.70710678118654752440;
    switch (m) {
    case 0: return make_double2(1.0, 0.0);
    case 1: return make_double2(c1, -s1);
    case 2: return make_double2(h, -h);
    case 3: return make_double2(s1, -c1);
    case 4: return make_double2(0.0, -1.0);
    case 5: return make_double2(-s1, -c1);
    case 6: return make_double2(-h, -h);
    default: return make_double2(-c1, -s1);
    }
}

// In-register DFT of R points (a power of two, <= 16), natural order in and out; INV
// conjugates the twiddles (the reference's inverse is conj(DFT(conj x)) with no 1/n,
// fft_func.cpp:556-653).
template <int R, bool INV>
__device__ __forceinline__ void dft_d(double2 (&v)[R])
{
    if (R == 1) return;
#pragma unroll
    for (int len = R; len >= 2; len >>= 1) {
#pragma unroll
        for (int s = 0; s < R; s += len) {
#pragma unroll
            for (int j = 0; j < len / 2; j++) {
                const double2 a = v[s + j], b = v[s + j + len / 2], d = dsub(a, b);
                v[s + j] = dadd(a, b);
                if (j == 0) {
                    v[s + j + len / 2] = d;
                } else if (4 * j == len) {
                    v[s + j + len / 2] = INV ? make_double2(-d.y, d.x) : make_double2(d.y, -d.x);
                } else {
                    double2 w = w16d(j * (16 / len));
                    if (INV) w.y = -w.y;
                    v[s + j + len / 2] = dmul(d, w);
                }
            }
        }
    }
    double2 t[R];
#pragma unroll
    for (int k = 0; k < R; k++) t[k] = v[bitrev_c(k, ilog2c<R>::v)];
#pragma unroll
    for (int k = 0; k < R; k++) v[k] = t[k];
}

// A line of N = R1 R2 points: step A is R2 register DFTs of R1 points (elements t2 + R2 r,
// then times W_N^(t2 k1)), step B is R1 DFTs of R2 points (over t2, outputs k1 + R1 k2).
// Between them element (k1, t2) sits at k1 (R2 + 1) + t2: the pad keeps the eight lanes of
// a 128-byte shared-memory phase on distinct banks when they differ in k1 (row passes).
template <int N>
struct Line {
    static constexpr int R1 = fft_split<N>::R1, R2 = fft_split<N>::R2, LEN = R1 * (R2 + 1);
    // rows per block of the Z passes, columns per block of the Y and X passes: the 2 R1 step-B
    // items of a line (both parity halves) over kF threads; a Y column tile is a 128-byte run
    static constexpr int ROWS = kF / (2 * R1), YC = 8, XC = kF / (2 * R1);
    static constexpr size_t XSMEM = (size_t)3 * 2 * N * XC * sizeof(double2);
    __device__ static int at(int k1, int t2) { return k1 * (R2 + 1) + t2; }
};

struct Mv64 {
    int ni, nj, nl;
    size_t N;
    const double2 *twi, *twj, *twl;   // exp(-2 pi i k / 2n), k < 2n, per axis
    const double2 *g;                 // [6][ni+1][nj+1][nl+1]
    double2 *work;                    // [3][ni][2nj][2nl]
    int conj;
};

struct Ep64 {
    int mode;                 // 0 raw convolution, 1 sv v - alpha_m conv on active cells
    double sv;
    const double2 *v;         // [3][N]
    const signed char *occ;   // [N]
    const int *mv;            // [nmat1]
    const double2 *alpha;     // [nmat1]
    int conj;
};

__device__ __forceinline__ size_t wrow(const Mv64 &a, int c, int i, int js)
{
    return (((size_t)c * a.ni + i) * (2 * a.nj) + js) * (2 * a.nl);
}

// Step A of one half h of a line whose R1 inputs of lane t2 are in v (overwritten).
template <int N, bool INV>
__device__ __forceinline__ void step_a(double2 (&v)[Line<N>::R1], int t2, const double2 *__restrict__ tw)
{
    dft_d<Line<N>::R1, INV>(v);
#pragma unroll
    for (int k1 = 1; k1 < Line<N>::R1; k1++) {
        double2 w = __ldg(&tw[2 * t2 * k1]);
        if (INV) w.y = -w.y;
        v[k1] = dmul(v[k1], w);
    }
}

// Z: rows (c, i, j0 ..) of the field, forward along l.  Items of a block are spread over its
// threads with the parity half fastest, so a warp's loads and stores are runs of the row.
template <int N>
__global__ void __launch_bounds__(kF) z_fwd(Mv64 a, const double2 *src)
{
    chain_enter();
    using S = Line<N>;
    constexpr int R1 = S::R1, R2 = S::R2, G = S::ROWS;
    __shared__ double2 sm[G * 2 * S::LEN];
    const int j0 = blockIdx.x * G, i = blockIdx.y, c = blockIdx.z;
    const int nr = a.nj - j0 < G ? a.nj - j0 : G;
    const double2 *s = src + (size_t)c * a.N + ((size_t)i * a.nj + j0) * N;
    for (int e = threadIdx.x; e < nr * 2 * R2; e += kF) {
        const int t2 = e % R2, h = (e / R2) % 2, t = e / (2 * R2);
        double2 v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++) {
            v[r] = s[t * N + t2 + R2 * r];
            if (h) v[r] = dmul(v[r], __ldg(&a.twl[t2 + R2 * r]));
        }
        step_a<N, false>(v, t2, a.twl);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) sm[(t * 2 + h) * S::LEN + S::at(k1, t2)] = v[k1];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nr * 2 * R1; e += kF) {
        const int h = e % 2, k1 = (e / 2) % R1, t = e / (2 * R1);
        double2 u[R2];
#pragma unroll
        for (int q = 0; q < R2; q++) u[q] = sm[(t * 2 + h) * S::LEN + S::at(k1, q)];
        dft_d<R2, false>(u);
        double2 *d = a.work + wrow(a, c, i, j0 + t);
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) d[2 * (k1 + R1 * k2) + h] = u[k2];
    }
}

// Y: spectral columns kz0 .. of plane (c, i), forward along j
template <int N>
__global__ void __launch_bounds__(kF) y_fwd(Mv64 a)
{
    chain_enter();
    using S = Line<N>;
    constexpr int R1 = S::R1, R2 = S::R2, TC = S::YC;
    __shared__ double2 sm[2][R1][R2][TC];
    const int t = threadIdx.x % TC, kz = blockIdx.x * TC + t, i = blockIdx.y, c = blockIdx.z;
    const bool ok = kz < 2 * a.nl;
    double2 *col = a.work + wrow(a, c, i, 0) + kz;
    const size_t rs = (size_t)2 * a.nl;
    // the inputs are read before any output row is written (the pass is in place)
    for (int e = threadIdx.x / TC; e < 2 * R2; e += kF / TC) {
        if (!ok) break;
        const int h = e % 2, t2 = e / 2;
        double2 v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++) {
            v[r] = col[(t2 + R2 * r) * rs];
            if (h) v[r] = dmul(v[r], __ldg(&a.twj[t2 + R2 * r]));
        }
        step_a<N, false>(v, t2, a.twj);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) sm[h][k1][t2][t] = v[k1];
    }
    __syncthreads();
    for (int e = threadIdx.x / TC; e < 2 * R1; e += kF / TC) {
        if (!ok) break;
        const int h = e % 2, k1 = e / 2;
        double2 u[R2];
#pragma unroll
        for (int q = 0; q < R2; q++) u[q] = sm[h][k1][q][t];
        dft_d<R2, false>(u);
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) col[(2 * (k1 + R1 * k2) + h) * rs] = u[k2];
    }
}

// YI: the same columns, inverse along j, j < N kept
template <int N>
__global__ void __launch_bounds__(kF) y_inv(Mv64 a)
{
    chain_enter();
    using S = Line<N>;
    constexpr int R1 = S::R1, R2 = S::R2, TC = S::YC;
    __shared__ double2 sm[2][R1][R2][TC];
    const int t = threadIdx.x % TC, kz = blockIdx.x * TC + t, i = blockIdx.y, c = blockIdx.z;
    const bool ok = kz < 2 * a.nl;
    double2 *col = a.work + wrow(a, c, i, 0) + kz;
    const size_t rs = (size_t)2 * a.nl;
    for (int e = threadIdx.x / TC; e < 2 * R2; e += kF / TC) {
        if (!ok) break;
        const int h = e % 2, t2 = e / 2;
        double2 v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++) v[r] = col[(2 * (t2 + R2 * r) + h) * rs];
        step_a<N, true>(v, t2, a.twj);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) sm[h][k1][t2][t] = v[k1];
    }
    __syncthreads();
    for (int e = threadIdx.x / TC; e < R1; e += kF / TC) {
        if (!ok) break;
        double2 u[R2], o[R2];
#pragma unroll
        for (int q = 0; q < R2; q++) {
            u[q] = sm[0][e][q][t];
            o[q] = sm[1][e][q][t];
        }
        dft_d<R2, true>(u);
        dft_d<R2, true>(o);
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) {
            const int j = e + R1 * k2;
            col[j * rs] = dadd(u[k2], dmul(o[k2], dconj(__ldg(&a.twj[j]))));
        }
    }
}

// X: columns (ky, kz0 ..), 3 components: forward along i, G product, inverse.  A thread of
// step B holds 3 x R2 frequencies, so the product and the first inverse step need no exchange.
template <int N>
__global__ void __launch_bounds__(kF) x_pass(Mv64 a)
{
    chain_enter();
    using S = Line<N>;
    constexpr int R1 = S::R1, R2 = S::R2, TC = S::XC;
    extern __shared__ double2 smd[];   // [3][2][R1][R2][TC]
    auto B = [&](int c, int h, int k1, int t2, int t) -> double2 & {
        return smd[((((c * 2 + h) * R1) + k1) * R2 + t2) * TC + t];
    };
    const int t = threadIdx.x % TC, g0 = threadIdx.x / TC, kz = blockIdx.x * TC + t, ky = blockIdx.y;
    const bool ok = kz < 2 * a.nl;
    double2 *col = a.work + wrow(a, 0, 0, ky) + kz;
    const size_t rs = (size_t)(2 * a.nj) * (2 * a.nl), cs = rs * N;
    for (int e = g0; e < 6 * R2; e += kF / TC) {
        if (!ok) break;
        const int h = e % 2, t2 = (e / 2) % R2, c = e / (2 * R2);
        double2 v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++) {
            v[r] = col[c * cs + (t2 + R2 * r) * rs];
            if (h) v[r] = dmul(v[r], __ldg(&a.twi[t2 + R2 * r]));
        }
        step_a<N, false>(v, t2, a.twi);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) B(c, h, k1, t2, t) = v[k1];
    }
    __syncthreads();
    if (ok) {
        const int h = g0 % 2, k1 = g0 / 2, nj = a.nj, nl = a.nl;
        const bool my = ky > nj, mz = kz > nl;
        const int oy = my ? 2 * nj - ky : ky, oz = mz ? 2 * nl - kz : kz;
        const size_t yz = (size_t)oy * (nl + 1) + oz, xs = (size_t)(nj + 1) * (nl + 1), per = (N + 1) * xs;
        double2 X[3][R2];
#pragma unroll
        for (int c = 0; c < 3; c++) {
#pragma unroll
            for (int q = 0; q < R2; q++) X[c][q] = B(c, h, k1, q, t);
            dft_d<R2, false>(X[c]);
        }
#pragma unroll
        for (int q = 0; q < R2; q++) {
            const int kx = 2 * (k1 + R1 * q) + h;
            const bool mx = kx > N;
            const double2 *G = a.g + (size_t)(mx ? 2 * N - kx : kx) * xs + yz;
            double2 g[6];
#pragma unroll
            for (int k = 0; k < 6; k++) g[k] = __ldg(&G[k * per]);
            if (mx ^ my) g[1] = make_double2(-g[1].x, -g[1].y);
            if (mx ^ mz) g[2] = make_double2(-g[2].x, -g[2].y);
            if (my ^ mz) g[4] = make_double2(-g[4].x, -g[4].y);
            if (a.conj)
#pragma unroll
                for (int k = 0; k < 6; k++) g[k] = dconj(g[k]);
            const double2 vx = X[0][q], vy = X[1][q], vz = X[2][q];
            X[0][q] = dadd(dadd(dmul(g[0], vx), dmul(g[1], vy)), dmul(g[2], vz));
            X[1][q] = dadd(dadd(dmul(g[1], vx), dmul(g[3], vy)), dmul(g[4], vz));
            X[2][q] = dadd(dadd(dmul(g[2], vx), dmul(g[4], vy)), dmul(g[5], vz));
        }
        // inverse, transposed split: R2 points over q, times W^-(k1 u); kept at (k1, u)
#pragma unroll
        for (int c = 0; c < 3; c++) {
            dft_d<R2, true>(X[c]);
#pragma unroll
            for (int u = 0; u < R2; u++)
                B(c, h, k1, u, t) = u ? dmul(X[c][u], dconj(__ldg(&a.twi[2 * k1 * u]))) : X[c][u];
        }
    }
    __syncthreads();
    // R1 points over k1 of both halves: outputs u + R2 k2
    for (int e = g0; e < 3 * R2; e += kF / TC) {
        if (!ok) break;
        const int u = e % R2, c = e / R2;
        double2 v[R1], w[R1];
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) {
            v[k1] = B(c, 0, k1, u, t);
            w[k1] = B(c, 1, k1, u, t);
        }
        dft_d<R1, true>(v);
        dft_d<R1, true>(w);
#pragma unroll
        for (int k2 = 0; k2 < R1; k2++) {
            const int i = u + R2 * k2;
            col[c * cs + i * rs] = dadd(v[k2], dmul(w[k2], dconj(__ldg(&a.twi[i]))));
        }
    }
}

// ZI: rows (c, i, j0 ..), inverse along l, l < N kept, epilogue
template <int N>
__global__ void __launch_bounds__(kF) z_inv(Mv64 a, Ep64 ep, double2 *out)
{
    chain_enter();
    using S = Line<N>;
    constexpr int R1 = S::R1, R2 = S::R2, G = S::ROWS;
    __shared__ double2 sm[G * 2 * S::LEN];
    const int j0 = blockIdx.x * G, i = blockIdx.y, c = blockIdx.z;
    const int nr = a.nj - j0 < G ? a.nj - j0 : G;
    for (int e = threadIdx.x; e < nr * 2 * R2; e += kF) {
        const int h = e % 2, t2 = (e / 2) % R2, t = e / (2 * R2);
        const double2 *s = a.work + wrow(a, c, i, j0 + t);
        double2 v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++) v[r] = s[2 * (t2 + R2 * r) + h];
        step_a<N, true>(v, t2, a.twl);
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) sm[(t * 2 + h) * S::LEN + S::at(k1, t2)] = v[k1];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nr * R1; e += kF) {
        const int k1 = e % R1, t = e / R1;
        double2 u[R2], o[R2];
#pragma unroll
        for (int q = 0; q < R2; q++) {
            u[q] = sm[(t * 2) * S::LEN + S::at(k1, q)];
            o[q] = sm[(t * 2 + 1) * S::LEN + S::at(k1, q)];
        }
        dft_d<R2, true>(u);
        dft_d<R2, true>(o);
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) {
            const int l = k1 + R1 * k2;
            const size_t q = ((size_t)i * a.nj + j0 + t) * N + l, oq = (size_t)c * a.N + q;
            const double2 conv = dadd(u[k2], dmul(o[k2], dconj(__ldg(&a.twl[l]))));
            double2 res = conv;
            if (ep.mode == 1) {
                const int m = ep.occ[q];
                if (!ep.mv[m]) {
                    res = dzero();
                } else {
                    double2 al = ep.alpha[m];
                    if (ep.conj) al = dconj(al);
                    const double2 sv = ep.sv != 0.0 ? make_double2(ep.v[oq].x * ep.sv, ep.v[oq].y * ep.sv) : dzero();
                    res = dsub(sv, dmul(al, conv));
                }
            }
            out[oq] = res;
        }
    }
}

inline unsigned nb(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

// f(std::integral_constant<int, n>) for a lattice edge n (a power of two, 2..128)
template <class F>
cudaError_t with_edge(int n, F &&f)
{
    switch (n) {
    case 2: return f(std::integral_constant<int, 2>{});
    case 4: return f(std::integral_constant<int, 4>{});
    case 8: return f(std::integral_constant<int, 8>{});
    case 16: return f(std::integral_constant<int, 16>{});
    case 32: return f(std::integral_constant<int, 32>{});
    case 64: return f(std::integral_constant<int, 64>{});
    case 128: return f(std::integral_constant<int, 128>{});
    }
    return cudaErrorInvalidValue;
}

// out = epilogue of G * src: the five passes
cudaError_t matvec64(const Mv64 &a, const Ep64 &ep, const double2 *src, double2 *out, cudaStream_t st)
{
    const int ni = a.ni, nj = a.nj, nl = a.nl;
    cudaError_t e = with_edge(nl, [&](auto n) {
        constexpr int N = decltype(n)::value;
        return launch_chained(true, z_fwd<N>, dim3(nb(nj, Line<N>::ROWS), ni, 3), kF, 0, st, 1, a, src);
    });
    if (e == cudaSuccess)
        e = with_edge(nj, [&](auto n) {
            constexpr int N = decltype(n)::value;
            return launch_chained(true, y_fwd<N>, dim3(nb(2 * nl, Line<N>::YC), ni, 3), kF, 0, st, 1, a);
        });
    if (e == cudaSuccess)
        e = with_edge(ni, [&](auto n) {
            constexpr int N = decltype(n)::value;
            if (cudaError_t r = raise_smem_limit((const void *)x_pass<N>, (int)Line<N>::XSMEM)) return r;
            return launch_chained(true, x_pass<N>, dim3(nb(2 * nl, Line<N>::XC), 2 * nj), kF, Line<N>::XSMEM, st, 1, a);
        });
    if (e == cudaSuccess)
        e = with_edge(nj, [&](auto n) {
            constexpr int N = decltype(n)::value;
            return launch_chained(true, y_inv<N>, dim3(nb(2 * nl, Line<N>::YC), ni, 3), kF, 0, st, 1, a);
        });
    if (e == cudaSuccess)
        e = with_edge(nl, [&](auto n) {
            constexpr int N = decltype(n)::value;
            return launch_chained(true, z_inv<N>, dim3(nb(nj, Line<N>::ROWS), ni, 3), kF, 0, st, 1, a, ep, out);
        });
    return e;
}

// ---------------------------------------------------------------- field operations
using F64 = Field64View;

__device__ __forceinline__ bool active(const F64 &f, size_t q) { return f.mv[f.occ[q]] != 0; }

// p = alpha_m exp(i k.(r - c)) E_inc on active cells, c = (n - 1) d0 / 2 (FirstApproximation,
// dda_func.cpp:654-689); with rhs: p = rhs on active cells
__global__ void first_approx64(F64 f, double d0, double k0, double k1, double k2, double2 e0,
                               double2 e1, double2 e2, const double2 *rhs, double2 *p)
{
    const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= f.N) return;
    const int l = (int)(q % f.nl), j = (int)((q / f.nl) % f.nj), i = (int)(q / ((size_t)f.nl * f.nj));
    double2 o[3] = {dzero(), dzero(), dzero()};
    if (active(f, q)) {
        if (rhs) {
            for (int c = 0; c < 3; c++) o[c] = rhs[c * f.N + q];
        } else {
            const double ph = k0 * (i * d0 - (f.ni - 1) * d0 / 2) + k1 * (j * d0 - (f.nj - 1) * d0 / 2) +
                              k2 * (l * d0 - (f.nl - 1) * d0 / 2);
            double s, co;
            sincos(ph, &s, &co);
            const double2 c1 = dmul(make_double2(co, s), f.alpha[f.occ[q]]);
            o[0] = dmul(c1, e0);
            o[1] = dmul(c1, e1);
            o[2] = dmul(c1, e2);
        }
    }
    for (int c = 0; c < 3; c++) p[c * f.N + q] = o[c];
}

// block sums of NV doubles per thread, added to acc[0 .. NV)
template <int NV>
__device__ void block_add(double (&v)[NV], double *acc)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    __shared__ double sh[NV][kT / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) sh[k][w] = v[k];
    __syncthreads();
    if (threadIdx.x < NV) {
        double t = 0.0;
        for (int u = 0; u < (int)(blockDim.x >> 5); u++) t += sh[threadIdx.x][u];
        atomicAdd(acc + threadIdx.x, t);
    }
}

// Block sums of Re sum a conj(b) (ldScalMulConj, dda_func.cpp:757-782) or, without b, of the sum
// over cells of |a| (ldError's numerator, 784-811), over active cells, added to acc in FP64.
__global__ void __launch_bounds__(kT) reduce64(F64 f, const double2 *a, const double2 *b, double *acc)
{
    double s[1] = {0.0};
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < f.N; q += (size_t)gridDim.x * blockDim.x) {
        if (!active(f, q)) continue;
        double t = 0.0;
        for (int c = 0; c < 3; c++) {
            const double2 x = a[c * f.N + q], y = b ? b[c * f.N + q] : x;
            t += x.x * y.x + x.y * y.y;
        }
        s[0] += b ? t : sqrt(t);
    }
    block_add<1>(s, acc);
}

// o = x + c1 y + c2 z on active cells; inactive cells: o = 0 when mask_zero, else unchanged
// (the reference's LinearComb forms, dda_func.cpp:813-974)
__global__ void lin3_64(F64 f, const double2 *x, double2 c1, const double2 *y, double2 c2,
                        const double2 *z, double2 *o, int mask_zero)
{
    const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= f.N) return;
    const bool act = active(f, q);
    for (int c = 0; c < 3; c++) {
        const size_t k = c * f.N + q;
        if (act) {
            double2 v = x[k];
            if (y) v = dadd(v, dmul(c1, y[k]));
            if (z) v = dadd(v, dmul(c2, z[k]));
            o[k] = v;
        } else if (mask_zero) {
            o[k] = dzero();
        }
    }
}

// simple iteration (dda_func.cpp:1471-1521): r = (p - alpha conv) - s, p -= tau r on active
// cells (w holds p - alpha conv there), both zero elsewhere
__global__ void simple64(F64 f, const double2 *w, const double2 *s, double2 *r, double2 *p, double tau)
{
    const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= f.N) return;
    const bool act = active(f, q);
    for (int c = 0; c < 3; c++) {
        const size_t k = c * f.N + q;
        if (act) {
            const double2 rr = dsub(w[k], s[k]);
            r[k] = rr;
            p[k] = dsub(p[k], make_double2(tau * rr.x, tau * rr.y));
        } else {
            r[k] = dzero();
            p[k] = dzero();
        }
    }
}

// far field of one direction per block row (FarField, dda_func.cpp:1576-1625) and CabsCext
// (1679-1727, centre n d0 / 2, cells skipped where alpha == 0), summed in FP64
__global__ void __launch_bounds__(kT) farfield64(F64 f, double d0, const double *ksc, const double2 *p,
                                                 double *esc)
{
    const double *k = ksc + 3 * blockIdx.y;
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < f.N; q += (size_t)gridDim.x * blockDim.x) {
        if (!active(f, q)) continue;
        const int l = (int)(q % f.nl), j = (int)((q / f.nl) % f.nj), i = (int)(q / ((size_t)f.nl * f.nj));
        const double ph = k[0] * (i * d0 - (f.ni - 1) * d0 / 2) + k[1] * (j * d0 - (f.nj - 1) * d0 / 2) +
                          k[2] * (l * d0 - (f.nl - 1) * d0 / 2);
        double s, co;
        sincos(ph, &s, &co);
        const double2 P[3] = {p[q], p[f.N + q], p[2 * f.N + q]};
        const double2 kp = make_double2(k[0] * P[0].x + k[1] * P[1].x + k[2] * P[2].x,
                                        k[0] * P[0].y + k[1] * P[1].y + k[2] * P[2].y);
        for (int c = 0; c < 3; c++) {
            const double2 v = make_double2(P[c].x - k[c] * kp.x, P[c].y - k[c] * kp.y);
            acc[2 * c] += co * v.x - s * v.y;
            acc[2 * c + 1] += co * v.y + s * v.x;
        }
    }
    for (int o = 16; o > 0; o >>= 1)
        for (int c = 0; c < 6; c++) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    __shared__ double sh[6][kT / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0)
        for (int c = 0; c < 6; c++) sh[c][w] = acc[c];
    __syncthreads();
    if (threadIdx.x < 6) {
        double t = 0.0;
        for (int u = 0; u < (int)(blockDim.x >> 5); u++) t += sh[threadIdx.x][u];
        atomicAdd(esc + 6 * blockIdx.y + threadIdx.x, t);
    }
}

__global__ void __launch_bounds__(kT) cabscext64(F64 f, int nmat1, double d0, double k0, double k1,
                                                 double k2, double2 e0, double2 e1, double2 e2,
                                                 const double2 *p, double *acc)
{
    double r1 = 0.0, r2 = 0.0;
    const double cx = f.ni * d0 / 2, cy = f.nj * d0 / 2, cz = f.nl * d0 / 2;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < f.N; q += (size_t)gridDim.x * blockDim.x) {
        const int m = f.occ[q];
        if (m < 0 || m >= nmat1) continue;
        const double2 a = f.alpha[m];
        if (a.x == 0.0 && a.y == 0.0) continue;
        const int l = (int)(q % f.nl), j = (int)((q / f.nl) % f.nj), i = (int)(q / ((size_t)f.nl * f.nj));
        const double ph = -(k0 * (i * d0 - cx) + k1 * (j * d0 - cy) + k2 * (l * d0 - cz));
        double s, co;
        sincos(ph, &s, &co);
        const double2 P[3] = {p[q], p[f.N + q], p[2 * f.N + q]};
        const double2 E[3] = {dconj(e0), dconj(e1), dconj(e2)};
        double2 pe = dzero();
        double pp = 0.0;
        for (int c = 0; c < 3; c++) {
            pe = dadd(pe, dmul(P[c], E[c]));
            pp += P[c].x * P[c].x + P[c].y * P[c].y;
        }
        r1 += dmul(make_double2(co, s), pe).y;
        // Im(pp / conj(a)) = pp Im(a) / |a|^2
        r2 += pp * a.y / (a.x * a.x + a.y * a.y) - (2.0 / 3.0) * pp;
    }
    for (int o = 16; o > 0; o >>= 1) {
        r1 += __shfl_xor_sync(0xffffffffu, r1, o);
        r2 += __shfl_xor_sync(0xffffffffu, r2, o);
    }
    __shared__ double sh[2][kT / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        sh[0][w] = r1;
        sh[1][w] = r2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t0 = 0.0, t1 = 0.0;
        for (int u = 0; u < (int)(blockDim.x >> 5); u++) {
            t0 += sh[0][u];
            t1 += sh[1][u];
        }
        atomicAdd(acc, t0);
        atomicAdd(acc + 1, t1);
    }
}

// ---------------------------------------------------------------- mixed precision (COCG)
__global__ void to_f32(const double2 *x, float2 *y, size_t n)
{
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
        y[q] = make_float2((float)x[q].x, (float)x[q].y);
}

__global__ void from_f32_masked(F64 f, const float2 *x, double2 *y)
{
    const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= f.N) return;
    const bool act = active(f, q);
    for (int c = 0; c < 3; c++) {
        const float2 v = x[c * f.N + q];
        y[c * f.N + q] = act ? make_double2(v.x, v.y) : dzero();
    }
}

// out = v - alpha_m conv - sub on active cells, 0 elsewhere, in FP64 from the float convolution;
// acc[0] += sum over cells of |out| (ldError's numerator)
__global__ void __launch_bounds__(kT) mixed_apply(F64 f, const double2 *v, const float2 *conv,
                                                  const double2 *sub, double2 *out, double *acc)
{
    double e[1] = {0.0};
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < f.N; q += (size_t)gridDim.x * blockDim.x) {
        const int m = f.occ[q];
        if (!f.mv[m]) {
            for (int c = 0; c < 3; c++) out[c * f.N + q] = dzero();
            continue;
        }
        const double2 al = f.alpha[m];
        double t = 0.0;
        for (int c = 0; c < 3; c++) {
            const size_t k = c * f.N + q;
            const float2 g = conv[k];
            const double2 o = dsub(dsub(v[k], dmul(al, make_double2(g.x, g.y))), sub[k]);
            out[k] = o;
            t += o.x * o.x + o.y * o.y;
        }
        e[0] += sqrt(t);
    }
    block_add<1>(e, acc);
}

// The Krylov scalars stay on the device: every reduction adds into a set of kSet doubles, the
// update kernels form their coefficients from the set, and the host reads one residual per
// iteration while the next iteration's matvec already runs.
constexpr int kSet = 12;
// CG set: <s,w> (0,1), <r,s> (2,3), <r,w> of the new r (4,5), sum |r| (6)
// BiCGStab set: rho (0,1), <g,h> (2,3), <w,r> (4,5), <w,w> (6,7), sum |r| (8)

__device__ __forceinline__ double2 set_at(const double *a, int k) { return make_double2(a[k], a[k + 1]); }
// a / b with b brought to [1, 4) by a power of two: unscaled, its square leaves the doubles' range for
// sums below 1e-154 or above 1e154 (a converged residual, right-hand sides in small or large
// units) while the quotient is an ordinary number.  The power is set bit by bit (subnormal sums
// end between 2^-51 and 2), as ilogb and scalbn took a microsecond of a step.  By zero or infinity
// part by part: infinite and zero coefficients, as a complex division gives them.
__device__ __forceinline__ double2 ddiv(double2 a, double2 b)
{
    const double m = fmax(fabs(b.x), fabs(b.y));
    if (!(m > 0.0) || isinf(m)) return make_double2(a.x / m, a.y / m);
    const int e = 2046 - (__double2hiint(m) >> 20);   // biased exponent of 1 / m to a power of two
    const double w = __hiloint2double((e > 1 ? e : 1) << 20, 0);
    const double2 c = make_double2(b.x * w, b.y * w);
    const double d = c.x * c.x + c.y * c.y;
    return make_double2((a.x * c.x + a.y * c.y) / d * w, (a.y * c.x - a.x * c.y) / d * w);
}
__device__ __forceinline__ void bil_add(double &re, double &im, double2 a, double2 b)
{
    re += a.x * b.x - a.y * b.y;
    im += a.x * b.y + a.y * b.x;
}

// acc[0..1] += sum a b (bilinear), acc[2..3] += sum c d, over active cells; CG: (s, w), (r, s)
__global__ void __launch_bounds__(kT) two_dots(F64 f, const double2 *a, const double2 *b, const double2 *c,
                                               const double2 *d, double *acc)
{
    chain_enter();
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < f.N; q += (size_t)gridDim.x * blockDim.x) {
        if (!active(f, q)) continue;
        for (int k = 0; k < 3; k++) {
            const size_t o = k * f.N + q;
            bil_add(v[0], v[1], a[o], b[o]);
            if (c) bil_add(v[2], v[3], c[o], d[o]);
        }
    }
    block_add<4>(v, acc);
}

// w = s - alpha_m conv on active cells (0 elsewhere) and the dots of CG in the same pass
__global__ void __launch_bounds__(kT) mixed_apply_dots(F64 f, const double2 *s, const float2 *conv, const double2 *r,
                                                       double2 *w, double *acc)
{
    chain_enter();
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < f.N; q += (size_t)gridDim.x * blockDim.x) {
        const int m = f.occ[q];
        if (!f.mv[m]) {
            for (int k = 0; k < 3; k++) w[k * f.N + q] = dzero();
            continue;
        }
        const double2 al = f.alpha[m];
        for (int k = 0; k < 3; k++) {
            const size_t o = k * f.N + q;
            const float2 g = conv[o];
            const double2 sv = s[o], wv = dsub(sv, dmul(al, make_double2(g.x, g.y)));
            w[o] = wv;
            bil_add(v[0], v[1], sv, wv);
            bil_add(v[2], v[3], r[o], sv);
        }
    }
    block_add<4>(v, acc);
}

// a = <r,s> / <s,w>: x = x0 - a s (x0 may be x); r -= a w on active cells; set[4..5] += sum r w, set[6] += sum |r|
__global__ void __launch_bounds__(kT) cg_update(F64 f, const double2 *x0, double2 *x, double2 *r, const double2 *s,
                                                const double2 *w, double *set)
{
    chain_enter();
    const double2 a = ddiv(set_at(set, 2), set_at(set, 0));
    double v[3] = {0.0, 0.0, 0.0};
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < f.N; q += (size_t)gridDim.x * blockDim.x) {
        if (!active(f, q)) continue;
        double t = 0.0;
        for (int c = 0; c < 3; c++) {
            const size_t k = c * f.N + q;
            const double2 sv = s[k], wv = w[k];
            x[k] = dsub(x0[k], dmul(a, sv));
            const double2 rv = dsub(r[k], dmul(a, wv));
            r[k] = rv;
            bil_add(v[0], v[1], rv, wv);
            t += rv.x * rv.x + rv.y * rv.y;
        }
        v[2] += sqrt(t);
    }
    block_add<3>(v, set + 4);
}

// b = <r,w> / <s,w>: s = r - b s on active cells (inactive cells keep their zeros); s32 (may
// be null) = float(s).  Posts the step's residual sum to the host and clears the next set: a
// copy and a clearing operation of their own between the kernels of a step cost 10 us
__global__ void cg_dir(F64 f, const double *set, double *next, double *post, const double2 *r, double2 *s, float2 *s32)
{
    chain_enter();
    const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q < kSet) next[q] = 0.0;
    if (q == 0) *post = set[6];
    if (q >= f.N) return;
    const double2 b = ddiv(set_at(set, 4), set_at(set, 0));
    const bool act = active(f, q);
    for (int c = 0; c < 3; c++) {
        const size_t k = c * f.N + q;
        double2 v = s[k];
        if (act) v = dsub(r[k], dmul(b, v));
        s[k] = v;
        if (s32) s32[k] = make_float2((float)v.x, (float)v.y);
    }
}

// BiCGStab (dda_func.cpp:1423-1469): la = rho / <g,h>, lw = <w,r> / <w,w> of a set
// s = r + lb s - lb lw h, lb = (rho la1) / (rho1 lw1), from the new rho and the last set;
// posts the last step's residual sum to the host (post may be null)
__global__ void bi_dir(F64 f, const double *last, const double *cur, double *post, const double2 *r, const double2 *h,
                       double2 *s)
{
    chain_enter();
    const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (post && q == 0) *post = last[8];
    if (q >= f.N) return;
    const double2 rho1 = set_at(last, 0), la = ddiv(rho1, set_at(last, 2)), lw = ddiv(set_at(last, 4), set_at(last, 6));
    const double2 lb = ddiv(dmul(set_at(cur, 0), la), dmul(rho1, lw)), c2 = dmul(lb, lw);
    const bool act = active(f, q);
    for (int c = 0; c < 3; c++) {
        const size_t k = c * f.N + q;
        s[k] = act ? dsub(dadd(r[k], dmul(lb, s[k])), dmul(c2, h[k])) : dzero();
    }
}

// r -= la h on active cells; clears the next set
__global__ void bi_r(F64 f, const double *set, double *next, const double2 *h, double2 *r)
{
    chain_enter();
    const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q < kSet) next[q] = 0.0;
    if (q >= f.N || !active(f, q)) return;
    const double2 la = ddiv(set_at(set, 0), set_at(set, 2));
    for (int c = 0; c < 3; c++) {
        const size_t k = c * f.N + q;
        r[k] = dsub(r[k], dmul(la, h[k]));
    }
}

// p = p - la s - lw r (0 on inactive cells); r -= lw w; set[8] += sum |r|, next[0..1] += <r,g>
__global__ void __launch_bounds__(kT) bi_update(F64 f, double *set, double *next, double2 *p, double2 *r,
                                                const double2 *s, const double2 *w, const double2 *g)
{
    chain_enter();
    const double2 la = ddiv(set_at(set, 0), set_at(set, 2)), lw = ddiv(set_at(set, 4), set_at(set, 6));
    double e[1] = {0.0}, v[2] = {0.0, 0.0};
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < f.N; q += (size_t)gridDim.x * blockDim.x) {
        if (!active(f, q)) {
            for (int c = 0; c < 3; c++) p[c * f.N + q] = dzero();
            continue;
        }
        double t = 0.0;
        for (int c = 0; c < 3; c++) {
            const size_t k = c * f.N + q;
            const double2 rv = r[k], rn = dsub(rv, dmul(lw, w[k]));
            p[k] = dsub(dsub(p[k], dmul(la, s[k])), dmul(lw, rv));
            r[k] = rn;
            bil_add(v[0], v[1], rn, g[k]);
            t += rn.x * rn.x + rn.y * rn.y;
        }
        e[0] += sqrt(t);
    }
    block_add<1>(e, set + 8);
    block_add<2>(v, next);
}

// the reference's cvector layout [N][3] <-> structure of arrays [3][N]
template <class T>
__global__ void aos_soa(const T *in, T *out, size_t N, int to_soa)
{
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < 3 * N; e += (size_t)gridDim.x * blockDim.x) {
        const size_t q = e / 3, c = e - 3 * q;
        if (to_soa) out[c * N + q] = in[e];
        else out[e] = in[c * N + q];
    }
}

}  // namespace

// ------------------------------------------------------------------ host side

template <class T>
static cudaError_t layout(const T *in, T *out, size_t N, int to_soa, cudaStream_t st)
{
    aos_soa<T><<<4 * 148, kT, 0, st>>>(in, out, N, to_soa);
    return cudaGetLastError();
}
cudaError_t field_to_soa(const float2 *aos, float2 *soa, size_t N, cudaStream_t st) { return layout(aos, soa, N, 1, st); }
cudaError_t field_to_aos(const float2 *soa, float2 *aos, size_t N, cudaStream_t st) { return layout(soa, aos, N, 0, st); }

// Pinned slot and event of a residual on its way to the host, and the sets of scalars.
cudaError_t KrylovScalars::ensure()
{
    cudaError_t e = cudaSuccess;
    if (!acc) e = cudaMalloc((void **)&acc, 3 * kSet * sizeof(double));
    if (e == cudaSuccess && !pin) e = cudaHostAlloc((void **)&pin, kSet * sizeof(double), cudaHostAllocDefault);
    if (e == cudaSuccess && !ready) e = cudaEventCreateWithFlags(&ready, cudaEventDisableTiming);
    return e;
}

void KrylovScalars::release()
{
    if (acc) cudaFree(acc);
    if (pin) cudaFreeHost(pin);
    if (ready) cudaEventDestroy(ready);
    acc = pin = nullptr;
    ready = nullptr;
}

double *KrylovScalars::set(int k) const { return acc + k * kSet; }

cudaError_t KrylovScalars::zero(int k, cudaStream_t st) const
{
    return cudaMemsetAsync(set(k), 0, kSet * sizeof(double), st);
}

cudaError_t KrylovScalars::send(const double *from, cudaStream_t st) const
{
    const cudaError_t e = cudaMemcpyAsync(pin, from, sizeof(double), cudaMemcpyDeviceToHost, st);
    return e == cudaSuccess ? sent(st) : e;
}

cudaError_t KrylovScalars::sent(cudaStream_t st) const { return cudaEventRecord(ready, st); }

cudaError_t KrylovScalars::wait(double &v) const
{
    const cudaError_t e = cudaEventSynchronize(ready);
    v = *pin;
    return e;
}

Fp64Buffers::~Fp64Buffers() { release(); }

void Fp64Buffers::release()
{
    void *ptrs[] = {g, tw, work, p, pmin, r, s, gg, h, w, b, alpha};
    for (void *q : ptrs)
        if (q) cudaFree(q);
    g = tw = work = p = pmin = r = s = gg = h = w = b = alpha = nullptr;
    scal.release();
    ni = nj = nl = 0;
}

cudaError_t Fp64Buffers::ensure(int ni_, int nj_, int nl_, double kd_, cudaStream_t st)
{
    if (g && ni == ni_ && nj == nj_ && nl == nl_ && kd == kd_) return cudaSuccess;
    release();
    const size_t N = (size_t)ni_ * nj_ * nl_, n3 = 3 * N;
    const size_t oct = (size_t)6 * (ni_ + 1) * (nj_ + 1) * (nl_ + 1);
    const size_t wst = (size_t)3 * ni_ * (2 * nj_) * (2 * nl_);
    cudaError_t e = cudaSuccess;
    auto A = [&](double2 **q, size_t n) {
        if (e == cudaSuccess) e = cudaMalloc((void **)q, n * sizeof(double2));
    };
    A(&g, oct);
    A(&tw, (size_t)2 * (ni_ + nj_ + nl_));
    A(&work, wst);
    A(&p, n3);
    A(&pmin, n3);
    A(&r, n3);
    A(&s, n3);
    A(&gg, n3);
    A(&h, n3);
    A(&w, n3);
    A(&b, n3);
    A(&alpha, 256);
    if (e == cudaSuccess) e = scal.ensure();
    if (e != cudaSuccess) {
        release();
        return e;
    }
    ni = ni_;
    nj = nj_;
    nl = nl_;
    kd = kd_;
    // twiddles exp(-2 pi i k / 2n), k < 2n, per axis, in FP64
    std::vector<double2> t((size_t)2 * (ni + nj + nl));
    const double pi = 3.14159265358979323846264338327950288;
    const int ns[3] = {ni, nj, nl};
    size_t o = 0;
    for (int ax = 0; ax < 3; ax++)
        for (int k = 0; k < 2 * ns[ax]; k++, o++)
            t[o] = make_double2(std::cos(-pi * k / ns[ax]), std::sin(-pi * k / ns[ax]));
    if ((e = cudaMemcpyAsync(tw, t.data(), t.size() * sizeof(double2), cudaMemcpyHostToDevice, st)) ||
        (e = green_build_octant64(ni, nj, nl, kd, g, st)) || (e = cudaStreamSynchronize(st))) {
        release();
        return e;
    }
    return cudaSuccess;
}

namespace {

struct Fp64Run {
    Fp64Buffers &B;
    cudaStream_t st;
    F64 f;
    Mv64 m;
    int nact;
    long long *launches;
    int matvecs = 0;

    // out = sv v - alpha_m conv(src) on active cells (0 elsewhere); conj: the conjugate
    // operator with conj(alpha) (Convolution_conj)
    cudaError_t matvec(const double2 *src, double2 *out, double sv, const double2 *v, int conj)
    {
        Mv64 a = m;
        a.conj = conj;
        Ep64 ep{1, sv, v, f.occ, f.mv, f.alpha, conj};
        *launches += 5;
        matvecs++;
        return matvec64(a, ep, src, out, st);
    }

    cudaError_t reduce(const double2 *a, const double2 *b, double &x)
    {
        cudaError_t e = cudaMemsetAsync(B.scal.acc, 0, sizeof(double), st);
        if (e) return e;
        reduce64<<<4 * 148, kT, 0, st>>>(f, a, b, B.scal.acc);
        *launches += 1;
        if ((e = cudaMemcpyAsync(&x, B.scal.acc, sizeof(double), cudaMemcpyDeviceToHost, st))) return e;
        return cudaStreamSynchronize(st);
    }
    cudaError_t herm(const double2 *a, const double2 *b, double &x) { return reduce(a, b, x); }
    cudaError_t err(const double2 *r, double &x)
    {
        const cudaError_t e = reduce(r, nullptr, x);
        x /= nact;
        return e;
    }
    cudaError_t lin3(const double2 *x, std::complex<double> c1, const double2 *y, std::complex<double> c2,
                     const double2 *z, double2 *o, int mask_zero)
    {
        lin3_64<<<nb(f.N, kT), kT, 0, st>>>(f, x, make_double2(c1.real(), c1.imag()), y,
                                             make_double2(c2.real(), c2.imag()), z, o, mask_zero);
        *launches += 1;
        return cudaGetLastError();
    }
    cudaError_t dots(const double2 *a, const double2 *b, const double2 *c, const double2 *d, double *acc)
    {
        *launches += 1;
        return launch_chained(true, two_dots, 4 * 148, kT, 0, st, 1, f, a, b, c, d, acc);
    }
    // the rest of a BiCGStab step after h = A s: set cur holds its rho, next (cleared on the way)
    // the next step's; p, r updated, the residual sum in set cur
    cudaError_t bicg_step(double2 *p, double2 *r, const double2 *s, const double2 *g, const double2 *h, double2 *w,
                          int cur, int next)
    {
        const KrylovScalars &K = B.scal;
        cudaError_t e = dots(g, h, nullptr, nullptr, K.set(cur) + 2);
        if (e) return e;
        if ((e = launch_chained(true, bi_r, nb(f.N, kT), kT, 0, st, 1, f, K.set(cur), K.set(next), h, r))) return e;
        if ((e = matvec(r, w, 1.0, r, 0))) return e;
        if ((e = dots(w, r, w, w, K.set(cur) + 4))) return e;
        *launches += 2;
        return launch_chained(true, bi_update, 4 * 148, kT, 0, st, 1, f, K.set(cur), K.set(next), p, r, s, w, g);
    }
    // a BiCGStab step's direction; post: the last step's residual sum goes to the host
    cudaError_t bicg_dir(const double2 *r, const double2 *h, double2 *s, int last, int cur, bool post)
    {
        const KrylovScalars &K = B.scal;
        *launches += 1;
        const cudaError_t e = launch_chained(true, bi_dir, nb(f.N, kT), kT, 0, st, 1, f, K.set(last), K.set(cur),
                                             post ? K.pin : nullptr, r, h, s);
        return e == cudaSuccess && post ? K.sent(st) : e;
    }
    cudaError_t copy(double2 *dst, const double2 *src)
    {
        return cudaMemcpyAsync(dst, src, 3 * f.N * sizeof(double2), cudaMemcpyDeviceToDevice, st);
    }
};

}  // namespace

#define CKE(x)                                                                               \
    do {                                                                                     \
        cudaError_t _e = (x);                                                                \
        if (_e != cudaSuccess) return _e;                                                    \
    } while (0)

cudaError_t solve_fp64(Fp64Buffers &B, const Fp64Problem &P, cudaStream_t st, Fp64Result &R,
                       long long *launches)
{
    const int ni = B.ni, nj = B.nj, nl = B.nl;
    const size_t N = (size_t)ni * nj * nl;
    CKE(cudaMemcpyAsync(B.alpha, P.alpha, P.nmat1 * sizeof(double2), cudaMemcpyHostToDevice, st));
    F64 f{N, ni, nj, nl, P.occ, P.mv, B.alpha};
    Mv64 m{ni, nj, nl, N, B.tw, B.tw + 2 * ni, B.tw + 2 * (ni + nj), B.g, B.work, 0};
    Fp64Run X{B, st, f, m, P.nact, launches};
    double2 *p = B.p, *pmin = B.pmin, *r = B.r, *s = B.s, *g = B.gg, *h = B.h, *w = B.w, *b = B.b;
    const size_t bytes = 3 * N * sizeof(double2);
    const int solver = P.solver;

    // right-hand side b (p_inc or the caller's), start p = x0 or b (dda_func.cpp:1102-1104)
    // (the caller's fields are [N][3]; the FFT work space is the staging buffer)
    if (P.rhs) {
        CKE(cudaMemcpyAsync(B.work, P.rhs, bytes, cudaMemcpyHostToDevice, st));
        CKE(layout(B.work, w, N, 1, st));
    }
    first_approx64<<<nb(N, kT), kT, 0, st>>>(f, P.d0, P.kinc[0], P.kinc[1], P.kinc[2],
                                             make_double2(P.einc[0], P.einc[1]),
                                             make_double2(P.einc[2], P.einc[3]),
                                             make_double2(P.einc[4], P.einc[5]), P.rhs ? w : nullptr, b);
    *launches += 1;
    if (P.x0) {
        CKE(cudaMemcpyAsync(B.work, P.x0, bytes, cudaMemcpyHostToDevice, st));
        CKE(layout(B.work, w, N, 1, st));
        CKE(X.lin3(w, 0.0, nullptr, 0.0, nullptr, p, 1));          // p = x0 on active cells
        CKE(X.matvec(p, w, 1.0, p, 0));                              // w = A p
        CKE(X.lin3(w, -1.0, b, 0.0, nullptr, r, 1));                // r = A p - b
    } else {
        CKE(X.copy(p, b));
        CKE(X.matvec(p, r, 0.0, nullptr, 0));                        // r = -alpha conv(p)
    }

    double RR1 = 0;
    if (solver == 0) CKE(X.copy(s, r));
    if (solver == 1) {
        CKE(X.herm(r, r, RR1));
        CKE(X.matvec(r, s, 1.0, r, 1));
    }
    if (solver == 2) {
        CKE(X.copy(g, r));
        CKE(X.copy(s, r));
        CKE(B.scal.zero(0, st));
        CKE(X.dots(r, g, nullptr, nullptr, B.scal.set(0)));
        CKE(X.matvec(s, h, 1.0, s, 0));
        CKE(X.bicg_step(p, r, s, g, h, w, 0, 1));
        CKE(B.scal.send(B.scal.set(0) + 8, st));
    }
    if (solver == 3) {
        CKE(X.copy(s, p));
        CKE(X.lin3(s, -1.0, r, 0.0, nullptr, p, 0));   // p = s - r (r vanishes off the target)
    }
    double err = 0;
    if (solver == 2) {
        CKE(B.scal.wait(err));
        err /= P.nact;
    } else {
        CKE(X.err(r, err));
    }
    double err_min = err;
    int step_min = 0, nt = 0;
    if (R.trace && nt < R.trace_len) R.trace[nt] = err;
    nt++;
    CKE(X.copy(pmin, p));
    const KrylovScalars &K = B.scal;
    if (solver == 0) CKE(K.zero(1, st));   // CG steps alternate between sets 0 and 1, from 1
    bool ahead = false;   // the next step's first matvec is already in the stream
    for (int o = 1; o <= P.max_step; o++) {   // dda_func.cpp:1301-1535
        if (err <= P.err_max) break;
        const bool best = err < err_min;
        if (best) {
            err_min = err;
            step_min = o - 1;
            // CG writes its next iterate to the other buffer; the two agree on inactive cells
            if (solver == 0) std::swap(p, pmin);
            else CKE(X.copy(pmin, p));
        }
        if (solver == 2) {
            if (!ahead) {
                CKE(X.bicg_dir(r, h, s, (o - 1) & 1, o & 1, false));
                CKE(X.matvec(s, h, 1.0, s, 0));
            }
            CKE(X.bicg_step(p, r, s, g, h, w, o & 1, (o + 1) & 1));
            // the next step's direction and first product run while the residual travels;
            // neither p nor r changes, so a step that turns out not to be needed costs nothing else
            if ((ahead = o < P.max_step)) {
                CKE(X.bicg_dir(r, h, s, o & 1, (o + 1) & 1, true));
                CKE(X.matvec(s, h, 1.0, s, 0));
            } else {
                CKE(K.send(K.set(o & 1) + 8, st));
            }
            CKE(K.wait(err));
        } else if (solver == 0) {
            if (!ahead) CKE(X.matvec(s, w, 1.0, s, 0));
            double *set = K.set(o & 1), *next = K.set((o + 1) & 1);
            CKE(X.dots(s, w, r, s, set));
            CKE(launch_chained(true, cg_update, 4 * 148, kT, 0, st, 1, f, best ? pmin : p, p, r, s, w, set));
            CKE(launch_chained(true, cg_dir, nb(N, kT), kT, 0, st, 1, f, set, next, K.pin, r, s, nullptr));
            CKE(K.sent(st));
            *launches += 2;
            if ((ahead = o < P.max_step)) CKE(X.matvec(s, w, 1.0, s, 0));
            CKE(K.wait(err));
        } else if (solver == 1) {
            CKE(X.matvec(s, w, 1.0, s, 0));
            double SS, RR;
            CKE(X.herm(s, s, SS));
            const double rA = -RR1 / SS;
            CKE(X.lin3(r, rA, w, 0.0, nullptr, r, 0));
            CKE(X.lin3(p, rA, s, 0.0, nullptr, p, 0));
            CKE(X.herm(r, r, RR));
            const double rB = RR / RR1;
            RR1 = RR;
            CKE(X.matvec(r, w, 1.0, r, 1));
            CKE(X.lin3(w, rB, s, 0.0, nullptr, s, 0));
        } else {
            CKE(X.matvec(p, w, 1.0, p, 0));
            simple64<<<nb(N, kT), kT, 0, st>>>(f, w, s, r, p, P.tau);
            *launches += 1;
        }
        if (solver == 0 || solver == 2) err /= P.nact;
        else CKE(X.err(r, err));
        if (R.trace && nt < R.trace_len) R.trace[nt] = err;
        nt++;
    }
    if (ahead) X.matvecs -= 1;   // of the step that was not taken
    R.steps = nt - 1;
    R.err = err;
    R.err_min = err < err_min ? err : err_min;
    R.step_min = -1;
    if (err > err_min) {   // best-iterate rollback, dda_func.cpp:1537-1548
        CKE(X.copy(p, pmin));
        R.step_min = step_min;
    }
    R.rolled_back = R.step_min >= 0;
    R.matvecs = X.matvecs;
    // CabsCext and the far field of the final dipoles
    CKE(cudaMemsetAsync(B.scal.acc, 0, 2 * sizeof(double), st));
    cabscext64<<<4 * 148, kT, 0, st>>>(f, P.nmat1, P.d0, P.kinc[0], P.kinc[1], P.kinc[2],
                                       make_double2(P.einc[0], P.einc[1]), make_double2(P.einc[2], P.einc[3]),
                                       make_double2(P.einc[4], P.einc[5]), p, B.scal.acc);
    *launches += 1;
    double cc[2];
    CKE(cudaMemcpyAsync(cc, B.scal.acc, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
    if (P.ndir > 0) {
        double *kd = nullptr, *ed = nullptr;
        CKE(cudaMallocAsync((void **)&kd, (size_t)P.ndir * 3 * sizeof(double), st));
        CKE(cudaMallocAsync((void **)&ed, (size_t)P.ndir * 6 * sizeof(double), st));
        CKE(cudaMemcpyAsync(kd, P.ksc, (size_t)P.ndir * 3 * sizeof(double), cudaMemcpyHostToDevice, st));
        CKE(cudaMemsetAsync(ed, 0, (size_t)P.ndir * 6 * sizeof(double), st));
        farfield64<<<dim3(2 * 148, P.ndir), kT, 0, st>>>(f, P.d0, kd, p, ed);
        *launches += 1;
        CKE(cudaMemcpyAsync(R.esc, ed, (size_t)P.ndir * 6 * sizeof(double), cudaMemcpyDeviceToHost, st));
        cudaFreeAsync(kd, st);
        cudaFreeAsync(ed, st);
    }
    CKE(cudaStreamSynchronize(st));
    double e2 = 0;
    for (int c = 0; c < 6; c++) e2 += P.einc[c] * P.einc[c];
    const double pi = 3.14159265358979323846264338327950288;
    R.cext = 4.0 * pi / e2 * cc[0];
    R.cabs = 4.0 * pi / e2 * cc[1];
    if (R.p) {
        CKE(layout(p, B.work, N, 0, st));
        CKE(cudaMemcpyAsync(R.p, B.work, bytes, cudaMemcpyDeviceToHost, st));
    }
    return cudaStreamSynchronize(st);
}

// ------------------------------------------------------------------ mixed precision (host)

MixedCgBuffers::~MixedCgBuffers() { release(); }

void MixedCgBuffers::release()
{
    void *ptrs[] = {x, r, s, w, b, best, alpha};
    for (void *q : ptrs)
        if (q) cudaFree(q);
    x = r = s = w = b = best = alpha = nullptr;
    scal.release();
    n3 = 0;
}

cudaError_t MixedCgBuffers::ensure(size_t n)
{
    if (x && n3 == n) return cudaSuccess;
    release();
    cudaError_t e = cudaSuccess;
    auto A = [&](double2 **q, size_t k) {
        if (e == cudaSuccess) e = cudaMalloc((void **)q, k * sizeof(double2));
    };
    A(&x, n);
    A(&r, n);
    A(&s, n);
    A(&w, n);
    A(&b, n);
    A(&best, n);
    A(&alpha, 256);
    if (e == cudaSuccess) e = scal.ensure();
    if (e != cudaSuccess) {
        release();
        return e;
    }
    n3 = n;
    return cudaSuccess;
}

cudaError_t f64_right_hand_side(const Field64View &f, double d0, const double *kinc,
                                const double *einc, const float2 *from_f32, double2 *out,
                                cudaStream_t st)
{
    if (from_f32) {
        from_f32_masked<<<nb(f.N, kT), kT, 0, st>>>(f, from_f32, out);
    } else {
        first_approx64<<<nb(f.N, kT), kT, 0, st>>>(f, d0, kinc[0], kinc[1], kinc[2],
                                                   make_double2(einc[0], einc[1]),
                                                   make_double2(einc[2], einc[3]),
                                                   make_double2(einc[4], einc[5]), nullptr, out);
    }
    return cudaGetLastError();
}

cudaError_t mixed_cg(MixedCgBuffers &B, const Field64View &f, const double2 *alpha_host, int nmat1,
                     int nact, double err_max, int max_outer, double inner_rel, int inner_max_step,
                     const ConvFn &conv, float2 *s32, float2 *conv32, float2 *x32, float2 *p32,
                     cudaStream_t st, MixedCgResult &R, long long *launches)
{
    const size_t N = f.N, n3 = 3 * N, bytes = n3 * sizeof(double2);
    const unsigned red = 4 * 148;
    const KrylovScalars &K = B.scal;
    // true residual r = x - alpha G*x - b and its discrepancy (ldError of it)
    auto true_residual = [&](double &err) -> cudaError_t {
        to_f32<<<red, kT, 0, st>>>(B.x, x32, n3);
        CKE(conv(x32, conv32));
        CKE(K.zero(2, st));
        mixed_apply<<<red, kT, 0, st>>>(f, B.x, conv32, B.b, B.r, K.set(2));
        *launches += 2;
        R.matvecs++;
        CKE(K.send(K.set(2), st));
        CKE(K.wait(err));
        err /= nact;
        return cudaSuccess;
    };
    CKE(cudaMemcpyAsync(B.alpha, alpha_host, nmat1 * sizeof(double2), cudaMemcpyHostToDevice, st));
    CKE(cudaMemcpyAsync(B.x, B.b, bytes, cudaMemcpyDeviceToDevice, st));   // x = b (p_inc)
    R = MixedCgResult();
    double err = 0;
    CKE(true_residual(err));
    R.history[0] = err;
    double err_best = err, anchor = err;
    CKE(cudaMemcpyAsync(B.best, B.x, bytes, cudaMemcpyDeviceToDevice, st));
    if (err > err_max) {
        CKE(K.zero(0, st));   // steps alternate between sets 0 and 1; set 2 is the true residual's
        CKE(cudaMemcpyAsync(B.s, B.r, bytes, cudaMemcpyDeviceToDevice, st));
        to_f32<<<red, kT, 0, st>>>(B.s, s32, n3);
        *launches += 1;
        int since = 0;
        const long long cap = (long long)(max_outer + 1) * inner_max_step;
        bool ahead = false;   // the next direction's convolution is already in the stream
        for (long long it = 0; it < cap; it++) {
            // w = A s (dda_func.cpp:1325-1357) and the dots of the step (1359-1371, without the
            // float casts); the residual travels to the host while the next convolution runs
            if (!ahead) CKE(conv(s32, conv32));
            double *set = K.set(it & 1), *next = K.set((it + 1) & 1);
            CKE(launch_chained(true, mixed_apply_dots, red, kT, 0, st, 1, f, B.s, conv32, B.r, B.w, set));
            R.matvecs++;
            CKE(launch_chained(true, cg_update, red, kT, 0, st, 1, f, B.x, B.x, B.r, B.s, B.w, set));
            CKE(launch_chained(true, cg_dir, nb(N, kT), kT, 0, st, 1, f, set, next, K.pin, B.r, B.s, s32));
            CKE(K.sent(st));
            *launches += 3;
            if ((ahead = it + 1 < cap)) CKE(conv(s32, conv32));
            double err_rec;
            CKE(K.wait(err_rec));
            err_rec /= nact;
            R.iterations++;
            since++;
            if (err_rec <= err_max || err_rec <= inner_rel * anchor || since >= inner_max_step) {
                ahead = false;
                CKE(true_residual(err));
                R.outer++;
                if (R.outer < 64) R.history[R.outer] = err;
                if (err < err_best) {
                    err_best = err;
                    CKE(cudaMemcpyAsync(B.best, B.x, bytes, cudaMemcpyDeviceToDevice, st));
                }
                if (err <= err_max || R.outer >= max_outer) break;
                // restart from the current solution: fresh direction s = r (true residual)
                CKE(cudaMemcpyAsync(B.s, B.r, bytes, cudaMemcpyDeviceToDevice, st));
                to_f32<<<red, kT, 0, st>>>(B.s, s32, n3);
                *launches += 1;
                anchor = err;
                since = 0;
            }
        }
    }
    if (err > err_best) CKE(cudaMemcpyAsync(B.x, B.best, bytes, cudaMemcpyDeviceToDevice, st));
    R.err = err < err_best ? err : err_best;
    to_f32<<<red, kT, 0, st>>>(B.x, p32, n3);
    *launches += 1;
    return cudaGetLastError();
}

}  // namespace ddagpu
