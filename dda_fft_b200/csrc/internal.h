// Internal types shared by the kernels and the host driver of libddagpu.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace ddagpu {

// Maximum lattice edge per axis handled by the fused FFT passes (powers of two).
constexpr int kMaxEdge = 128;
constexpr int kMinEdge = 2;
constexpr int kMaxMaterials = 255;   // occupancy bytes index materials 0..255
constexpr int kAcc = 8;              // FP64 reduction slots per right-hand side

// Per right-hand-side solver scalars, resident on the device.  The reference keeps
// these in long double and casts each coefficient to float before use
// (dda_func.cpp:1219,1260,1319,1362,1368,1375,1381,1424,1464); here the full-precision
// values are FP64 and the applied coefficients are the float casts.
struct RhsState {
    double acc[kAcc];       // reduction accumulators, consumed and zeroed by scalar kernels
    double2 ldA, ldW, rho1, rho, den;  // complex scalars of CG / BiCGStab
    double RR1;             // AA*: <r, r>_H of the previous step
    float2 cA, cB, cW, c2;  // float coefficients currently applied
    float rA, rB;           // AA* real coefficients
    double err, err_min;    // mean residual norm (ldError) and best so far
    double err_max;         // stopping threshold (float value of Error_max)
    int step_min;           // step of the best iterate
    int active;             // 1 while iterating
    int need_copy;          // 1: copy p -> p_min at this step
    int restored;           // 1: final p was replaced by p_min
    int steps;              // last completed step
    int nact;               // active cells
};

// Geometry of one lattice and its device-resident tables.
struct Lat {
    int ni, nj, nl;
    size_t N;               // ni * nj * nl
    const float2 *tw_i, *tw_j, *tw_l;   // [W_n^k, k<n ; W_2n^j, j<n] per axis
    // sized y/z passes, in their lanes' order (n = R1 R2, matvec_yz.cu): ty[k1 R2 + t2] = W_nj^(t2 k1),
    // tz the same for the nl / zs points of a z line, fz[s nl + l] = W_2nl^(s l), s < 2 zs
    const float2 *ty, *tz, *fz;
};

// Epilogue of the inverse pass: out = sv * v - a_m * conv on active cells, 0 elsewhere;
// mode 0 writes conv unchanged (plain convolution).
struct Epilogue {
    int mode;               // 0 raw convolution, 1 masked solver form
    int conj;               // use conj(alpha)
    float sv;               // scale of v
    const float2 *v;        // field v, same layout as out (may be null if sv == 0)
    const signed char *occ; // [N] material per cell (per right-hand side if occ_stride)
    size_t occ_stride;      // bytes between the occupancies of consecutive right-hand sides
    const float2 *alpha;    // [nrhs][nmat1] polarisability per material
    const int *mv;          // [nmat1] active material flags
    int nmat1;              // materials including index 0
};

// Launch of a kernel that starts with chain_enter: its blocks may become resident while the
// previous kernel of the stream drains, which takes 1 to 2 us out of each step from kernel to
// kernel (products on 8 x 64 x 32 x 4 11.2 -> 9.6 us, 64^3 x 1 47 -> 43, 64^3 x 24 827 -> 820).
// chained false: a plain launch, as inside a recorded graph, whose kernels follow each other
// without the host.
template <class... P, class... A>
cudaError_t launch_chained(bool chained, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                           unsigned cluster, const A &...args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2]{};
    if (cluster > 1) {
        at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        at[cfg.numAttrs].val.clusterDim.x = cluster;
        at[cfg.numAttrs].val.clusterDim.y = at[cfg.numAttrs].val.clusterDim.z = 1;
        cfg.numAttrs++;
    }
    if (chained) {
        at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs++;
    }
    cfg.attrs = at;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, P(args)...);
    if (e != cudaSuccess) cudaGetLastError();   // reported here, not by whoever asks next
    return e;
}

struct MatvecArgs {
    Lat L;
    int nrhs;
    const float2 *src;      // [nrhs][3][N] input field
    size_t fstride;         // 3 N
    float2 *work;           // [nrhs][3][ni][2nj][2nl]
    size_t wstride;
    const float4 *ahat;     // octant Green tensor [ni+1][nj+1][3][z_entries], two components each (zorder.cuh)
    int zs;                 // z split of the sized passes (set by launch_matvec_fast)
    int chained;            // passes launched one into the other's end (set by launch_matvec_fast)
    int conj;               // use conj(Ahat)
    float2 *out;            // [nrhs][3][N]
    Epilogue ep;
    const int *rhs_active;  // [nrhs] or null
    int tile_x;             // columns per CTA of the x pass (generic kernels)
    int rows_g;             // rows per staging group of the y/z passes (generic kernels)
    int fast;               // 1: compile-time-sized kernels (matvec_yz.cu, matvec_x.cu)
    int fx, fyz;            // launch variants of the fast x pass (0..11) and y/z passes (0..2)
    int *err;               // device flag set by a kernel whose bounded wait gave up (or null)
    const void *tmaps;      // host CUtensorMap of the work buffer (TMA x variants), or null
    int wait_selftest;      // 1: the bulk-copy wait waits (briefly) for a phase that never completes
    // step 0 from the incident field (compile-time-sized passes only): the forward y/z pass
    // computes its input p = alpha_m exp(i k.(r - c)) E_inc on active cells (0 elsewhere)
    // from the occupancy and materials of ep instead of reading src, and writes it to inc_out
    int inc;
    // with inc: right-hand sides 2k, 2k+1 are the two polarisations of one orientation with
    // the same polarisabilities, so p_inc = phi(r) E_q with one scalar phi = alpha_m
    // exp(i k.(r - c)); the forward passes transform phi once per pair (into component slot
    // 0 of right-hand side 2k) and the x pass forms G * (phi E_q) for both polarisations
    int pair;
    const float2 *inc_tab;  // [nrhs][nj + nl + ni] phase tables (y, z, x)
    const double *einc;     // [nrhs][6] incident field
    float2 *inc_out;        // [nrhs][3][N]
};

// Dynamic shared memory limit of a kernel on the current device, raised to at least
// `bytes` and never lowered: the limit is a per-process property of the kernel, shared by
// every context, so a context on a smaller lattice must not shrink what a larger one set
// (matvec.cu).
cudaError_t raise_smem_limit(const void *kernel, int bytes);

// kernels (matvec.cu)
cudaError_t kernel_binary_version(int *version);   // of the loaded module, e.g. 100
cudaError_t launch_matvec(const MatvecArgs &a, cudaStream_t st);
size_t matvec_smem_yz(const Lat &L, int rows_g);
size_t matvec_smem_x(const Lat &L, int tile_x);
cudaError_t matvec_prepare(const Lat &L, int tile_x, int rows_g);

// compile-time-sized passes for edges 4..128 (matvec_fast.cu: dispatch; matvec_x.cu, matvec_yz.cu)
bool matvec_fast_supported(const Lat &L);
constexpr int kXVariants = 12;     // launch variants of the fast x pass (9..11: TMA tensor tiles)
constexpr int kYZVariants = 3;     // launch variants of the fast y/z passes
// Shared-memory limits of the passes that a variant launches for `form` (0 a field, 1 the incident
// field, 2 that of a polarisation pair), no others: asking for one loads the kernel.  The carveout
// stays the driver's choice (the largest one cost 15%: what the passes leave, L1 uses for the
// Green tensor, twiddles and row sectors).
cudaError_t matvec_fast_prepare(const Lat &L, int fx, int fyz, int form);
int matvec_fast_x_tile(int nl);           // spectral columns per TMA tile, 0: row too short
constexpr bool fast_x_waits(int fx) { return (fx >= 3 && fx < 6) || fx >= 9; }   // x variants with a bounded wait
void matvec_fast_defaults(const Lat &L, bool has_tmap, int *fx, int *fyz);   // untuned launch variants
cudaError_t launch_matvec_fast(const MatvecArgs &a, cudaStream_t st);
// CTAs per plane of the y/z passes: at most 4096 pairs (64 KB of shared memory) each
__host__ __device__ constexpr int matvec_z_split(int nj, int nl) { return nj * nl <= 4096 ? 1 : nj * nl <= 8192 ? 2 : 4; }
// per edge, one object each (Makefile)
template <int NJ> cudaError_t yz_prepare(int nl, int fyz, int form);
template <int NJ> cudaError_t yz_launch(const MatvecArgs &a, int fwd, cudaStream_t st);
template <int NI> cudaError_t x_prepare(int nl, int fx, int form);
template <int NI> cudaError_t x_launch(const MatvecArgs &a, cudaStream_t st);
#define DDA_EDGES(F) F(4) F(8) F(16) F(32) F(64) F(128)
#define DDA_DECLARE(N)                                                                        \
    template <> cudaError_t yz_prepare<N>(int nl, int fyz, int form);                         \
    template <> cudaError_t yz_launch<N>(const MatvecArgs &a, int fwd, cudaStream_t st);      \
    template <> cudaError_t x_prepare<N>(int nl, int fx, int form);                           \
    template <> cudaError_t x_launch<N>(const MatvecArgs &a, cudaStream_t st);
DDA_EDGES(DDA_DECLARE)
#undef DDA_DECLARE

// Pinned host memory of at least `bytes` (*size), from blocks given back before where one fits
// (pinned.cu).  No work on the device may use a block that is given back.
cudaError_t pinned_take(size_t bytes, unsigned char **p, size_t *size);
void pinned_give(unsigned char *p, size_t size);

// smaller factor R2 of an edge's line split (pair.cuh line_split)
constexpr int line_r2(int n) { return n <= 8 ? 2 : n <= 32 ? 4 : 8; }

// Green tensor (green.cu)
cudaError_t green_build_octant(int ni, int nj, int nl, double kd, float4 *ahat, cudaStream_t st);
cudaError_t green_project_dense(int ni, int nj, int nl, const float2 *dense_dev, float4 *ahat,
                                cudaStream_t st);
size_t ahat_elems(int ni, int nj, int nl);   // float4

}  // namespace ddagpu
