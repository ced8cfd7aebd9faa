// Dispatch of the compile-time-sized matvec passes (matvec_yz.cu, matvec_x.cu: one object per edge).
#include "internal.h"

namespace ddagpu {

namespace {

bool fast_edge(int n) { return n >= 4 && n <= 128 && (n & (n - 1)) == 0; }

}  // namespace

bool matvec_fast_supported(const Lat &L) { return fast_edge(L.ni) && fast_edge(L.nj) && fast_edge(L.nl); }

// spectral columns per TMA tile of the x pass; 0 where the rows are shorter
int matvec_fast_x_tile(int nl) { return nl >= 8 ? 16 : 0; }

void matvec_fast_defaults(const Lat &L, bool has_tmap, int *fx, int *fyz)
{
    *fx = L.ni == 64 ? 1 : has_tmap ? 9 : 6;
    *fyz = (long long)L.nj * L.nl <= 1024 ? 1 : 0;
}

cudaError_t matvec_fast_prepare(const Lat &L, int fx, int fyz, int form)
{
    cudaError_t e = cudaErrorInvalidValue;
    switch (L.nj) {
#define CASE(N) case N: e = yz_prepare<N>(L.nl, fyz, form); break;
        DDA_EDGES(CASE)
#undef CASE
    }
    if (e != cudaSuccess) return e;
    switch (L.ni) {
#define CASE(N) case N: return x_prepare<N>(L.nl, fx, form);
        DDA_EDGES(CASE)
#undef CASE
    }
    return cudaErrorInvalidValue;
}

static cudaError_t yz(const MatvecArgs &a, int fwd, cudaStream_t st)
{
    switch (a.L.nj) {
#define CASE(N) case N: return yz_launch<N>(a, fwd, st);
        DDA_EDGES(CASE)
#undef CASE
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_matvec_fast(const MatvecArgs &args, cudaStream_t st)
{
    if (args.fx >= 9 && args.L.nl >= 8 && !args.tmaps) return cudaErrorInvalidValue;   // no tensor maps for the TMA variants
    MatvecArgs a = args;
    a.zs = matvec_z_split(a.L.nj, a.L.nl);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaError_t e = cudaStreamIsCapturing(st, &cap)) return e;
    a.chained = cap == cudaStreamCaptureStatusNone;
    cudaError_t e = yz(a, 1, st);
    if (e != cudaSuccess) return e;
    switch (a.L.ni) {
#define CASE(N) case N: e = x_launch<N>(a, st); break;
        DDA_EDGES(CASE)
#undef CASE
    default: e = cudaErrorInvalidValue;
    }
    return e == cudaSuccess ? yz(a, 0, st) : e;
}

}  // namespace ddagpu
