// Random targets of libddagpu (agglomerates, random ellipsoids): host placement, GPU rasterisation.
#pragma once
#include <cuda_runtime.h>

namespace ddagpu {

long long anthrax_count(int ni, int nj, int nl, float packing, float radius, float ratio);
int anthrax_place(unsigned long long *state, int ni, float radius, float length, int count,
                  float *cyl13, long long max_tries);
cudaError_t anthrax_rasterize(const float *cyl13, int count, int ni, int nj, int nl,
                              signed char *occ_dev, int *ndip_dev, cudaStream_t st);
// no realisations (monomer lists one after the other in cyl13) into occ_dev [2 no][N], each at 2k
// and 2k + 1 (both polarisations), and their dipole counts; scratch holds anthrax_batch_scratch bytes
size_t anthrax_batch_scratch(int ni, int nj, int nl, int no, size_t total);
cudaError_t anthrax_rasterize_batch(const float *cyl13, const int *counts, int no, int ni, int nj, int nl,
                                    signed char *occ_dev, int *ndip_dev, cudaStream_t st, void *scratch);
// occupancies src [no][N] to occ [2 no][N] (each twice) and their active cells to nact [no];
// src and occ 16-byte aligned
cudaError_t launch_spread_occupancies(const signed char *src, signed char *occ, size_t N, int no, const int *mv,
                                      int nmat1, int *nact, cudaStream_t st);

int random_ellipsoid_seeds(unsigned long long *state, int ni, int nj, int nl, float b_a, float c_a,
                           int nseeds, float *seeds3);
cudaError_t random_ellipsoid_fill(const float *seeds3, const int *counts, int nsorts, int ni, int nj,
                                  int nl, float b_a, float c_a, signed char *occ_dev, int *ndip_dev,
                                  cudaStream_t st);

}  // namespace ddagpu
