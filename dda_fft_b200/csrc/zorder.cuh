// Order of the spectral z axis in the work buffer and in the Green tensor of the sized passes.
#pragma once

namespace ddagpu {

// Bin of spectral column `col` of a row whose y/z passes split the z axis zs ways: col =
// 2 (r ML + m) + h holds bin 2 (zs m + r) + h
__host__ __device__ inline int z_bin(int col, int nl, int zs)
{
    const int zpos = col >> 1, ml = nl / zs, r = zpos / ml;
    return 2 * (zs * (zpos - r * ml) + r) + (col & 1);
}
// z order of the Green octant for those rows: by class r, then m and parity (a run of columns
// reads a run of entries), or with `split` by parity first (a run of zpos reads a run per parity)
__host__ __device__ inline int z_entries(int nl, int zs) { return 2 * zs * (nl / (2 * zs) + 1); }
__host__ __device__ inline int z_order(int oz, int nl, int zs, int split)
{
    const int k = oz >> 1, h = oz & 1, n = nl / (2 * zs) + 1;
    return split ? (h * zs + k % zs) * n + k / zs : (k % zs) * 2 * n + 2 * (k / zs) + h;
}
// the pass at edge 64 takes runs of columns, the packed one at the others runs of zpos
__host__ __device__ inline int z_parity_split(int ni) { return ni != 64; }

}  // namespace ddagpu
