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
// z order of the Green octant for those rows: bins by parity, then class r, then m, so that a run
// of columns (of the mirrored half too) reads two runs of entries
__host__ __device__ inline int z_entries(int nl, int zs) { return 2 * zs * (nl / (2 * zs) + 1); }
__host__ __device__ inline int z_order(int oz, int nl, int zs)
{
    const int k = oz >> 1;
    return ((oz & 1) * zs + k % zs) * (nl / (2 * zs) + 1) + k / zs;
}

}  // namespace ddagpu
