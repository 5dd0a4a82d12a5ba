// Table of the z derivative of physical fields (DBYD2 * stretch, dbyd2.f90:8-237;
// zderiv_kernel in mhd_step.cu): each pencil on chunks of ZCS levels, one per
// thread, whose carries are sums over the ZKB nearest chunks.
//
// Per boundary code the rows PS_* [PS_COUNT][nzp] of the solve for y = f' -
// (C2/alpha) (f(j+1) - f(j-1)) (as pencil.cu: stretch and the coefficients sit in
// the rows), the products [2][nw][ZKB - 1] of the 1..4 chunk multipliers below /
// above a chunk, and the closures [2 ends][PE_COUNT].
#pragma once
#include "internal.cuh"

constexpr int ZCS = 10, ZKB = 5;      // levels per thread; chunks summed by a carry
__host__ __device__ inline int z_chunks(int nz) { return (nz + ZCS - 1) / ZCS; }
__host__ __device__ inline int z_code_size(int nz) {
    const int nw = z_chunks(nz);
    return PS_COUNT * nw * ZCS + 2 * nw * (ZKB - 1) + 2 * PE_COUNT;
}
