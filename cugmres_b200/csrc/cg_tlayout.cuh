// Layout of the matvec's N x L intermediate T: the columns in groups of G =
// t_group values (64 bytes), T[c / G][row][c % G].
//
// With plain rows of L values a column's elements lay L apart (32 KB at L = 2048 in
// FP64): every load and store of the column pass touched one sector of a line per
// row, and the lines of one column shared a few DRAM and L2 sets.  Here they are 64
// bytes apart, the rest of a line belonging to columns that neighbouring blocks work
// on, while the neighbouring lanes of a row pass still read and write 64 bytes at a
// time.  Products, us a call, rows of L / groups of 32 / 64 / 128 bytes: FP64 385^2
// 37.5 / 37.5 / 35.9 / 35.7, 1024^2 90.3 / 91.0 / 89.2 / 89.5, 2048^2 351 / 334 / 324 / 345;
// FP32 512^2 35.0 / 30.9 / 30.4 / 32.1, 1024^2 65.6 / 64.1 / 62.7 / 65.4, 2048^2 205 / 192 /
// 189 / 202 (32 bytes scatter the row passes' accesses, 128 the column pass's).
#pragma once

#include "cg_common.cuh"

namespace cg {

template <typename C> __host__ __device__ constexpr int t_group() { return 64 / (int)sizeof(C); }
// first element of column c; its element of `row` follows at row * t_group
template <typename C> __device__ __forceinline__ size_t t_column(int c, int N) {
    constexpr int G = t_group<C>();
    return (size_t)(c / G) * G * N + c % G;
}

}  // namespace cg
