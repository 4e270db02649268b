// Sparse linear maps (Lie <-> tensor) in a packed form: y = scale M x [+ y].
#pragma once

#include <vector>

#include "common.cuh"

namespace rpyb {

// Sizes of a packed map; its arrays follow one another in one block:
//   double tab[ntab], uint32 goff[groups + 1], perm[32 groups], len[32 groups],
//   ent[slots]
// Rows are taken 32 to a group, one per warp lane; entry j of lane l of group
// g is ent[goff[g] + 32 j + l] = column | value id << 20 for j < len[32 g + l]
// (entries past len pad the group and are not used), tab holds the distinct
// values and perm[32 g + l] the lane's row, or 0xffffffff past the last row.
struct PackedMap {
    int64_t n_rows = 0, n_cols = 0;
    int64_t groups = 0, slots = 0, ntab = 0;
    const void* block = nullptr;   // device
};

inline size_t packed_map_bytes(const PackedMap& m)
{
    return (size_t)(m.ntab * 8 + (m.groups + 1) * 4 + m.groups * 64 * 4 + m.slots * 4);
}

// Packs a CSR map (host arrays).  Returns false when a column does not fit 20
// bits or the distinct values 12 bits.  Entries whose column lies outside
// [0, n_cols) are left out.
bool pack_map(int64_t n_rows, int64_t n_cols, const int64_t* ptr, const int64_t* idx,
              const double* val, PackedMap& m, std::vector<unsigned char>& block);

// y[b] = scale M x[b] (+ y[b] when accumulating), float64 arithmetic, terms of
// a row in the CSR order.
int launch_packed_map(int dtype, const PackedMap& m, int64_t batch, void* y, int64_t ld_y,
                      const void* x, int64_t ld_x, double scale, bool accumulate, cudaStream_t s);

}  // namespace rpyb
