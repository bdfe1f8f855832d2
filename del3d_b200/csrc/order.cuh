// The build's own insertion order (order.cu): one radix sort of space-filling
// curve keys in place of the reference's spatial sort.
#pragma once

#include "common.cuh"

#include <cstdint>

namespace d3g {

/// Levels a build's own order uses at most (growth 2 of 2^27 points: 22).
constexpr int kMaxOrderLevels = 32;

/// Levels of a set of n points when each level is `growth` times the points
/// before it: n, n / growth, ... while at least 64 points are left (as the
/// reference's multiscale split, src/spatial_sort.cpp:130-137, at growth 8).
__host__ __device__ inline int order_levels(int64_t n, int growth) {
    int k = 1;
    while (n >= 64 && k < kMaxOrderLevels) {
        n /= growth;
        ++k;
    }
    return k;
}

/// What one pass over the input says of each set: its bounding box, whether
/// its coordinates make the filters exact (see k_set_exact), and whether any
/// coordinate of the call is not finite.
struct SetScan {
    DevBuf<unsigned long long> box;   // per set: order keys of min x, y, z, max x, y, z
    DevBuf<int> span;                 // nsets lowest set bits, then nsets tops
};
int scan_sets(const double* d_xyz, const int64_t* d_off, int nsets, int64_t n, SetScan& S, uint32_t* d_nonfinite,
              cudaStream_t s);

/// The vertices of every set in the build's own order.
struct OwnOrder {
    DevBuf<int32_t> vert;        // per vertex: the global index of its first copy
    DevBuf<int32_t> rep;         // with repeated points: per vertex the local index it is reported under
    DevBuf<int32_t> level_start; // nsets * levels + 1: first vertex of each (set, level)
    DevBuf<unsigned long long> keys;   // per vertex its sorted key, the Hilbert index in the low curve_bits
    int curve_bits = 0;
    int64_t nv = 0;              // distinct points
    int levels = 0;              // levels per set in level_start
    bool ok = false;             // false: the keys cannot tell the points apart (use the spatial sort)
};
/// Orders every set coarse to fine, each level along a Hilbert curve, and finds
/// the repeated points.  `S` from scan_sets.  Synchronises `s`.
int own_order_sets(const double* d_xyz, const int64_t* h_off, const int64_t* d_off, int nsets, int growth,
                   const SetScan& S, OwnOrder& O, cudaStream_t s);

}  // namespace d3g
