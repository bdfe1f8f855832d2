// The build's own insertion order (order.cu): one radix sort of space-filling
// curve keys in place of the reference's spatial sort.
#pragma once

#include "common.cuh"

#include <cstdint>

namespace d3g {

/// Levels a build's own order uses at most (growth 2 of 2^27 points: 25).
constexpr int kMaxOrderLevels = 32;

/// The coarsest levels of every set together have about this many points (fewer
/// if the set has), so that one block can build them in shared memory
/// (k_coarse), which has room for kCoarseCap: the number of points in a level
/// comes from a hash and scatters by its square root.
constexpr int kCoarsePoints = 790;
constexpr int kCoarseCap = 880;

/// The first levels of a set of n points: the ones up to kCoarsePoints points, a
/// half (1 / growth) of what is left each while 16 points are (the reference's
/// multiscale split, src/spatial_sort.cpp:130-137, stops at 64: its levels bound
/// a walk's length, these also how many groups may insert at a time).
__host__ __device__ inline int coarse_levels(int64_t n, int growth) {
    int k = 1;
    for (int64_t m = n < kCoarsePoints ? n : kCoarsePoints; m >= 16; m /= growth) ++k;
    return k;
}

/// All levels of a set of n points: behind the coarse ones, levels that make the
/// points in so far `growth` times as many.
__host__ __device__ inline int order_levels(int64_t n, int growth) {
    int k = coarse_levels(n, growth);
    for (int64_t m = kCoarsePoints; m < n && k < kMaxOrderLevels; m *= growth) ++k;
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
/// the repeated points.  `S` and `d_nonfinite` from scan_sets (an error status where it
/// is raised).  Synchronises `s`.
int own_order_sets(const double* d_xyz, const int64_t* h_off, const int64_t* d_off, int nsets, int growth,
                   const SetScan& S, const uint32_t* d_nonfinite, OwnOrder& O, cudaStream_t s);

}  // namespace d3g
