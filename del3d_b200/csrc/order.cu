// The build's own insertion order.
//
// The cells do not depend on the order points go in (see build.cu), so a build
// need not pay for the reference's order, whose quickselects are serial in
// depth and take passes over every run of equal coordinates: 63 ms of "big
// splits" for 10^7 uniform points, 62 ms for the 100^3 lattice, where the runs
// are 10^4 long.  Here a point's place is one 64-bit key,
//
//     set | level | Hilbert index of its cell in the set's bounding cube
//
// sorted by one radix sort.  The level comes from a hash of the coordinates, so
// equal points share their whole key and end up next to each other: the
// repeated points are found in the sorted keys, without the sorts of every
// coordinate that the spatial sort needs after it.  The reference's order
// decides one thing, which copy of a repeated point keeps its index (the last
// one in that order, src/triangulation.cpp:77-81); it is worked out only when
// there are repeated points.
//
// Bound by the radix sort's passes over 12-byte pairs (8 of them).  Whole builds
// on one B200, spatial sort and coordinate sorts -> this: 10^7 uniform points
// 272 -> 191 ms, the 100^3 lattice 131-224 -> 69 ms, 10^6 uniform 71.8 -> 57.3
// ms, 4096 mixed sets (35 M points) 664 -> 593 ms.
#include "device_util.cuh"
#include "order.cuh"

#include <algorithm>
#include <vector>

namespace d3g {

int spatial_order_sets_device(const double* d_xyz, const int64_t* h_off, const int64_t* d_off, int nsets,
                              int32_t* d_order, cudaStream_t s, double level_ratio = 0.125);

namespace {

constexpr unsigned kFullMask = 0xffffffffu;
/// Points with equal keys looked through for equal points; a longer run (many
/// copies of one point, or a set far denser than its bounding cube's grid in
/// one place) is sorted again by the grid of its own bounding cube.
constexpr int kKeyRun = 32;
/// How often: each time makes the cells at least 2^13 times smaller (2^21 times with
/// few runs).  Where runs are left even then, or a set's extent overflows, the call goes
/// to the spatial sort.
constexpr int kRefine = 12;

__device__ __forceinline__ int set_of(const int64_t* __restrict__ off, int nsets, int64_t g) {
    int lo = 0, hi = nsets - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void k_scan_init(unsigned long long* box, int* span, int nsets) {
    for (int i = int(blockIdx.x) * blockDim.x + threadIdx.x; i < 6 * nsets; i += gridDim.x * blockDim.x) {
        box[i] = i % 6 < 3 ? ~0ull : 0ull;
        if (i < 2 * nsets) span[i] = i < nsets ? (1 << 20) : -(1 << 20);
    }
}

/// One pass over the coordinates: each warp takes kScanRun consecutive points,
/// keeps box and span of the set it is in in registers and adds them to the
/// set's with one atomic each when the set ends.  Bound by reading the points.
constexpr int kScanRun = 1024;
__global__ void __launch_bounds__(256) k_scan_sets(const double* __restrict__ xyz, const int64_t* __restrict__ off,
                                                   int nsets, int64_t n, unsigned long long* __restrict__ box,
                                                   int* __restrict__ span, uint32_t* __restrict__ nonfinite) {
    const int lane = threadIdx.x & 31;
    const int64_t first = ((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * kScanRun;
    if (first >= n) return;
    const int64_t last = min(n, first + kScanRun);
    unsigned long long lo[3], hi[3];
    Span sp;
    bool bad = false;
    auto clear = [&]() {
        for (int a = 0; a < 3; ++a) {
            lo[a] = ~0ull;
            hi[a] = 0ull;
        }
        sp = Span();
    };
    auto flush = [&](int set) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            for (int a = 0; a < 3; ++a) {
                lo[a] = min(lo[a], __shfl_xor_sync(kFullMask, lo[a], o));
                hi[a] = max(hi[a], __shfl_xor_sync(kFullMask, hi[a], o));
            }
            sp.emin = min(sp.emin, __shfl_xor_sync(kFullMask, sp.emin, o));
            sp.top = max(sp.top, __shfl_xor_sync(kFullMask, sp.top, o));
        }
        if (lane < 3) {
            const unsigned long long l = lane == 0 ? lo[0] : (lane == 1 ? lo[1] : lo[2]);
            const unsigned long long h = lane == 0 ? hi[0] : (lane == 1 ? hi[1] : hi[2]);
            atomicMin(box + 6 * int64_t(set) + lane, l);
            atomicMax(box + 6 * int64_t(set) + 3 + lane, h);
        } else if (lane == 3 && !sp.empty()) {
            atomicMin(span + set, sp.emin);
            atomicMax(span + nsets + set, sp.top);
        }
        clear();
    };
    clear();
    int cur = set_of(off, nsets, first);
    int64_t end = off[cur + 1];
    for (int64_t p0 = first; p0 < last;) {
        while (p0 >= end) end = off[++cur + 1];   // empty sets hold no point
        const int64_t stop = min(last, end);
        for (int64_t p = p0 + lane; p < stop; p += 32) {
            for (int a = 0; a < 3; ++a) {
                const double x = xyz[3 * p + a];
                if (!isfinite(x)) {
                    bad = true;
                    continue;
                }
                const unsigned long long k = dbl_order_key(x);
                lo[a] = min(lo[a], k);
                hi[a] = max(hi[a], k);
                sp.add(x);
            }
        }
        p0 = stop;
        __syncwarp();
        flush(cur);
    }
    if (__any_sync(kFullMask, bad) && lane == 0) atomicOr(nonfinite, 1u);
}

/// A 64-bit finaliser (shift, multiply, shift): every input bit reaches every
/// output bit.  Constant and shifts are those published as "degski64".
__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
    x ^= x >> 32;
    x *= 0xD6E8FEB86659FD93ull;
    x ^= x >> 32;
    x *= 0xD6E8FEB86659FD93ull;
    x ^= x >> 32;
    return x;
}

__device__ __forceinline__ unsigned long long coord_bits(double x) {   // -0.0 equals +0.0
    return x == 0.0 ? 0ull : (unsigned long long)__double_as_longlong(x);
}

/// Spreads the low 21 bits of x to every third bit.
__device__ __forceinline__ unsigned long long spread3(unsigned x) {
    unsigned long long v = x & 0x1FFFFFu;
    v = (v | v << 32) & 0x001F00000000FFFFull;
    v = (v | v << 16) & 0x001F0000FF0000FFull;
    v = (v | v << 8) & 0x100F00F00F00F00Full;
    v = (v | v << 4) & 0x10C30C30C30C30C3ull;
    v = (v | v << 2) & 0x1249249249249249ull;
    return v;
}

/// Hilbert index of cell (x, y, z) of a 2^bits grid, by Skilling's transform
/// ("Programming the Hilbert curve", AIP Conf. Proc. 707, 2004): from the high
/// bit down, undo the rotations and reflections of each subcube, then Gray
/// encode.
__device__ __forceinline__ unsigned long long hilbert3(unsigned x, unsigned y, unsigned z, int bits) {
    for (unsigned q = 1u << (bits - 1); q > 1; q >>= 1) {
        const unsigned p = q - 1;
        if (x & q) x ^= p;
        if (y & q) x ^= p;
        else {
            const unsigned t = (x ^ y) & p;
            x ^= t;
            y ^= t;
        }
        if (z & q) x ^= p;
        else {
            const unsigned t = (x ^ z) & p;
            x ^= t;
            z ^= t;
        }
    }
    y ^= x;
    z ^= y;
    unsigned t = 0;
    for (unsigned q = 1u << (bits - 1); q > 1; q >>= 1)
        if (z & q) t ^= q - 1;
    x ^= t;
    y ^= t;
    z ^= t;
    return spread3(x) << 2 | spread3(y) << 1 | spread3(z);
}

/// The cell of x, on a grid of 2^bits cells from lo on; scale 0 for one point or an
/// overflow.
__device__ __forceinline__ unsigned cell_of(double x, double lo, double scale, int bits) {
    const double f = (x - lo) * scale;
    return f > 0.0 ? min(unsigned(f), (1u << bits) - 1) : 0u;
}

/// The key of every point.  A point's level comes from its hash as a fraction of
/// 2^32: the coarse levels share the part below kCoarsePoints / n, each `growth`
/// times the points before it, the others the part above, likewise.
__global__ void __launch_bounds__(256) k_order_keys(const double* __restrict__ xyz, const int64_t* __restrict__ off,
                                                    int nsets, int64_t n, const unsigned long long* __restrict__ box,
                                                    int growth, int bits, int level_bits,
                                                    unsigned long long* __restrict__ keys,
                                                    int32_t* __restrict__ idx) {
    for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += int64_t(gridDim.x) * blockDim.x) {
        const int set = nsets > 1 ? set_of(off, nsets, p) : 0;
        const unsigned long long* b = box + 6 * int64_t(set);
        double ext = 0.0, lo[3];
        for (int a = 0; a < 3; ++a) {
            lo[a] = dbl_from_order_key(b[a]);
            ext = fmax(ext, dbl_from_order_key(b[3 + a]) - lo[a]);
        }
        // 2^bits cells along the longest side.
        const double scale = ext > 0.0 ? double((1u << bits) - 1) / ext : 0.0;
        unsigned q[3];
        unsigned long long h = 0;
        for (int a = 0; a < 3; ++a) {
            const double x = xyz[3 * p + a];
            q[a] = cell_of(x, lo[a], scale, bits);
            h = mix64(h + 0x9E3779B97F4A7C15ull + coord_bits(x));
        }
        const int64_t ns = off[set + 1] - off[set];
        const int nlev = order_levels(ns, growth), ncoarse = coarse_levels(ns, growth);
        const uint64_t one = uint64_t(1) << 32, t0 = ns <= kCoarsePoints ? one : one * kCoarsePoints / uint64_t(ns);
        uint64_t r = h >> 32;
        int lev;
        if (r < t0) {
            lev = ncoarse - 1;
            for (; lev > 0 && r * unsigned(growth) < t0; --lev) r *= unsigned(growth);
        } else {
            lev = ncoarse;
            for (uint64_t t = t0 * unsigned(growth); lev < nlev - 1 && r >= t; t *= unsigned(growth)) ++lev;
        }
        const unsigned long long code = (unsigned long long)set << level_bits | unsigned(lev);
        keys[p] = code << (3 * bits) | hilbert3(q[0], q[1], q[2], bits);
        idx[p] = int32_t(p);
    }
}

__device__ __forceinline__ bool equal_points(const double* __restrict__ xyz, int64_t i, int64_t j) {
    return xyz[3 * i] == xyz[3 * j] && xyz[3 * i + 1] == xyz[3 * j + 1] && xyz[3 * i + 2] == xyz[3 * j + 2];
}

/// Over the sorted keys (the set above bit `set_shift`): the first copy of every
/// point (head[i] == i for one), and how many others there are (flags[0], and per
/// set from flags[2] on); flags[1] is raised by a run of equal keys too long to be
/// looked through.  The finite check's result goes behind the flags, to be read back
/// with them.
__global__ void __launch_bounds__(256) k_first_copies(const double* __restrict__ xyz,
                                                      const unsigned long long* __restrict__ keys,
                                                      const int32_t* __restrict__ idx, int64_t n, int nsets,
                                                      int set_shift, const uint32_t* __restrict__ nonfinite,
                                                      int32_t* __restrict__ head, int* __restrict__ flags) {
    if (blockIdx.x == 0 && threadIdx.x == 0) flags[2 + nsets] = int(*nonfinite);
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const unsigned long long k = keys[i];
        int64_t first = i, j = i - 1;
        for (; j >= 0 && i - j <= kKeyRun && keys[j] == k; --j)
            if (equal_points(xyz, idx[i], idx[j])) first = j;
        if (i - j > kKeyRun && j >= 0 && keys[j] == k) atomicOr(flags + 1, 1);
        head[i] = int32_t(first);
        if (first != i) {
            atomicAdd(flags, 1);
            atomicAdd(flags + 2 + (nsets > 1 ? int(k >> set_shift) : 0), 1);
        }
    }
}

// ---- long runs of equal keys --------------------------------------------------------
//
// A run's points share set, level and cell.  The runs longer than kKeyRun are sorted
// again by the Hilbert index in their own bounding cubes, together (run | index), and
// what is left of them once more, until no run is long but those of one point's
// copies, whose cube has no extent.  tie[i]: 0 where i's key differs from that of the
// one before, 1 where it is equal, 2 where the points are.

enum : uint8_t { TIE_NONE = 0, TIE_KEY = 1, TIE_COPY = 2 };

__global__ void k_tie_init(const unsigned long long* __restrict__ keys, int64_t n, uint8_t* __restrict__ tie) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        tie[i] = i > 0 && keys[i] == keys[i - 1] ? TIE_KEY : TIE_NONE;
}

/// Heads of runs, to be summed up into every point's run number (plus one).
__global__ void k_run_heads(const uint8_t* __restrict__ tie, int64_t n, int32_t* __restrict__ head) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i <= n; i += int64_t(gridDim.x) * blockDim.x)
        head[i] = i < n && tie[i] == TIE_NONE ? 1 : 0;
}

/// start[r]: run r's first point, over the exclusive sums of the heads (n + 1 of them).
__global__ void k_run_starts(const uint8_t* __restrict__ tie, const int32_t* __restrict__ before, int64_t n,
                             int32_t* __restrict__ start) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i <= n; i += int64_t(gridDim.x) * blockDim.x)
        if (i == n || tie[i] == TIE_NONE) start[before[i]] = int32_t(i);
}

__device__ __forceinline__ int run_of(const uint8_t* __restrict__ tie, const int32_t* __restrict__ before, int64_t i) {
    return before[i] - (tie[i] == TIE_NONE ? 0 : 1);
}

/// Flags the points of the long runs (not those of copies), and of these the first.
__global__ void k_long_flags(const uint8_t* __restrict__ tie, const int32_t* __restrict__ before,
                             const int32_t* __restrict__ start, int64_t n, int32_t* __restrict__ in,
                             int32_t* __restrict__ first) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i <= n; i += int64_t(gridDim.x) * blockDim.x) {
        int yes = 0, head = 0;
        if (i < n) {
            const int r = run_of(tie, before, i), a = start[r], e = start[r + 1];
            yes = e - a > kKeyRun && tie[a + 1] == TIE_KEY ? 1 : 0;
            head = yes && a == i ? 1 : 0;
        }
        in[i] = yes;
        first[i] = head;
    }
}

/// The flagged points side by side: where they stand (at) and their run among the
/// long ones (seg); the sums are exclusive, of n + 1 flags.
__global__ void k_long_gather(const int32_t* __restrict__ in, const int32_t* __restrict__ first, int64_t n,
                              int32_t* __restrict__ at, int32_t* __restrict__ seg) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        if (in[i + 1] == in[i]) continue;
        at[in[i]] = int32_t(i);
        seg[in[i]] = first[i + 1] - 1;
    }
}

__global__ void k_box_init(unsigned long long* box, int nseg) {
    for (int i = int(blockIdx.x) * blockDim.x + threadIdx.x; i < 6 * nseg; i += gridDim.x * blockDim.x)
        box[i] = i % 6 < 3 ? ~0ull : 0ull;
}

/// The bounding boxes of the long runs; a warp whose points are all of one run adds
/// them up first.
__global__ void __launch_bounds__(256) k_long_boxes(const double* __restrict__ xyz, const int32_t* __restrict__ idx,
                                                    const int32_t* __restrict__ at, const int32_t* __restrict__ seg,
                                                    int m, unsigned long long* __restrict__ box) {
    const int lane = threadIdx.x & 31;
    const int padded = (m + 31) & ~31;
    for (int j = int(blockIdx.x) * blockDim.x + threadIdx.x; j < padded; j += gridDim.x * blockDim.x) {
        const bool have = j < m;
        const int s = have ? seg[j] : -1;
        const int64_t p = have ? idx[at[j]] : 0;
        const int s0 = __shfl_sync(kFullMask, s, 0);
        const bool one = __all_sync(kFullMask, s >= 0 && s == s0);
        for (int a = 0; a < 3; ++a) {
            unsigned long long lo = have ? dbl_order_key(xyz[3 * p + a]) : 0ull, hi = lo;
            if (one)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    lo = min(lo, __shfl_xor_sync(kFullMask, lo, o));
                    hi = max(hi, __shfl_xor_sync(kFullMask, hi, o));
                }
            if (have && (!one || lane == 0)) {
                atomicMin(box + 6 * int64_t(s) + a, lo);
                atomicMax(box + 6 * int64_t(s) + 3 + a, hi);
            }
        }
    }
}

__global__ void __launch_bounds__(256) k_long_keys(const double* __restrict__ xyz, const int32_t* __restrict__ idx,
                                                   const int32_t* __restrict__ at, const int32_t* __restrict__ seg,
                                                   int m, const unsigned long long* __restrict__ box, int bits,
                                                   unsigned long long* __restrict__ keys,
                                                   int32_t* __restrict__ val) {
    for (int j = int(blockIdx.x) * blockDim.x + threadIdx.x; j < m; j += gridDim.x * blockDim.x) {
        const unsigned long long* b = box + 6 * int64_t(seg[j]);
        const int32_t p = idx[at[j]];
        double ext = 0.0, lo[3];
        for (int a = 0; a < 3; ++a) {
            lo[a] = dbl_from_order_key(b[a]);
            ext = fmax(ext, dbl_from_order_key(b[3 + a]) - lo[a]);
        }
        const double scale = ext > 0.0 ? double((1u << bits) - 1) / ext : 0.0;
        unsigned q[3];
        for (int a = 0; a < 3; ++a) q[a] = cell_of(xyz[3 * int64_t(p) + a], lo[a], scale, bits);
        keys[j] = (unsigned long long)seg[j] << (3 * bits) | hilbert3(q[0], q[1], q[2], bits);
        val[j] = p;
    }
}

/// The sorted points back in their places.
__global__ void k_long_scatter(const unsigned long long* __restrict__ keys, const int32_t* __restrict__ val,
                               const int32_t* __restrict__ at, int m, const unsigned long long* __restrict__ box,
                               int seg_shift, int32_t* __restrict__ idx, uint8_t* __restrict__ tie) {
    for (int j = int(blockIdx.x) * blockDim.x + threadIdx.x; j < m; j += gridDim.x * blockDim.x) {
        const unsigned long long k = keys[j];
        const unsigned long long* b = box + 6 * (k >> seg_shift);
        uint8_t t = TIE_NONE;
        if (j > 0 && (keys[j - 1] >> seg_shift) == (k >> seg_shift)) {
            double ext = 0.0;
            for (int a = 0; a < 3; ++a) ext = fmax(ext, dbl_from_order_key(b[3 + a]) - dbl_from_order_key(b[a]));
            t = ext == 0.0 ? TIE_COPY : (keys[j - 1] == k ? TIE_KEY : TIE_NONE);
        }
        idx[at[j]] = val[j];
        tie[at[j]] = t;
    }
}

/// k_first_copies by the ties.
__global__ void __launch_bounds__(256) k_first_tied(const double* __restrict__ xyz,
                                                    const unsigned long long* __restrict__ keys,
                                                    const int32_t* __restrict__ idx, const uint8_t* __restrict__ tie,
                                                    const int32_t* __restrict__ before,
                                                    const int32_t* __restrict__ start, int64_t n, int nsets,
                                                    int set_shift, int32_t* __restrict__ head,
                                                    int* __restrict__ flags) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        int64_t first = i;
        if (tie[i] == TIE_COPY) first = start[run_of(tie, before, i)];
        else
            for (int64_t j = i; tie[j] == TIE_KEY; --j)
                if (equal_points(xyz, idx[i], idx[j - 1])) first = j - 1;
        head[i] = int32_t(first);
        if (first != i) {
            atomicAdd(flags, 1);
            atomicAdd(flags + 2 + (nsets > 1 ? int(keys[i] >> set_shift) : 0), 1);
        }
    }
}

/// The coordinates of some sets side by side: set list[k] at off_of[k].
__global__ void __launch_bounds__(256) k_gather_sets(const double* __restrict__ xyz, const int64_t* __restrict__ off,
                                                     const int* __restrict__ list, const int64_t* __restrict__ off_of,
                                                     int m, int64_t n, double* __restrict__ out) {
    for (int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; p < n; p += int64_t(gridDim.x) * blockDim.x) {
        const int k = set_of(off_of, m, p);
        const int64_t from = off[list[k]] + (p - off_of[k]);
        for (int a = 0; a < 3; ++a) out[3 * p + a] = xyz[3 * from + a];
    }
}

/// Ranks in the reference's order, from that order of the sets of `list` (see
/// k_gather_sets; null: all sets).
__global__ void k_ranks(const int32_t* __restrict__ order, const int64_t* __restrict__ off,
                        const int* __restrict__ list, const int64_t* __restrict__ off_of, int m, int64_t n,
                        int32_t* __restrict__ rank) {
    for (int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; r < n; r += int64_t(gridDim.x) * blockDim.x) {
        const int k = set_of(off_of, m, r);
        rank[off[list ? list[k] : k] + order[r]] = int32_t(r - off_of[k]);
    }
}

/// With repeated points, each is reported under the copy whose rank in the
/// reference's order is the last: best[first copy] = (rank + 1) << 32 | local index
/// (0: no other copy).
__global__ void __launch_bounds__(256) k_best_copies(const int32_t* __restrict__ idx,
                                                     const int32_t* __restrict__ head,
                                                     const int32_t* __restrict__ rank,
                                                     const int64_t* __restrict__ off, int nsets, int64_t n,
                                                     unsigned long long* __restrict__ best) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const int32_t h = head[i];
        if (h == i) continue;
        const int32_t g = idx[i], f = idx[h];
        const int64_t set = off[set_of(off, nsets, g)];
        atomicMax(best + h, max((unsigned long long)(rank[g] + 1) << 32 | unsigned(g - set),
                                (unsigned long long)(rank[f] + 1) << 32 | unsigned(f - set)));
    }
}

/// The vertices are the first copies.
__global__ void __launch_bounds__(256) k_compact_copies(const unsigned long long* __restrict__ keys,
                                                        const int32_t* __restrict__ idx,
                                                        const int32_t* __restrict__ head,
                                                        const int32_t* __restrict__ pos,
                                                        const unsigned long long* __restrict__ best,
                                                        const int64_t* __restrict__ off, int nsets, int64_t n,
                                                        int32_t* __restrict__ vert, int32_t* __restrict__ rep,
                                                        unsigned long long* __restrict__ vkeys) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        if (head[i] != i) continue;
        const int32_t g = idx[i], v = pos[i];
        vert[v] = g;
        rep[v] = best[i] ? int32_t(best[i]) : int32_t(g - off[set_of(off, nsets, g)]);
        vkeys[v] = keys[i];
    }
}

__global__ void k_head_flags(const int32_t* __restrict__ head, int64_t n, int32_t* __restrict__ flag) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        flag[i] = head[i] == i ? 1 : 0;
}

/// start[c] = the first vertex of (set, level) c, over the vertices' sorted
/// keys (c = key >> shift, or its rank set * levels + level).
__global__ void k_level_starts(const unsigned long long* __restrict__ keys, int64_t nv, int shift, int level_bits,
                               int levels, int64_t total, int32_t* __restrict__ start) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i <= nv; i += int64_t(gridDim.x) * blockDim.x) {
        auto code = [&](int64_t v) {
            const unsigned long long c = keys[v] >> shift;
            return int64_t(c >> level_bits) * levels + int64_t(c & ((1ull << level_bits) - 1));
        };
        const int64_t from = i > 0 ? code(i - 1) + 1 : 0;
        const int64_t to = i < nv ? code(i) : total;
        for (int64_t c = from; c <= to; ++c) start[c] = int32_t(i);
    }
}

}  // namespace

int scan_sets(const double* d_xyz, const int64_t* d_off, int nsets, int64_t n, SetScan& S, uint32_t* d_nonfinite,
              cudaStream_t s) {
    D3G_TRY(S.box.alloc(size_t(6) * size_t(nsets), s));
    D3G_TRY(S.span.alloc(size_t(2) * size_t(nsets), s));
    k_scan_init<<<grid_for(6 * int64_t(nsets), 256), 256, 0, s>>>(S.box.p, S.span.p, nsets);
    const int64_t warps = (n + kScanRun - 1) / kScanRun;
    k_scan_sets<<<grid_for(warps * 32, 256, 1 << 30), 256, 0, s>>>(d_xyz, d_off, nsets, n, S.box.p, S.span.p,
                                                                   d_nonfinite);
    D3G_CUDA(cudaGetLastError());
    return D3G_OK;
}

namespace {

/// Sorts the long runs of equal keys (see above) and finds the first copies (head and
/// flags as k_first_copies; flags[1] stays raised if runs are left).
int refine_runs(const double* d_xyz, int64_t n, int nsets, int set_shift, const unsigned long long* keys, int32_t* idx,
                int32_t* head, int* flags, size_t nflags, cudaStream_t s) {
    DevBuf<uint8_t> tie;
    DevBuf<int32_t> before, start, in, first, at, seg, val, val2;
    DevBuf<unsigned long long> box, sub, sub2;
    D3G_TRY(tie.alloc(size_t(n), s));
    for (DevBuf<int32_t>* d : {&before, &start, &in, &first}) D3G_TRY(d->alloc(size_t(n) + 2, s));
    k_tie_init<<<grid_for(n, 256), 256, 0, s>>>(keys, n, tie.p);
    int left = 0;
    for (int pass = 0;; ++pass) {
        k_run_heads<<<grid_for(n + 1, 256), 256, 0, s>>>(tie.p, n, before.p);
        D3G_TRY(exclusive_scan(before.p, before.p, n + 1, s));
        k_run_starts<<<grid_for(n + 1, 256), 256, 0, s>>>(tie.p, before.p, n, start.p);
        k_long_flags<<<grid_for(n + 1, 256), 256, 0, s>>>(tie.p, before.p, start.p, n, in.p, first.p);
        D3G_TRY(exclusive_scan(in.p, in.p, n + 1, s));
        D3G_TRY(exclusive_scan(first.p, first.p, n + 1, s));
        int m = 0, nseg = 0;
        D3G_CUDA(cudaMemcpyAsync(&m, in.p + n, sizeof m, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaMemcpyAsync(&nseg, first.p + n, sizeof nseg, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaStreamSynchronize(s));
        left = m;
        if (m == 0 || pass == kRefine) break;
        const int seg_bits = bits_for(uint64_t(nseg)), bits = std::min(21, (64 - seg_bits) / 3);
        for (DevBuf<int32_t>* d : {&at, &seg, &val, &val2}) D3G_TRY(d->alloc(size_t(m), s));
        for (DevBuf<unsigned long long>* d : {&sub, &sub2}) D3G_TRY(d->alloc(size_t(m), s));
        D3G_TRY(box.alloc(size_t(6) * size_t(nseg), s));
        k_long_gather<<<grid_for(n, 256), 256, 0, s>>>(in.p, first.p, n, at.p, seg.p);
        k_box_init<<<grid_for(6 * int64_t(nseg), 256), 256, 0, s>>>(box.p, nseg);
        k_long_boxes<<<grid_for(m, 256), 256, 0, s>>>(d_xyz, idx, at.p, seg.p, m, box.p);
        k_long_keys<<<grid_for(m, 256), 256, 0, s>>>(d_xyz, idx, at.p, seg.p, m, box.p, bits, sub.p, val.p);
        D3G_TRY(sort_pairs(sub.p, sub2.p, val.p, val2.p, m, 0, 3 * bits + seg_bits, s));
        k_long_scatter<<<grid_for(m, 256), 256, 0, s>>>(sub2.p, val2.p, at.p, m, box.p, 3 * bits, idx, tie.p);
        D3G_CUDA(cudaGetLastError());
    }
    D3G_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * nflags, s));
    if (left > 0) {
        D3G_CUDA(cudaMemsetAsync(flags + 1, 1, sizeof(int), s));
        return D3G_OK;
    }
    k_first_tied<<<grid_for(n, 256), 256, 0, s>>>(d_xyz, keys, idx, tie.p, before.p, start.p, n, nsets, set_shift, head,
                                                  flags);
    D3G_CUDA(cudaGetLastError());
    return D3G_OK;
}

}  // namespace

int own_order_sets(const double* d_xyz, const int64_t* h_off, const int64_t* d_off, int nsets, int growth,
                   const SetScan& S, const uint32_t* d_nonfinite, OwnOrder& O, cudaStream_t s) {
    const int64_t n = h_off[nsets];
    O.ok = false;
    O.nv = 0;
    int64_t max_n = 0;
    for (int i = 0; i < nsets; ++i) max_n = std::max<int64_t>(max_n, h_off[i + 1] - h_off[i]);
    O.levels = order_levels(max_n, growth);
    const int level_bits = bits_for(uint64_t(O.levels - 1));
    const int set_bits = nsets > 1 ? bits_for(uint64_t(nsets - 1)) : 0;
    const int bits = std::min(21, (64 - level_bits - set_bits) / 3);
    const int shift = 3 * bits;
    DevBuf<unsigned long long> keys, keys2;
    DevBuf<int32_t> idx, idx2, head;
    DevBuf<int> flags;
    D3G_TRY(keys.alloc(size_t(n), s));
    D3G_TRY(keys2.alloc(size_t(n), s));
    D3G_TRY(idx.alloc(size_t(n), s));
    D3G_TRY(idx2.alloc(size_t(n), s));
    D3G_TRY(head.alloc(size_t(n), s));
    D3G_TRY(flags.alloc(3 + size_t(nsets), s));
    D3G_CUDA(cudaMemsetAsync(flags.p, 0, sizeof(int) * flags.n, s));
    k_order_keys<<<grid_for(n, 256), 256, 0, s>>>(d_xyz, d_off, nsets, n, S.box.p, growth, bits, level_bits, keys2.p,
                                                  idx2.p);
    D3G_TRY(sort_pairs(keys2.p, keys.p, idx2.p, idx.p, n, 0, shift + level_bits + set_bits, s));
    k_first_copies<<<grid_for(n, 256), 256, 0, s>>>(d_xyz, keys.p, idx.p, n, nsets, shift + level_bits, d_nonfinite,
                                                     head.p, flags.p);
    const int64_t total = int64_t(nsets) * O.levels;
    D3G_TRY(O.level_start.alloc(size_t(total) + 1, s));
    k_level_starts<<<grid_for(n + 1, 256), 256, 0, s>>>(keys.p, n, shift, level_bits, O.levels, total,
                                                        O.level_start.p);
    std::vector<int> hflags(flags.n);
    auto read_flags = [&]() -> int {
        D3G_CUDA(cudaMemcpyAsync(hflags.data(), flags.p, sizeof(int) * flags.n, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaStreamSynchronize(s));
        return D3G_OK;
    };
    D3G_TRY(read_flags());
    if (hflags.back()) {      // (its points cannot be ordered)
        set_error("d3g_build: non-finite coordinate");
        return D3G_ERR_INVALID_INPUT;
    }
    if (hflags[1]) {
        D3G_TRY(refine_runs(d_xyz, n, nsets, shift + level_bits, keys.p, idx.p, head.p, flags.p, flags.n, s));
        D3G_TRY(read_flags());
        if (hflags[1]) return D3G_OK;
    }
    O.nv = n - hflags[0];
    if (hflags[0] > 0) {
        // Which copy keeps its index is the reference's order's to say, so the sets with
        // copies are put in that order (4096 mixed sets, a fourth of them with one
        // point in 97 twice: order 61 -> 23 ms, the build 437 -> 399).
        std::vector<int> list;
        std::vector<int64_t> hoff_of(1, 0);
        for (int i = 0; i < nsets; ++i) {
            if (!hflags[size_t(i) + 2]) continue;
            list.push_back(i);
            hoff_of.push_back(hoff_of.back() + (h_off[i + 1] - h_off[i]));
        }
        const int m = int(list.size());
        const int64_t nm = hoff_of.back();
        DevBuf<int> dlist;
        DevBuf<int64_t> doff_of;
        DevBuf<double> some;
        DevBuf<int32_t> order, rank;
        D3G_TRY(order.alloc(size_t(nm), s));
        D3G_TRY(rank.alloc(size_t(n), s));
        const double* pts = d_xyz;
        const int64_t* off_of = d_off;
        if (m < nsets) {
            D3G_TRY(dlist.alloc(size_t(m), s));
            D3G_TRY(doff_of.alloc(size_t(m) + 1, s));
            D3G_TRY(some.alloc(size_t(3) * size_t(nm), s));
            D3G_CUDA(cudaMemcpyAsync(dlist.p, list.data(), sizeof(int) * size_t(m), cudaMemcpyHostToDevice, s));
            D3G_CUDA(cudaMemcpyAsync(doff_of.p, hoff_of.data(), sizeof(int64_t) * (size_t(m) + 1),
                                     cudaMemcpyHostToDevice, s));
            k_gather_sets<<<grid_for(nm, 256), 256, 0, s>>>(d_xyz, d_off, dlist.p, doff_of.p, m, nm, some.p);
            pts = some.p;
            off_of = doff_of.p;
        }
        D3G_TRY(spatial_order_sets_device(pts, hoff_of.data(), off_of, m, order.p, s));
        k_ranks<<<grid_for(nm, 256), 256, 0, s>>>(order.p, d_off, dlist.p, off_of, m, nm, rank.p);
        DevBuf<unsigned long long> best;
        D3G_TRY(best.alloc(size_t(n), s));
        D3G_CUDA(cudaMemsetAsync(best.p, 0, sizeof(unsigned long long) * size_t(n), s));
        k_best_copies<<<grid_for(n, 256), 256, 0, s>>>(idx.p, head.p, rank.p, d_off, nsets, n, best.p);
        k_head_flags<<<grid_for(n, 256), 256, 0, s>>>(head.p, n, idx2.p);
        D3G_TRY(exclusive_scan(idx2.p, idx2.p, n, s));
        D3G_TRY(O.vert.alloc(size_t(O.nv), s));
        D3G_TRY(O.rep.alloc(size_t(O.nv), s));
        k_compact_copies<<<grid_for(n, 256), 256, 0, s>>>(keys.p, idx.p, head.p, idx2.p, best.p, d_off, nsets, n,
                                                          O.vert.p, O.rep.p, keys2.p);
        k_level_starts<<<grid_for(O.nv + 1, 256), 256, 0, s>>>(keys2.p, O.nv, shift, level_bits, O.levels, total,
                                                               O.level_start.p);
    } else {
        O.vert.swap(idx);
    }
    D3G_CUDA(cudaGetLastError());
    O.keys.swap(hflags[0] > 0 ? keys2 : keys);
    O.curve_bits = shift;
    O.ok = true;
    return D3G_OK;
}

}  // namespace d3g
