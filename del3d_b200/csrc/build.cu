// The Delaunay build on the device: del3d::Delaunay::build
// (src/triangulation.cpp:65-120, 702-769, 932-968) as parallel insertion.
//
// Why a parallel build can return the reference's tets: in_sphere never
// returns ZERO (symbolic perturbation, src/predicates.cpp:206-232) and the hull
// conflict rule is fixed (src/triangulation.cpp:588-602), so the set of finite
// cells is a function of the point set alone, whatever the insertion order.
// The device therefore inserts many points at once.  By default the build's own
// order (order.cu) puts the points into levels that double what is in, the
// first levels of up to 148 sets are built in shared memory (k_coarse), and
// k_insert_groups inserts the others asynchronously under per-tet locks (see
// "asynchronous insertion" below and insert_groups.cuh).  What it cannot do goes
// through k_insert_full, and what that leaves through lockstep rounds, which
// schedule = 1 uses for every point:
//
//   * Points are grouped into levels, along a Hilbert curve in each; each level
//     is cut into chunks, one per worker.  A worker inserts its chunk's points
//     one per round, so the points in flight in a round are spread along the
//     curve, i.e. far apart.
//   * k_cavity   each worker walks from the last vertex it inserted to the tet
//                its point conflicts with (visibility walk, exact orient3d),
//                then grows the conflict region breadth-first with the
//                reference's in_conflict rule, claiming every region tet and
//                every tet across its boundary with a 64-bit atomicMin of
//                (round, point rank) - the earliest point in insertion order
//                wins ties.  A worker that meets a claim of an earlier point
//                stops at once: it would lose anyway.
//   * k_check    a worker wins if it still holds every claim.  Winners' regions
//                and their one-ring of outside tets are pairwise disjoint, so
//                winners can re-star concurrently without locks.
//   * k_restar   each winner re-stars its region (one new tet per boundary
//                facet, src/tds.h:160-221), reusing its region's slots, and
//                advances to its next point.  The earliest pending point always
//                wins, so every round makes progress.
//
// The output is canonicalised (even rotation, lexicographic sort), so it is
// identical across runs whatever order the rounds happened to take.
#include "build_api.cuh"

#include <cuda/atomic>
#include "device_util.cuh"
#include "order.cuh"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <numeric>
#include <optional>
#include <utility>
#include <vector>

namespace d3g {

int spatial_order_device(const double* d_xyz, int64_t n, int32_t* d_order, cudaStream_t s);
int spatial_order_sets_device(const double* d_xyz, const int64_t* h_off, const int64_t* d_off, int nsets,
                              int32_t* d_order, cudaStream_t s, double level_ratio = 0.125);
int multiscale_bounds(int64_t n, int64_t* b, int cap, double ratio = 0.125);

namespace {

constexpr int kInf = -1;
constexpr int kWalkLimit = 1 << 20;
constexpr int kRotateLimit = 1 << 16;
constexpr int kRoundsPerBatch = 16;
// Scratch of a worker in a normal round, and of each of the kBigSlots workers
// served at a time in a big round.
constexpr int kCavCap = 256;                     // boundary facets: twice the tets
constexpr int kBigSlots = 64, kBigCav = 16384;   // boundary facets: twice the tets

enum : int { WS_DONE = 0, WS_CAND = 1, WS_LOST = 2, WS_WIN = 3, WS_PARKED = 4, WS_FAIL = 5 };

/// Vertex v's coordinates.  A vertex takes 32 bytes (x, y, z and a pad): one
/// sector and one 256-bit load, where three packed doubles straddle two sectors
/// half of the time and take three loads.
__device__ __forceinline__ Pt vpt(const double* __restrict__ vx, int v) {
    double x, y, z, pad;
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(x), "=d"(y), "=d"(z), "=d"(pad)
        : "l"(vx + 4 * int64_t(v)));
    return Pt{x, y, z};
}

__device__ __forceinline__ int at(const int4& t, int i) {
    return i == 0 ? t.x : (i == 1 ? t.y : (i == 2 ? t.z : t.w));
}
__device__ __forceinline__ void set_at(int4& t, int i, int v) {
    if (i == 0) t.x = v;
    else if (i == 1) t.y = v;
    else if (i == 2) t.z = v;
    else t.w = v;
}
__device__ __forceinline__ int inf_pos(const int4& t) {
    return t.x == kInf ? 0 : (t.y == kInf ? 1 : (t.z == kInf ? 2 : (t.w == kInf ? 3 : -1)));
}
__device__ __forceinline__ int pos_of(const int4& t, int v) {
    return t.x == v ? 0 : (t.y == v ? 1 : (t.z == v ? 2 : 3));
}

struct Tables {
    int4* rec;                 // per tet 32 bytes, one sector: its vertices (kInf = the infinite
                               // vertex) and its neighbours (tet * 4 + the facet facing back);
                               // a slot without a live tet has its first two vertices equal
    unsigned long long* claim; // per-round ownership claims
    int* lock;                 // lock words of the asynchronous passes (null: lockstep rounds only)
    int* fnew;                 // per tet facet: the new tet built on it (restar scratch)
    int* vert_tet;             // one live tet incident to each inserted vertex
    int* tet_count;
    int cap;
    int walk_limit;            // steps of a lockstep walk before ST_WALK_LIMIT
    const int32_t* vset;       // the point set of each vertex (batched builds share the tables)
    __device__ int4& tv(int t) const { return rec[2 * int64_t(t)]; }
    __device__ int4& tn(int t) const { return rec[2 * int64_t(t) + 1]; }
    /// Neighbour entry `enc` (tet * 4 + facet).
    __device__ int& link(int enc) const { return reinterpret_cast<int*>(&tn(enc >> 2))[enc & 3]; }
    __device__ bool alive(int t) const { return tv(t).x != tv(t).y; }
    /// Ends tet t: all four vertices one of its own, so that a walk which still
    /// reads the slot stays in range.
    __device__ void kill(int t) const {
        const int x = max(tv(t).x, tv(t).y);   // at most one vertex is kInf
        tv(t) = make_int4(x, x, x, x);
    }
};

struct Workers {
    const int* list;  // big mode: the workers served (warp i serves list[i]); null otherwise
    int* parked;  // 1 while the worker's point needs the big scratch
    int* cur;     // current point (vertex id) of each worker
    int* beg;     // start of its chunk
    int* end;     // end of its chunk
    int* pos;     // next position to visit, relative to beg (chunks are walked cyclically)
    int* left;    // positions still to visit after the current point
    int* nwon;    // points this worker inserted in the current level
    int* last;    // last vertex it inserted (-1: none yet)
    int* guide;   // an inserted vertex near its chunk, for the first walk
    int* state;
    int* ncav;
    int* nfac;
    int* cav;     // worker-major scratch: cav_cap region tets per worker
    int* fac;     // fac_cap boundary facets (tet * 4 + facet) per worker
    int4* st_v;   // fac_cap staged new tets per worker (vertices) ...
    int4* st_n;   // ... and neighbours
    int* wset;        // set of each worker
    const int4* skips; // per set: its first tet's vertices (inserted before the rounds)
    const uint8_t* set_exact;  // per set: EX_*, what its coordinates make exact
    int cav_cap;
    int fac_cap;
    int n;
};

struct Round {
    const unsigned* round;    // current round number (device), set by k_round_begin
    int* counters;            // [0] active workers, [1] parked workers, [2] winners,
                              // [3] workers parked this round
    unsigned long long* sums; // [0] region tets, [1] boundary facets of the winners
    unsigned long long* totals; // [0] winners, [1] attempts, [2] rounds with work,
                                // [3] parked workers, [4] stalled round seen, [5] active
    unsigned long long* steps;  // timing runs only (else null): [0] walk steps,
                                // [1] breadth-first steps, over all attempts
    uint32_t* status;
    unsigned long long* pstats; // [0] conflict tests, [1] of which the filter left uncertain,
                                // [2] of which exactly degenerate (tie-break), [3] largest
                                // conflict region inserted (tets)
};

/// A thread's conflict-test counters, added to Round::pstats once at the end
/// of a launch (flush_counters).  `flags` holds the uncertain count in its low half
/// and the tie count above.  The insertion kernels keep them in shared memory, one
/// slot per thread, so that they take no registers from the loops they count in -
/// and no more than 15 bytes a thread: with 16, five blocks of k_insert_groups<8, ...>
/// take more than 196 KB, and L1 shrinks from 60 to 28 KB (10^7 uniform points 102 ->
/// 108 ms).
constexpr int kCounterThreads = 128;   // the insertion kernels' block size

struct SharedCounters {
    unsigned* tests;
    unsigned long long* flags;
    uint16_t* max_region;   // (regions hold kBigCapacity tets at most here)
    __device__ void count(int r) const {
        tests[threadIdx.x] += 1;
        flags[threadIdx.x] += (unsigned long long)(unsigned((r >> 2) & 1)) << 32 | unsigned((r >> 1) & 1);
    }
    __device__ void region(int c) const { max_region[threadIdx.x] = uint16_t(max(int(max_region[threadIdx.x]), c)); }
    __device__ void clear() const {
        tests[threadIdx.x] = 0;
        flags[threadIdx.x] = 0;
        max_region[threadIdx.x] = 0;
    }
};

#define D3G_SHARED_COUNTERS(name)                                \
    __shared__ unsigned name##_t[kCounterThreads];               \
    __shared__ unsigned long long name##_f[kCounterThreads];     \
    __shared__ uint16_t name##_m[kCounterThreads];               \
    const SharedCounters name{name##_t, name##_f, name##_m};     \
    name.clear()

/// Sums the warp's counters into R.pstats (one atomic per counter per warp).
__device__ void flush_counters(const SharedCounters& c, const Round& R) {
    unsigned long long t = c.tests[threadIdx.x], u = c.flags[threadIdx.x] & 0xFFFFFFFFu,
                       z = c.flags[threadIdx.x] >> 32;
    int m = c.max_region[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        t += __shfl_xor_sync(0xffffffffu, t, o);
        u += __shfl_xor_sync(0xffffffffu, u, o);
        z += __shfl_xor_sync(0xffffffffu, z, o);
        m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    }
    if ((threadIdx.x & 31) == 0) {
        if (t) atomicAdd(R.pstats, t);
        if (u) atomicAdd(R.pstats + 1, u);
        if (z) atomicAdd(R.pstats + 2, z);
        if (m) atomicMax(R.pstats + 3, (unsigned long long)m);
    }
}

/// Claim key of point v this round: (~round) << 32 makes every newer round win
/// against stale claims; the point rank breaks ties (earliest wins).
__device__ __forceinline__ unsigned long long claim_key(const Round& R, int v) {
    return ((unsigned long long)(0xFFFFFFFFu - *R.round) << 32) |
           (unsigned long long)(uint32_t(v)) << 1;
}

__global__ void k_round_begin(Round R) {
    unsigned* r = const_cast<unsigned*>(R.round);
    *r += 1;
    R.counters[0] = R.counters[1] = R.counters[2] = R.counters[3] = 0;
}

/// Folds one round's counters into the running totals; flags a round in which
/// workers were active but nobody won (the earliest pending point must win).
__global__ void k_round_end(Round R) {
    const int active = R.counters[0], parked = R.counters[1], won = R.counters[2];
    R.totals[0] += (unsigned long long)won;
    R.totals[1] += (unsigned long long)(active + won);
    if (active + won > 0) R.totals[2] += 1;
    R.totals[3] = (unsigned long long)parked;
    // A worker parked this round may have claimed tets of every other candidate.
    if (active > 0 && won == 0 && R.counters[3] == 0) R.totals[4] = 1;
    R.totals[5] = (unsigned long long)active;
}

/// orient3d of tet (q0,q1,q2,q3) with vertex i replaced by p (one call site);
/// `ex`: the set's coordinates make the filter exact.
__device__ __forceinline__ int orient_replaced(const Pt* q, int i, const Pt& p, bool ex, uint32_t* st) {
    const Pt& A = i == 0 ? p : q[0];
    const Pt& B = i == 1 ? p : q[1];
    const Pt& C = i == 2 ? p : q[2];
    const Pt& D = i == 3 ? p : q[3];
    return orient3d_x(A, B, C, D, ex, st);
}

/// Whether the normal that in_circle_filter computes for facet (a, b, d) points to
/// the right side of its plane.  The filter's value is that of in_sphere with the
/// facet's vertices and the point p + normal, so its sign hangs on that side, but its
/// bound is relative to the normal's rounded length: on a facet whose vertices are
/// collinear but for rounding it can certify the wrong sign.  Each component is off by
/// at most 4 eps of the sum of its two products' sizes (8 here).
__device__ __forceinline__ bool normal_certain(const Pt& a, const Pt& b, const Pt& d) {
    const double px = fsub(b.x, a.x), py = fsub(b.y, a.y), pz = fsub(b.z, a.z);
    const double qx = fsub(d.x, a.x), qy = fsub(d.y, a.y), qz = fsub(d.z, a.z);
    const double x0 = fmul(py, qz), x1 = fmul(pz, qy), y0 = fmul(pz, qx), y1 = fmul(px, qz), z0 = fmul(px, qy),
                 z1 = fmul(py, qx);
    const double longest = fmax(fmax(fabs_(fsub(x0, x1)), fabs_(fsub(y0, y1))), fabs_(fsub(z0, z1)));
    const double sizes = fadd(fadd(fadd(fabs_(x0), fabs_(x1)), fadd(fabs_(y0), fabs_(y1))), fadd(fabs_(z0), fabs_(z1)));
    return longest > fmul(8.0 * kEps, sizes);
}

/// coplanar_in_circle for the hull case of the conflict test (rare: the point
/// lies in the plane of a hull facet), out of line so that its code stays out
/// of the hot path's instruction stream.  It is coplanar_in_circle except on facets
/// without a certain normal, which go to the exact stage where that reaches: the
/// reference takes the filter's sign there (src/predicates2.cpp:182-231), and in an
/// unlucky order of insertions a wrong one gives a region that is no ball, or other
/// cells.
__device__ __noinline__ int hull_in_circle(double ax, double ay, double az, double bx, double by, double bz,
                                           double dx, double dy, double dz, double px, double py, double pz,
                                           int ia, int ib, int id_, int ip, uint32_t* st) {
    const Pt a{ax, ay, az}, b{bx, by, bz}, d{dx, dy, dz}, p{px, py, pz};
    const InCircleFilter f = in_circle_filter(a, b, d, p);
    if (f.certain) {
        bool use = normal_certain(a, b, d);
        if (!use) {
            Span s;
            s.add(ax); s.add(ay); s.add(az); s.add(bx); s.add(by); s.add(bz);
            s.add(dx); s.add(dy); s.add(dz); s.add(px); s.add(py); s.add(pz);
            use = limbs_for(7 * (s.bits() + 1) + 9) > kMaxLimbs;
        }
        if (use) return sign_of(f.det);
    }
    return in_circle_degenerate(ax, ay, az, bx, by, bz, dx, dy, dz, px, py, pz, ia, ib, id_, ip, f.det, 1, st);
}

/// Outcome bits of a conflict test: in conflict; the floating-point filter
/// could not certify the sign (the set's exact filter value, the exact stage or
/// a tie-break decided it); the exact value was zero (decided by the symbolic
/// perturbation, or the hull in-circle test); and, from in_conflict_fast only,
/// undecided (the exact stage is needed).
enum : int { CT_IN = 1, CT_UNCERTAIN = 2, CT_TIE = 4, CT_UNDECIDED = 8 };

/// What a set's coordinates make exact (k_set_exact).
enum : int { EX_ORIENT = 1, EX_SPHERE = 2, EX_BOTH = 3, EX_GRID = 4 };

/// in_sphere's exact sign for a set whose filter is not exact and, when it is
/// zero, the reference's tie-break (src/predicates.cpp:206-232): the sign, plus
/// 4 if the tie-break gave it.  Out of line.
__device__ __noinline__ int in_sphere_exact_tie(double ax, double ay, double az, double bx, double by, double bz,
                                                double cx, double cy, double cz, double dx, double dy, double dz,
                                                double ex, double ey, double ez, int id0, int id1, int id2, int id3,
                                                int id4, double fdet, uint32_t* st) {
    const int s = in_sphere_degenerate(ax, ay, az, bx, by, bz, cx, cy, cz, dx, dy, dz, ex, ey, ez, id0, id1, id2, id3,
                                       id4, fdet, 0, st);
    if (s != 0) return s;
    return 4 + in_sphere_perturb(Pt{ax, ay, az}, Pt{bx, by, bz}, Pt{cx, cy, cz}, Pt{dx, dy, dz}, Pt{ex, ey, ez},
                                 id0, id1, id2, id3, id4, st);
}

/// The reference's conflict test, src/triangulation.cpp:588-602, with its
/// outcome bits (CT_*).  `ex`: the point set's coordinates span few enough bits
/// that the orient3d and in_sphere filters compute their determinants exactly.
__device__ int conflict_test(const int4 t, const Pt& p, int pid, const double* __restrict__ vx, bool ex,
                             uint32_t* st) {
    const int ip = inf_pos(t);
    if (ip >= 0) {
        // For each slot of the infinite vertex, the three finite vertices in
        // the order that makes orient3d(a, b, d, p) the half-space test.
        const int o0 = ip == 0 ? 2 : (ip == 1 ? 2 : (ip == 2 ? 1 : 0));
        const int o1 = ip == 0 ? 1 : (ip == 1 ? 3 : (ip == 2 ? 0 : 1));
        const int o2 = ip == 0 ? 3 : (ip == 1 ? 0 : (ip == 2 ? 3 : 2));
        const int va = at(t, o0), vb = at(t, o1), vd = at(t, o2);
        const Pt a = vpt(vx, va), b = vpt(vx, vb), d = vpt(vx, vd);
        const Orient3dFilter f = orient3d_filter(a, b, d, p);
        const int unc = f.certain ? 0 : CT_UNCERTAIN;
        const int s = (f.certain || ex) ? -sign_of(f.det) : orient3d_exact(a, b, d, p, f.det, st);
        if (s != 0) return (s > 0 ? CT_IN : 0) | unc;
        return (hull_in_circle(a.x, a.y, a.z, b.x, b.y, b.z, d.x, d.y, d.z, p.x, p.y, p.z, va, vb, vd, pid, st) > 0
                    ? CT_IN : 0) | unc | CT_TIE;
    }
    const Pt a = vpt(vx, t.x), b = vpt(vx, t.y), c = vpt(vx, t.z), d = vpt(vx, t.w);
    const InSphereFilter f = in_sphere_filter(a, b, c, d, p);
    if (f.certain) return f.det < 0.0 ? CT_IN : 0;   // in_sphere = -sign(det)
    if (ex && f.det != 0.0) return (f.det < 0.0 ? CT_IN : 0) | CT_UNCERTAIN;
    if (ex)
        return (in_sphere_tiebreak_exact(a.x, a.y, a.z, b.x, b.y, b.z, c.x, c.y, c.z, d.x, d.y, d.z, p.x, p.y, p.z,
                                         t.x, t.y, t.z, t.w, pid, st) > 0 ? CT_IN : 0) | CT_UNCERTAIN | CT_TIE;
    const int r = in_sphere_exact_tie(a.x, a.y, a.z, b.x, b.y, b.z, c.x, c.y, c.z, d.x, d.y, d.z, p.x, p.y, p.z, t.x,
                                      t.y, t.z, t.w, pid, f.det, st);
    const bool tie = r > 1;
    return ((tie ? r - 4 : r) > 0 ? CT_IN : 0) | CT_UNCERTAIN | (tie ? CT_TIE : 0);
}

/// conflict_test out of line: for the once-per-insertion seed check of k_insert_full
/// (one inline copy, in the breadth-first growth, is enough) and for the tests that
/// the filters of k_insert_groups leave undecided.
__device__ __noinline__ int conflict_test_exact(int4 t, double px, double py, double pz, int pid,
                                               const double* __restrict__ vx, bool ex, uint32_t* st) {
    return conflict_test(t, Pt{px, py, pz}, pid, vx, ex, st);
}

constexpr unsigned kFull = 0xffffffffu;

/// Advances worker w to the next point of its chunk (walked cyclically),
/// skipping its set's first-tet vertices; -1 when the chunk is done.
__device__ int next_point(const Workers& W, int w) {
    const int b = W.beg[w], len = W.end[w] - b;
    const int4 sk = W.skips[W.wset[w]];
    int pos = W.pos[w], left = W.left[w];
    int v = -1;
    while (left > 0) {
        const int c = b + pos;
        pos = pos + 1 == len ? 0 : pos + 1;
        --left;
        if (c != sk.x && c != sk.y && c != sk.z && c != sk.w) {
            v = c;
            break;
        }
    }
    W.pos[w] = pos;
    W.left[w] = left;
    W.cur[w] = v;
    return v;
}

// ---- the insertion kernels ---------------------------------------------------
//
// A worker is served by a group of G lanes (G = 32, 16, 8 or 4), so one warp
// serves 32 / G workers side by side.  Few workers: G = 32 shortens each
// worker's chain of dependent memory accesses (8 region tets per step).  Many
// workers (more than the GPU keeps resident as warps): a small G packs them into
// fewer warps, so the whole round fits the resident warps and its time is one
// chain instead of several waves of chains.  Control flow stays uniform over
// the warp - every loop runs until all of its groups are done - so the groups'
// memory accesses are issued together and warp votes cover all 32 lanes; a
// group reads its own bits of each vote.

template <int G>
struct Lanes {
    int lane, sub, gbase;
    unsigned gm;   // the group's bits in a warp-wide vote
    __device__ Lanes() {
        lane = threadIdx.x & 31;
        sub = lane & (G - 1);
        gbase = lane - sub;
        gm = G == 32 ? kFull : (((1u << G) - 1u) << gbase);
    }
    /// The group's bits of a warp-wide vote, lane 0 of the group at bit 0.
    __device__ unsigned own(unsigned vote) const { return G == 32 ? vote : (vote & gm) >> gbase; }
};

/// Visibility walk from each live group's start tet to a tet in conflict with
/// its point p: the finite tet containing p, or the infinite tet beyond the hull
/// facet the walk crosses.  Lanes 0-3 of a group test the four facets of a step;
/// the first negative one in a pseudo-random cyclic order is crossed (never the
/// facet just crossed).  Returns the tet (same in every lane of the group), or
/// -1 for a group that is not live or hit the walk limit.
template <int G>
__device__ int walk_g(bool live, int t, const Pt& p, int pid, const Tables& T, const double* __restrict__ vx,
                      bool ex, uint32_t* st, const Lanes<G>& L, int* nsteps) {
    int4 tv = make_int4(0, 0, 0, 0);
    if (live) {
        tv = T.tv(t);
        const int ip = inf_pos(tv);
        if (ip >= 0) {
            t = at(T.tn(t), ip) >> 2;
            tv = T.tv(t);
        }
    }
    int prev = -1, found = -1;
    uint32_t h = uint32_t(pid) * 2654435761u + 12345u;
    bool walking = live;
    for (int step = 0; __any_sync(kFull, walking); ++step) {
        int4 tn = make_int4(0, 0, 0, 0);
        bool neg = false;
        if (walking) {
            tn = T.tn(t);
            h = h * 1664525u + 1013904223u;
            if (L.sub < 4 && (at(tn, L.sub) >> 2) != prev) {
                const Pt q[4] = {vpt(vx, tv.x), vpt(vx, tv.y), vpt(vx, tv.z), vpt(vx, tv.w)};
                neg = orient_replaced(q, L.sub, p, ex, st) < 0;
            }
        }
        const unsigned m = L.own(__ballot_sync(kFull, neg)) & 0xFu;
        if (walking) {
            *nsteps = step + 1;
            if (m == 0) {
                found = t;
                walking = false;
            } else {
                const int s0 = int(h >> 30);
                const unsigned rot = ((m >> s0) | (m << (4 - s0))) & 0xFu;
                const int i = (s0 + __ffs(int(rot)) - 1) & 3;
                const int next = at(tn, i) >> 2;
                const int4 nv = T.tv(next);
                if (inf_pos(nv) >= 0) {
                    found = next;
                    walking = false;
                } else {
                    prev = t;
                    t = next;
                    tv = nv;
                    if (step + 1 >= T.walk_limit) {
                        report(st, ST_WALK_LIMIT);
                        walking = false;
                    }
                }
            }
        }
    }
    return found;
}

/// One group of G lanes per worker: locate the worker's point, then grow its
/// conflict region breadth-first, G/4 region tets (G facets) per step, claiming
/// every region tet (key) and every tet across the region boundary (key|1).
template <int G>
__global__ void __launch_bounds__(128, 8) k_cavity(Tables T, Workers W, Round R, const double* __restrict__ vx,
                                                int first) {
    const Lanes<G> L;
    D3G_SHARED_COUNTERS(ctr);
    const int slot = first + int((blockIdx.x * blockDim.x + threadIdx.x) / G);
    bool live = slot < W.n;
    int w = 0, v = -1;
    if (live) {
        w = W.list ? W.list[slot] : slot;
        v = W.cur[w];
        // Normal rounds leave parked workers alone; big rounds serve only those.
        if (v < 0 || (W.parked[w] != 0) != (W.list != nullptr)) {
            if (L.sub == 0) W.state[w] = v < 0 ? WS_DONE : WS_PARKED;
            live = false;
        }
    }
    if (!__any_sync(kFull, live)) return;
    const Pt p = live ? vpt(vx, v) : Pt{0.0, 0.0, 0.0};
    const bool ex = live && (W.set_exact[W.wset[w]] & EX_BOTH) == EX_BOTH;
    int start = 0;
    if (live) start = T.vert_tet[W.last[w] >= 0 ? W.last[w] : W.guide[w]];
    int wsteps = 0;
    const int seed = walk_g<G>(live, start, p, v, T, vx, ex, R.status, L, &wsteps);
    if (R.steps && live && L.sub == 0) atomicAdd(R.steps, (unsigned long long)wsteps);
    if (live && seed < 0) {
        if (L.sub == 0) W.state[w] = WS_FAIL;
        live = false;
    }
    const unsigned long long key = live ? claim_key(R, v) : 0ull;
    const unsigned long long mine = key >> 1;
    int* cav = W.cav + int64_t(live ? slot : 0) * W.cav_cap;
    int* fac = W.fac + int64_t(live ? slot : 0) * W.fac_cap;
    int lost = 0;
    if (live && L.sub == 0) {
        const unsigned long long old = atomicMin(T.claim + seed, key);
        lost = (old >> 1) < mine;
        cav[0] = seed;
    }
    lost = __shfl_sync(kFull, lost, L.gbase);
    if (live && lost) {
        if (L.sub == 0) W.state[w] = WS_LOST;
        live = false;
    }
    __syncwarp();
    const unsigned lt = (1u << L.lane) - 1u;
    int ncav = 1, nfac = 0, head = 0;
    bool growing = live;
    while (__any_sync(kFull, growing)) {
        if (R.steps && growing && L.sub == 0) atomicAdd(R.steps + 1, 1ull);
        const int nproc = growing ? min(ncav - head, G / 4) : 0;
        const bool valid = (L.sub >> 2) < nproc;
        const int i = L.sub & 3;
        int c = 0, nb = 0;
        int kind = 0;   // 0: nothing, 1: boundary facet, 2: new region tet, 3: re-check
        bool abort = false;
        if (valid) {
            c = cav[head + (L.sub >> 2)];
            nb = at(T.tn(c), i) >> 2;
            const unsigned long long old = atomicMin(T.claim + nb, key | 1ull);
            if (old == key) {
                kind = 0;                               // already in the region
            } else if (old == (key | 1ull)) {
                kind = 3;                               // seen by us: decided below
            } else if ((old >> 1) < mine) {
                abort = true;                           // an earlier point holds it
            } else {
                const int r = conflict_test(T.tv(nb), p, v, vx, ex, R.status);
                ctr.count(r);
                if (r & CT_IN) {
                    const unsigned long long o2 = atomicMin(T.claim + nb, key);
                    if ((o2 >> 1) < mine) abort = true;
                    else kind = 2;
                } else {
                    kind = 1;
                }
            }
        }
        const unsigned ab0 = L.own(__ballot_sync(kFull, abort));
        if (growing && ab0) {
            if (L.sub == 0) W.state[w] = WS_LOST;
            growing = false;
        }
        __syncwarp();
        if (growing && kind == 3) {
            // Another lane of this step may have just turned it into a region tet.
            const unsigned long long now = __ldcg(T.claim + nb);
            if (now == key) kind = 0;
            else if ((now >> 1) < mine) abort = true;
            else kind = 1;
        }
        const unsigned ab = L.own(__ballot_sync(kFull, growing && abort));
        if (growing && ab) {
            if (L.sub == 0) W.state[w] = WS_LOST;
            growing = false;
        }
        const unsigned mc = __ballot_sync(kFull, growing && kind == 2) & L.gm;
        const unsigned mf = __ballot_sync(kFull, growing && kind == 1) & L.gm;
        if (growing && (ncav + __popc(mc) > W.cav_cap || nfac + __popc(mf) > W.fac_cap)) {
            if (L.sub == 0) {
                // Too big for this scratch: park the worker until a big round
                // (or, in a big round, report that even that was not enough).
                W.state[w] = WS_PARKED;
                if (W.list) report(R.status, ST_CAVITY_CAPACITY);
                else W.parked[w] = 1;
                atomicAdd(R.counters + 3, 1);   // its claims may have blocked others
            }
            growing = false;
        }
        if (growing) {
            if (kind == 2) cav[ncav + __popc(mc & lt)] = nb;
            if (kind == 1) fac[nfac + __popc(mf & lt)] = c * 4 + i;
            ncav += __popc(mc);
            nfac += __popc(mf);
            head += nproc;
            if (head >= ncav) {
                if (L.sub == 0) {
                    W.ncav[w] = ncav;
                    W.nfac[w] = nfac;
                    W.state[w] = WS_CAND;
                }
                growing = false;
            }
        }
        __syncwarp();
    }
    flush_counters(ctr, R);
}

/// One group per candidate: it wins if it still holds every claim it made.
template <int G>
__global__ void __launch_bounds__(128, 8) k_check(Tables T, Workers W, Round R, int first) {
    const Lanes<G> L;
    const int slot = first + int((blockIdx.x * blockDim.x + threadIdx.x) / G);
    bool live = slot < W.n;
    int w = 0;
    if (live) {
        w = W.list ? W.list[slot] : slot;
        live = W.state[w] == WS_CAND;
    }
    if (!__any_sync(kFull, live)) return;
    bool ok = true;
    if (live) {
        const int v = W.cur[w];
        const unsigned long long key = claim_key(R, v);
        const int* cav = W.cav + int64_t(slot) * W.cav_cap;
        const int* fac = W.fac + int64_t(slot) * W.fac_cap;
        const int ncav = W.ncav[w], nfac = W.nfac[w];
        for (int k = L.sub; k < ncav; k += G) ok = ok && T.claim[cav[k]] == key;
        for (int k = L.sub; k < nfac; k += G) {
            const int f = fac[k];
            ok = ok && T.claim[at(T.tn(f >> 2), f & 3) >> 2] == (key | 1ull);
        }
    }
    const bool win = L.own(__ballot_sync(kFull, !ok)) == 0;
    if (live && L.sub == 0) {
        W.state[w] = win ? WS_WIN : WS_LOST;
        if (win) atomicMax(R.pstats + 3, (unsigned long long)W.ncav[w]);
    }
}

/// Neighbour of new tet facet j (the new tet replaces facet i of region tet c):
/// facet j is {v} + edge (va, vb), and its neighbour is the new tet on the other
/// boundary facet through that edge, reached by turning around the edge inside
/// the region (reference src/tds.h:160-221).  Returns the encoded neighbour
/// (tet * 4 + facet), or -1 if the region is inconsistent.
__device__ int restar_neighbour(const Tables& T, int c, const int4& cv, int i, int j,
                                unsigned long long key) {
    int a = -1, b = -1;
    for (int m = 0; m < 4; ++m)
        if (m != i && m != j) {
            if (a < 0) a = m;
            else b = m;
        }
    const int va = at(cv, a), vb = at(cv, b);
    int cur = c, f = j, steps = 0;
    for (;;) {
        const int enc = at(T.tn(cur), f);
        const int nb = enc >> 2;
        if (T.claim[nb] != key) {   // (cur, f) is a boundary facet
            const int4 tc = T.tv(cur);
            const int wpos = 6 - f - pos_of(tc, va) - pos_of(tc, vb);
            if (wpos < 0 || wpos > 3 || wpos == f) return -1;
            return T.fnew[cur * 4 + f] * 4 + wpos;
        }
        const int4 tb = T.tv(nb);
        const int g = enc & 3;
        f = 6 - g - pos_of(tb, va) - pos_of(tb, vb);
        cur = nb;
        if (f < 0 || f > 3 || f == g || ++steps > kRotateLimit) return -1;
    }
}

/// One group per winner: re-star its region, one boundary facet per lane.
template <int G>
__global__ void __launch_bounds__(128, 8) k_restar(Tables T, Workers W, Round R, int first) {
    __shared__ int sh_count[3];
    const Lanes<G> L;
    const int slot = first + int((blockIdx.x * blockDim.x + threadIdx.x) / G);
    if (threadIdx.x < 3) sh_count[threadIdx.x] = 0;
    __syncthreads();
    const bool exists = slot < W.n;
    const int w = exists ? (W.list ? W.list[slot] : slot) : 0;
    const int state = exists ? W.state[w] : WS_DONE;
    const int v = exists ? W.cur[w] : -1;
    const bool winner = state == WS_WIN;
    bool advanced = false;
    if (__any_sync(kFull, winner)) {
        const unsigned long long key = winner ? claim_key(R, v) : 0ull;
        const int64_t sl = winner ? slot : 0;
        const int* cav = W.cav + sl * W.cav_cap;
        const int* fac = W.fac + sl * W.fac_cap;
        int4* sv = W.st_v + sl * W.fac_cap;
        int4* sn = W.st_n + sl * W.fac_cap;
        const int C = winner ? W.ncav[w] : 0, F = winner ? W.nfac[w] : 0;
        const int extra = F > C ? F - C : 0;
        int base = 0, ok = winner ? 1 : 0;
        if (winner && L.sub == 0 && extra > 0) {
            base = atomicAdd(T.tet_count, extra);
            if (base + extra > T.cap) {
                report(R.status, ST_TET_CAPACITY);
                ok = 0;
            }
        }
        base = __shfl_sync(kFull, base, L.gbase);
        ok = __shfl_sync(kFull, ok, L.gbase);
        // 1a: the new tet of each boundary facet.
        if (ok)
            for (int k = L.sub; k < F; k += G) T.fnew[fac[k]] = k < C ? cav[k] : base + (k - C);
        __syncwarp();
        // 1b: vertices and neighbours, from the region as it was.
        bool bad = false;
        for (int k0 = 0; __any_sync(kFull, ok && k0 < F); k0 += G) {
            const int k = k0 + L.sub;
            if (ok && k < F) {
                const int c = fac[k] >> 2, i = fac[k] & 3;
                const int4 cv = T.tv(c);
                const int4 cn = T.tn(c);
                int4 nv = cv, nn = cn;
                set_at(nv, i, v);
                for (int j = 0; j < 4 && !bad; ++j) {
                    if (j == i) continue;
                    const int e = restar_neighbour(T, c, cv, i, j, key);
                    if (e < 0) bad = true;
                    else set_at(nn, j, e);
                }
                sv[k] = nv;
                sn[k] = nn;
            }
        }
        if (L.own(__ballot_sync(kFull, bad))) {
            if (L.sub == 0) report(R.status, ST_INTERNAL);
            ok = 0;
        }
        __syncwarp();
        if (ok) {
            // 2: write the new tets and re-point the outside neighbours.
            for (int k = L.sub; k < F; k += G) {
                const int id = k < C ? cav[k] : base + (k - C);
                const int4 nv = sv[k], nn = sn[k];
                const int i = fac[k] & 3;
                T.tv(id) = nv;
                T.tn(id) = nn;
                if (T.lock && k >= C) T.lock[id] = 0;   // the slot's first tet
                const int enc = at(nn, i);
                T.link(enc) = id * 4 + i;
                if (nv.x != kInf) T.vert_tet[nv.x] = id;
                if (nv.y != kInf) T.vert_tet[nv.y] = id;
                if (nv.z != kInf) T.vert_tet[nv.z] = id;
                if (nv.w != kInf) T.vert_tet[nv.w] = id;
            }
            for (int k = F + L.sub; k < C; k += G) T.kill(cav[k]);
            advanced = true;
            if (L.sub == 0) {
                atomicAdd(R.sums, (unsigned long long)C);
                atomicAdd(R.sums + 1, (unsigned long long)F);
            }
        }
    }
    if (L.sub == 0 && exists) {
        int cur = v;
        if (advanced) {
            W.last[w] = v;
            W.parked[w] = 0;
            W.nwon[w] += 1;
            cur = next_point(W, w);
        }
        if (cur >= 0 && W.parked[w]) atomicAdd(sh_count + 1, 1);     // waits for a big round
        else if (state != WS_DONE && cur >= 0) atomicAdd(sh_count, 1);
        if (advanced) atomicAdd(sh_count + 2, 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (sh_count[0]) atomicAdd(R.counters, sh_count[0]);
        if (sh_count[1]) atomicAdd(R.counters + 1, sh_count[1]);
        if (sh_count[2]) atomicAdd(R.counters + 2, sh_count[2]);
    }
}

// ---- asynchronous insertion --------------------------------------------------
//
// The rounds above insert in lockstep: every round waits for its slowest
// worker.  k_insert_groups (insert_groups.cuh) and k_insert_full below let every
// group of lanes, or warp, run at its own pace instead.  A persistent grid takes
// the level's points from a queue.  An insertion try-locks every tet it reads
// to decide its conflict region - the region tets and the tets across the
// region boundary - and holds the locks until its new tets are written, so
// insertions whose locks succeed touch disjoint tets and commute: the result
// is that of some sequential order, hence (the tet set does not depend on the
// insertion order) the canonical set.  A lock held by another insertion makes
// this one give back its locks and try again after a back-off; after some
// failures, and for a conflict region too large for its scratch, the point is
// left for a later pass, which finishes it.  The only wait for a lock while
// others are held is that of the widest groups, which poll a lock of a lower
// priority kWaitPolls times and then give way; every loop is bounded.
//
// Lock word of a tet: 0 free, -1 a slot no tet has been written to yet, else
// (owner << 1) | ring, owner = group or warp slot + 1; ring = 1 for a tet
// across the region boundary, 0 for a region tet.  Locks are taken with acquire
// ordering; after the tets are written they are released by a warp barrier, then
// a fence in every lane, then plain stores (k_insert_groups), or by a barrier and
// compare-and-swaps with release ordering (k_insert_full).  Every read of tet
// data that other warps write goes to L2 (__ldcg), not the SM's L1.

constexpr int kAsyncRetries = 6;
// Passes of k_insert_full over the points left to it before the rounds.
constexpr int kLeftPasses = 8;
// Level growth of a build by lockstep rounds alone, when a set's filters are
// exact or the whole build has fewer than kSmallBuildPoints points (else 8).
constexpr int kExactSetGrowth = 4;
constexpr int64_t kSmallBuildPoints = 65536;
constexpr int kAsyncWalkLimit = 1 << 14;
// BRIO level growth of an asynchronous build's own order: a level's depth is
// (growth - 1) * alpha insertions in a row while the GPU is not full, so short
// levels have the least depth per point.
constexpr int kGroupGrowth = 2;
// Passes of k_insert_groups over what the last level left.
constexpr int kLastPasses = 3;
// Passes with the exact stage over the points with undecided tests that are left
// after the last level.
constexpr int kExactPasses = 3;
// Each level is followed by a look at how many points with undecided tests wait; from
// the first that finds more than one in kUndecidedShare of the points so far, every
// level is followed by a pass with the exact stage.  (Fewer wait for the end.)  A point
// that is not in makes the regions of those after it larger, and a test that one point
// cannot decide is met by the next ones near it: with passes from the level of 4096
// points on, a set with half of its 300000 points in one corner of 2^-30 of its
// extent took 990 ms, without any 11 s.
constexpr int kUndecidedShare = 128;
// Groups with room for kBigCapacity, and points the last pass of a single one takes at
// most.
constexpr int kBigGroups = 16;
constexpr int kLonePoints = 256;
// Vertices of the level before, to either side along the curve, among which a
// vertex's guide is the nearest.
constexpr int kGuideReach = 4;
// The neighbour records of a warp's first kHandedTn region tets, read under
// their locks together with their vertices, are kept in shared memory for the
// growth step that expands them (instead of being read from L2 again there).
constexpr int kHandedTn = 64;

struct AsyncCtx {
    int* lock;                      // per tet lock word
    int* next;                      // chunk queue head
    int* leftover;                  // points left for the rounds
    int* n_leftover;
    int64_t stride;                 // entry q of the queue is worker (q * stride) % nw
    int nw;
    unsigned long long* ekey;       // per warp slot: 3 edge keys per boundary facet (re-star)
    unsigned long long* stats;      // [0] lock conflicts, [1] walk restarts, [2] invalid seeds,
                                    // [3] regions too big, [4] points left,
                                    // [5] points with a test the filters could not decide
};

using LockRef = cuda::atomic_ref<int, cuda::thread_scope_device>;

__device__ __forceinline__ bool try_lock(int* lock, int t, int value, int* seen) {
    int expected = 0;
    const bool ok = LockRef(lock[t]).compare_exchange_strong(expected, value, cuda::memory_order_acquire,
                                                             cuda::memory_order_relaxed);
    *seen = ok ? 0 : expected;
    return ok;
}

/// Releases tet t if `value` still holds it (a ring tet may be listed twice).
__device__ __forceinline__ void unlock_if(int* lock, int t, int value) {
    int expected = value;
    LockRef(lock[t]).compare_exchange_strong(expected, 0, cuda::memory_order_release, cuda::memory_order_relaxed);
}

__device__ __forceinline__ int4 ld4(const int4* p) { return __ldcg(p); }

/// orient3d of tet `t` with vertex i replaced by p, from the filter alone: the
/// sign when the filter decides it (or `ex`: the set's coordinates make the
/// filter's value exact), else 2.  An even permutation of that call puts p last,
/// so only the facet's three vertices are read; choosing them by index costs a few
/// selects where choosing among four points' coordinates costs 24.
template <class M>
__device__ __forceinline__ int orient_facet_filter(const M& m, const int4& t, int i, const Pt& p, bool ex) {
    const int x = i == 0 ? t.z : (i == 2 ? t.y : t.x);
    const int y = i == 0 ? t.y : (i == 1 ? t.z : (i == 2 ? t.x : t.y));
    const int z = i == 3 ? t.z : t.w;
    const Orient3dFilter f = orient3d_filter(m.point(x), m.point(y), m.point(z), p);
    if (f.certain || ex) return -sign_of(f.det);
    return 2;
}

/// Visibility walk on a mesh other warps are changing: reads go to L2 and may
/// be stale, so the tet it returns is only a candidate, checked under its lock.
/// Returns -1 after kAsyncWalkLimit steps (or the build's walk limit, if lower).
__device__ int walk_async(int t, const Pt& p, int pid, const Tables& T, const double* __restrict__ vx,
                          bool ex, uint32_t* st, int lane) {
    int4 tv = ld4(&T.tv(t));
    {
        const int ip = inf_pos(tv);
        if (ip >= 0) {
            t = at(ld4(&T.tn(t)), ip) >> 2;
            tv = ld4(&T.tv(t));
        }
    }
    int4 tn = ld4(&T.tn(t));
    int prev = -1;
    uint32_t h = uint32_t(pid) * 2654435761u + 12345u;
    const int limit = min(kAsyncWalkLimit, T.walk_limit);
    for (int step = 0; step < limit; ++step) {
        // While lanes 0-3 test the four facets, lanes 4-7 fetch the four
        // neighbours' vertices and lanes 8-11 their neighbours: the step to
        // the chosen neighbour then waits for no further memory read.
        int4 pre = make_int4(0, 0, 0, 0);
        if (lane >= 4 && lane < 12) {
            const int nbr = at(tn, lane & 3) >> 2;
            pre = lane < 8 ? ld4(&T.tv(nbr)) : ld4(&T.tn(nbr));
        }
        h = h * 1664525u + 1013904223u;
        const int s0 = int(h >> 30);
        bool neg = false;
        if (lane < 4 && (at(tn, lane) >> 2) != prev && tv.x != kInf && tv.y != kInf && tv.z != kInf &&
            tv.w != kInf) {
            const Pt a = vpt(vx, tv.x), b = vpt(vx, tv.y), c = vpt(vx, tv.z), d = vpt(vx, tv.w);
            const Pt A = lane == 0 ? p : a, B = lane == 1 ? p : b, C = lane == 2 ? p : c, D = lane == 3 ? p : d;
            const int o = orient3d_x(A, B, C, D, ex, st);
            neg = o < 0;
        }
        const unsigned m = __ballot_sync(kFull, neg) & 0xFu;
        if (m == 0) return t;
        const unsigned rot = ((m >> s0) | (m << (4 - s0))) & 0xFu;
        const int i = (s0 + __ffs(int(rot)) - 1) & 3;
        const int next = at(tn, i) >> 2;
        const int4 nv = make_int4(__shfl_sync(kFull, pre.x, 4 + i), __shfl_sync(kFull, pre.y, 4 + i),
                                  __shfl_sync(kFull, pre.z, 4 + i), __shfl_sync(kFull, pre.w, 4 + i));
        const int4 nn = make_int4(__shfl_sync(kFull, pre.x, 8 + i), __shfl_sync(kFull, pre.y, 8 + i),
                                  __shfl_sync(kFull, pre.z, 8 + i), __shfl_sync(kFull, pre.w, 8 + i));
        if (inf_pos(nv) >= 0) return next;
        prev = t;
        t = next;
        tv = nv;
        tn = nn;
    }
    return -1;
}

/// A vertex's coordinates read again from memory (the read-only path), as a
/// volatile load so that the compiler does not keep an earlier read of them
/// alive in registers across the code in between.
__device__ __forceinline__ Pt ld_vertex(const double* __restrict__ vx, int v) {
    double x, y, z, pad;
    asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(x), "=d"(y), "=d"(z), "=d"(pad)
                 : "l"(vx + 4 * int64_t(v)));
    return Pt{x, y, z};
}

/// The symbolic perturbation of an exactly cospherical in_sphere(a, b, c, d, p)
/// (reference src/predicates.cpp:206-232) for the conflict test of tet t and
/// vertex pid, when the set's coordinates make the orient3d filter exact.  The
/// five points are distinct vertices, so their lexicographic order is strict:
/// walking down it from the largest, the largest is p -> NEGATIVE; else the
/// orient3d with that point's slot replaced by p decides if it is not zero;
/// else the next largest, once more; else NEGATIVE.  Points are read again
/// from memory each time they are needed, so the tie-break adds no live state
/// to the loop around it.
template <class M>
__device__ __forceinline__ int in_sphere_tiebreak_ex(const M& m, const int4 t, int pid) {
    int skip = -1;
#pragma unroll 1
    for (int r = 0; r < 2; ++r) {
        int best = -1;
        Pt bp{0.0, 0.0, 0.0};
#pragma unroll 1
        for (int k = 0; k < 5; ++k) {
            if (k == skip) continue;
            const Pt q = m.again(k < 4 ? at(t, k) : pid);
            if (best < 0 || lexico_less(bp, q)) {
                best = k;
                bp = q;
            }
        }
        if (best == 4) return -1;
        const Pt pp = m.again(pid);
        const Pt A = best == 0 ? pp : m.again(t.x), B = best == 1 ? pp : m.again(t.y),
                 C = best == 2 ? pp : m.again(t.z), D = best == 3 ? pp : m.again(t.w);
        const int o = -sign_of(orient3d_filter(A, B, C, D).det);
        if (o != 0) return o;
        skip = best;
    }
    return -1;
}

/// Error bound of in_sphere_filter from the squared distances alone.  Each pair
/// sum |x1 y2| + |x2 y1| of the permanent is at most l = max lift (Cauchy-
/// Schwarz), each coordinate at most sqrt(l), so the permanent is at most
/// 12 l^(5/2), and det^2 > (12 bound)^2 l^5 certifies what the filter would
/// certify.  `l` is taken from the lifts' high words, rounded up; the range
/// check keeps l^5 and det^2 normal (outside it the filter's own bound decides).
__device__ __forceinline__ bool in_sphere_far(double det, double alift, double blift, double clift, double dlift) {
    const int h = max(max(__double2hiint(alift), __double2hiint(blift)),
                      max(__double2hiint(clift), __double2hiint(dlift)));   // lifts are not negative
    constexpr int kLow = (1023 - 180) << 20, kHigh = (1023 + 180) << 20;
    const double l = __hiloint2double(h + 1, 0), l2 = fmul(l, l);
    constexpr double c = 12.0 * kInSphereBound * (1.0 + 1e-6);
    return h > kLow && h < kHigh && fmul(det, det) > fmul(fmul(fmul(l2, l2), l), c * c);
}

/// in_sphere_filter's arithmetic, operation for operation (so its value and
/// its decision are bit-identical), in an order that retires values early:
/// lifts right after the differences, each product pair folded at once into
/// its minor and its permanent pair sum (|x*y| = |x|*|y| exactly).
__device__ __forceinline__ InSphereFilter in_sphere_filter_lean(const Pt& a, const Pt& b, const Pt& c, const Pt& d,
                                                                const Pt& e) {
    const double aex = fsub(a.x, e.x), aey = fsub(a.y, e.y), aez = fsub(a.z, e.z);
    const double bex = fsub(b.x, e.x), bey = fsub(b.y, e.y), bez = fsub(b.z, e.z);
    const double cex = fsub(c.x, e.x), cey = fsub(c.y, e.y), cez = fsub(c.z, e.z);
    const double dex = fsub(d.x, e.x), dey = fsub(d.y, e.y), dez = fsub(d.z, e.z);
    const double alift = fadd(fadd(fmul(aex, aex), fmul(aey, aey)), fmul(aez, aez));
    const double blift = fadd(fadd(fmul(bex, bex), fmul(bey, bey)), fmul(bez, bez));
    const double clift = fadd(fadd(fmul(cex, cex), fmul(cey, cey)), fmul(cez, cez));
    const double dlift = fadd(fadd(fmul(dex, dex), fmul(dey, dey)), fmul(dez, dez));
    double ab, bc, cd, da, ac, bd;
    {
        const double p = fmul(aex, bey), q = fmul(bex, aey);
        ab = fsub(p, q);
    }
    {
        const double p = fmul(bex, cey), q = fmul(cex, bey);
        bc = fsub(p, q);
    }
    {
        const double p = fmul(cex, dey), q = fmul(dex, cey);
        cd = fsub(p, q);
    }
    {
        const double p = fmul(dex, aey), q = fmul(aex, dey);
        da = fsub(p, q);
    }
    {
        const double p = fmul(aex, cey), q = fmul(cex, aey);
        ac = fsub(p, q);
    }
    {
        const double p = fmul(bex, dey), q = fmul(dex, bey);
        bd = fsub(p, q);
    }
    const double abc = fadd(fsub(fmul(aez, bc), fmul(bez, ac)), fmul(cez, ab));
    const double bcd = fadd(fsub(fmul(bez, cd), fmul(cez, bd)), fmul(dez, bc));
    const double cda = fadd(fadd(fmul(cez, da), fmul(dez, ac)), fmul(aez, cd));
    const double dab = fadd(fadd(fmul(dez, ab), fmul(aez, bd)), fmul(bez, da));
    const double det = fadd(fsub(fmul(dlift, abc), fmul(clift, dab)), fsub(fmul(blift, cda), fmul(alift, bcd)));
    if (in_sphere_far(det, alift, blift, clift, dlift)) return InSphereFilter{det, true};
    const double sab = fadd(fabs_(fmul(aex, bey)), fabs_(fmul(bex, aey)));
    const double sbc = fadd(fabs_(fmul(bex, cey)), fabs_(fmul(cex, bey)));
    const double scd = fadd(fabs_(fmul(cex, dey)), fabs_(fmul(dex, cey)));
    const double sda = fadd(fabs_(fmul(dex, aey)), fabs_(fmul(aex, dey)));
    const double sac = fadd(fabs_(fmul(aex, cey)), fabs_(fmul(cex, aey)));
    const double sbd = fadd(fabs_(fmul(bex, dey)), fabs_(fmul(dex, bey)));
    const double aezp = fabs_(aez), bezp = fabs_(bez), cezp = fabs_(cez), dezp = fabs_(dez);
    const double pa = fadd(fadd(fmul(scd, bezp), fmul(sbd, cezp)), fmul(sbc, dezp));
    const double pb = fadd(fadd(fmul(sda, cezp), fmul(sac, dezp)), fmul(scd, aezp));
    const double pc = fadd(fadd(fmul(sab, dezp), fmul(sbd, aezp)), fmul(sda, bezp));
    const double pd = fadd(fadd(fmul(sbc, aezp), fmul(sac, bezp)), fmul(sab, cezp));
    const double permanent = fadd(fadd(fadd(fmul(pa, alift), fmul(pb, blift)), fmul(pc, clift)), fmul(pd, dlift));
    const double errbound = fmul(kInSphereBound, permanent);
    InSphereFilter r;
    r.det = det;
    r.certain = (det > errbound) || (-det > errbound);
    return r;
}

/// coplanar_orientation3 (the first non-zero orient2d of the xy, yz and xz
/// projections) for a set whose coordinates make the orient2d determinants
/// exact in double: each is the sign of its determinant.
__device__ __forceinline__ int coplanar_orientation3_ex(const Pt& p, const Pt& q, const Pt& r) {
    int o = sign_of(fsub(fmul(fsub(q.x, p.x), fsub(r.y, p.y)), fmul(fsub(q.y, p.y), fsub(r.x, p.x))));
    if (o != 0) return o;
    o = sign_of(fsub(fmul(fsub(q.y, p.y), fsub(r.z, p.z)), fmul(fsub(q.z, p.z), fsub(r.y, p.y))));
    if (o != 0) return o;
    return sign_of(fsub(fmul(fsub(q.x, p.x), fsub(r.z, p.z)), fmul(fsub(q.z, p.z), fsub(r.x, p.x))));
}

/// The cocircular tie-break (reference src/predicates2.cpp:241-258) of four
/// distinct vertices va, vb, vd, pid of such a set: walking down their
/// lexicographic order from the largest, the first that is pid gives NEGATIVE;
/// the first other one whose replacement by pid gives a non-zero coplanar
/// orientation gives it times the orientation of (va, vb, vd); else the
/// opposite of that orientation.  Points are read again from memory, as in
/// in_sphere_tiebreak_ex.
template <class M>
__device__ __forceinline__ int in_circle_tiebreak_ex(const M& m, int va, int vb, int vd, int pid) {
    const int local = coplanar_orientation3_ex(m.again(va), m.again(vb), m.again(vd));
    unsigned excluded = 0;
#pragma unroll 1
    for (int r = 0; r < 3; ++r) {
        int best = -1;
        Pt bp{0.0, 0.0, 0.0};
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            if (excluded & (1u << k)) continue;
            const Pt q = m.again(k == 0 ? va : (k == 1 ? vb : (k == 2 ? vd : pid)));
            if (best < 0 || !lexico_less(q, bp)) {   // a later slot wins ties
                best = k;
                bp = q;
            }
        }
        excluded |= 1u << best;
        if (best == 3) return -1;
        const Pt pp = m.again(pid);
        const Pt A = best == 0 ? pp : m.again(va), B = best == 1 ? pp : m.again(vb),
                 C = best == 2 ? pp : m.again(vd);
        const int o = coplanar_orientation3_ex(A, B, C);
        if (o != 0) return o * local;
    }
    return -local;
}

/// in_sphere of tet t and vertex pid in 64-bit integers, for points of a set
/// whose coordinates are multiples of 1 / inv: exact where no difference exceeds
/// kNearSteps steps (72 kNearSteps^5 < 2^63).  Returns its sign, or 2 where the
/// points are too far apart or the set has no such grid.  Points are read again,
/// as in in_sphere_tiebreak_ex.
constexpr double kNearSteps = 2600.0;
template <class M>
__device__ __forceinline__ int in_sphere_near(const M& m, const int4 t, int pid, double inv) {
    const Pt e = m.again(pid);
    bool near = inv > 0.0;
    auto steps = [&](int v, long long& x, long long& y, long long& z) {
        const Pt p = m.again(v);
        const double dx = fmul(fsub(p.x, e.x), inv), dy = fmul(fsub(p.y, e.y), inv), dz = fmul(fsub(p.z, e.z), inv);
        near = near && fabs_(dx) <= kNearSteps && fabs_(dy) <= kNearSteps && fabs_(dz) <= kNearSteps;
        x = (long long)dx;
        y = (long long)dy;
        z = (long long)dz;
    };
    long long ax, ay, az, bx, by, bz, cx, cy, cz, dx, dy, dz;
    steps(t.x, ax, ay, az);
    steps(t.y, bx, by, bz);
    steps(t.z, cx, cy, cz);
    steps(t.w, dx, dy, dz);
    if (!near) return 2;
    const long long ab = ax * by - bx * ay, bc = bx * cy - cx * by, cd = cx * dy - dx * cy, da = dx * ay - ax * dy,
                    ac = ax * cy - cx * ay, bd = bx * dy - dx * by;
    const long long abc = az * bc - bz * ac + cz * ab, bcd = bz * cd - cz * bd + dz * bc,
                    cda = cz * da + dz * ac + az * cd, dab = dz * ab + az * bd + bz * da;
    const long long det = ((dx * dx + dy * dy + dz * dz) * abc - (cx * cx + cy * cy + cz * cz) * dab) +
                          ((bx * bx + by * by + bz * bz) * cda - (ax * ax + ay * ay + az * az) * bcd);
    return det > 0 ? -1 : (det < 0 ? 1 : 0);   // in_sphere = -sign(det)
}

/// The hull in-circle test (reference src/triangulation.cpp:588-602, a point
/// in the plane of the hull facet (va, vb, vd) of infinite tet `tet`: in
/// conflict iff inside the facet's circumcircle, a tie by the cocircular
/// perturbation) for a set whose coordinates make orient3d exact, without
/// the in-circle determinant: the sphere through va, vb, vd and the apex x of
/// the finite tet across the facet cuts the facet's plane in the facet's
/// circumcircle, and a point of that plane has the same power with respect
/// to both, so sign in_circle(va, vb, vd, p) = sign det_in_sphere(va, vb, vd,
/// x, p) * sign det_orient3d(va, vb, vd, x); the first is exact in double
/// (`sphere`: the set's coordinates make it so) or in 64 bits (in_sphere_near).  The caller
/// holds the lock of `tet`, so the finite tet across its facet is not being
/// rewritten.  Returns 1 (inside), -1 (outside), or 0 if the apex is unusable
/// (the caller then leaves the test undecided).
template <bool kNear, class M>
__device__ __forceinline__ int hull_in_circle_ex(const M& m, int tet, int ip, int va, int vb, int vd, int pid,
                                                 bool sphere) {
    const int f = at(m.tn4(tet), ip) >> 2;
    const int4 fv = m.tv4(f);
    int x = -1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int w = at(fv, k);
        if (w != va && w != vb && w != vd) x = w;
    }
    if (x < 0) return 0;   // kInf is negative
    const Pt a = m.again(va), b = m.again(vb), d = m.again(vd), xp = m.again(x);
    const int so = sign_of(orient3d_filter(a, b, d, xp).det);
    if (so == 0) return 0;
    if (!kNear && !sphere) return 0;
    const int ss = sphere ? sign_of(in_sphere_filter_lean(a, b, d, xp, m.again(pid)).det)
                          : -in_sphere_near(m, make_int4(va, vb, vd, x), pid, m.inv(pid));
    if (ss == -2) return 0;
    if (ss != 0) return ss * so;
    return in_circle_tiebreak_ex(m, va, vb, vd, pid);
}

/// The conflict test of k_insert_groups (reference src/triangulation.cpp:588-602,
/// as conflict_test) of tet `tet` = t, with its outcome bits; CT_UNDECIDED when
/// the filter cannot decide and the exact stage is needed.  Call-free: where the
/// set's coordinates make the filters exact (`ex`: EX_*), or (kNear) the points
/// lie near enough on its grid, an undecided call is settled inline, an exactly
/// cospherical one by its tie-break and a point in the plane of a hull facet by
/// its in-circle test.
template <bool kNear, class M>
__device__ __forceinline__ int in_conflict_fast(const M& m, int tet, const int4 t, const Pt& p, int pid, int ex) {
    const int ip = inf_pos(t);
    if (ip >= 0) {
        const int o0 = ip == 0 ? 2 : (ip == 1 ? 2 : (ip == 2 ? 1 : 0));
        const int o1 = ip == 0 ? 1 : (ip == 1 ? 3 : (ip == 2 ? 0 : 1));
        const int o2 = ip == 0 ? 3 : (ip == 1 ? 0 : (ip == 2 ? 3 : 2));
        const Pt a = m.point(at(t, o0)), b = m.point(at(t, o1)), d = m.point(at(t, o2));
        const Orient3dFilter f = orient3d_filter(a, b, d, p);
        if (f.certain) return f.det < 0.0 ? CT_IN : 0;   // orient3d = -sign(det)
        if ((ex & EX_ORIENT) && f.det != 0.0) return (f.det < 0.0 ? CT_IN : 0) | CT_UNCERTAIN;
        if (ex & EX_ORIENT) {
            const int h = hull_in_circle_ex<kNear>(m, tet, ip, at(t, o0), at(t, o1), at(t, o2), pid, ex & EX_SPHERE);
            if (h != 0) return (h > 0 ? CT_IN : 0) | CT_UNCERTAIN | CT_TIE;
        }
        return CT_UNDECIDED;
    }
    const Pt a = m.point(t.x), b = m.point(t.y), c = m.point(t.z), d = m.point(t.w);
    const InSphereFilter f = in_sphere_filter_lean(a, b, c, d, p);
    if (f.certain) return f.det < 0.0 ? CT_IN : 0;   // in_sphere = -sign(det)
    int s = 0;
    if (ex & EX_SPHERE) s = -sign_of(f.det);
    else s = kNear ? in_sphere_near(m, t, pid, m.inv(pid)) : 2;
    if (s == 2) return CT_UNDECIDED;
    if (s != 0) return (s > 0 ? CT_IN : 0) | CT_UNCERTAIN;
    return (in_sphere_tiebreak_ex(m, t, pid) > 0 ? CT_IN : 0) | CT_UNCERTAIN | CT_TIE;
}

enum : int { AI_DONE = 0, AI_RETRY = 1, AI_LEAVE = 2, AI_DEFER = 3 };

#include "insert_groups.cuh"

/// Key of the edge (a, b), either order.
__device__ __forceinline__ unsigned long long edge_key(int a, int b) {
    const unsigned ua = unsigned(a + 1), ub = unsigned(b + 1);
    return ua < ub ? ((unsigned long long)ua << 32) | ub : ((unsigned long long)ub << 32) | ua;
}

/// Edge keys of facets p0 < p1 < p2 (the positions other than i) of a tet with
/// vertices c: facet j's edge joins the two positions other than i and j.
__device__ __forceinline__ void facet_edge_keys(const int4 c, int i, unsigned long long& e0,
                                                unsigned long long& e1, unsigned long long& e2) {
    const int p0 = i == 0 ? 1 : 0, p1 = i <= 1 ? 2 : 1, p2 = i <= 2 ? 3 : 2;
    const int a0 = at(c, p0), a1 = at(c, p1), a2 = at(c, p2);
    e0 = edge_key(a1, a2);
    e1 = edge_key(a0, a2);
    e2 = edge_key(a0, a1);
}

/// One insertion of point v by the whole warp, starting the walk at tet t0.
/// AI_DONE: inserted; AI_RETRY: a lock was taken by another warp (nothing
/// changed, every lock given back); AI_LEAVE: leave it for the rounds.  Every
/// test runs to its end here: the exact stage, the hull in-circle test and the
/// tie-breaks, out of line.
__device__ int insert_full(int v, int t0, const Tables& T, const Workers& W, const AsyncCtx& A,
                            const double* __restrict__ vx, bool ex, uint32_t* st, int slot, int lane,
                            unsigned long long* nC, unsigned long long* nF, const SharedCounters& ctr,
                            int4* htn) {
    const int owner = slot + 1;
    const int region = owner << 1, ring = region | 1;
    const Pt p = vpt(vx, v);
    const int seed = walk_async(t0, p, v, T, vx, ex, st, lane);
    if (seed < 0) {
        if (lane == 0) atomicAdd(A.stats + 1, 1ull);
        return AI_RETRY;
    }
    int* cav = W.cav + int64_t(slot) * W.cav_cap;
    int* fac = W.fac + int64_t(slot) * W.fac_cap;
    // Seed: lock it, then check under the lock that it is alive and in conflict.
    int res = 0;   // 0 ok, 1 lock held by another, 2 not a valid seed

    if (lane == 0) {
        int seen = 0;
        if (!try_lock(A.lock, seed, region, &seen)) {
            res = 1;
        } else {
            // The walk read tets other warps were rewriting: a tet read half
            // written (vertices new, neighbours not yet) can send it on through a
            // slot not yet filled in - into another set's tets in a batched
            // build.  Only a live tet of v's own set can seed the region.
            int r = 0;
            const int4 stv = ld4(&T.tv(seed));
            htn[0] = ld4(&T.tn(seed));
            if (stv.x != stv.y && T.vset[stv.x != kInf ? stv.x : stv.y] == T.vset[v]) {
                r = conflict_test_exact(stv, p.x, p.y, p.z, v, vx, ex, st);
                ctr.count(r);
            }
            if (r & CT_IN) {
                cav[0] = seed;
            } else {
                unlock_if(A.lock, seed, region);
                res = 2;
            }
        }
    }
    res = __shfl_sync(kFull, res, 0);
    if (res != 0) {
        if (lane == 0) atomicAdd(A.stats + (res == 1 ? 0 : 2), 1ull);
        return AI_RETRY;
    }
    __syncwarp();
    const unsigned lt = (1u << lane) - 1u;
    int ncav = 1, nfac = 0, head = 0;
    int outcome = AI_DONE;
    while (head < ncav) {
        const int nproc = min(ncav - head, 8);
        const bool valid = (lane >> 2) < nproc;
        const int i = lane & 3;
        int c = 0, nb = 0, kind = 0, got = -1;   // got: a tet this lane locked in this step
        bool abort = false;
        int4 found_tn = make_int4(0, 0, 0, 0);
        if (valid) {
            const int pidx = head + (lane >> 2);
            c = cav[pidx];
            nb = at(pidx < kHandedTn ? htn[pidx] : ld4(&T.tn(c)), i) >> 2;
            int seen = 0;
            if (try_lock(A.lock, nb, ring, &seen)) {
                got = nb;
                const int4 ntv = ld4(&T.tv(nb));
                found_tn = ld4(&T.tn(nb));
                const int r = conflict_test(ntv, p, v, vx, ex, st);
                ctr.count(r);
                if (r & CT_IN) {
                    LockRef(A.lock[nb]).store(region, cuda::memory_order_relaxed);
                    kind = 2;
                } else {
                    kind = 1;
                }
            } else if (seen == region) {
                kind = 0;                                 // already in the region
            } else if (seen == ring) {
                kind = 3;                                 // locked by us this step: decided below
            } else {
                abort = true;                             // another warp holds it
            }
        }
        __syncwarp();
        if (kind == 3) kind = __ldcg(A.lock + nb) == region ? 0 : 1;
        const bool ab = __any_sync(kFull, abort);
        const unsigned mc = __ballot_sync(kFull, kind == 2);
        const unsigned mf = __ballot_sync(kFull, kind == 1);
        const bool full = ncav + __popc(mc) > W.cav_cap || nfac + __popc(mf) > W.fac_cap;
        if (ab || full) {
            // Give everything back: this step's new locks, the region, the ring.
            if (got >= 0) unlock_if(A.lock, got, kind == 2 ? region : ring);
            __syncwarp();
            for (int k = lane; k < nfac; k += 32) {
                const int f = fac[k];
                unlock_if(A.lock, at(ld4(&T.tn(f >> 2)), f & 3) >> 2, ring);
            }
            __syncwarp();
            for (int k = lane; k < ncav; k += 32) unlock_if(A.lock, cav[k], region);
            if (lane == 0) atomicAdd(A.stats + (ab ? 0 : 3), 1ull);
            outcome = ab ? AI_RETRY : AI_LEAVE;
            break;
        }
        if (kind == 2) cav[ncav + __popc(mc & lt)] = nb;
        if (kind == 1) fac[nfac + __popc(mf & lt)] = c * 4 + i;
        if (kind == 2 && ncav + __popc(mc & lt) < kHandedTn) htn[ncav + __popc(mc & lt)] = found_tn;
        ncav += __popc(mc);
        nfac += __popc(mf);
        head += nproc;
        __syncwarp();
    }
    if (outcome != AI_DONE) return outcome;

    // Re-star (as k_restar), reading the locked region through L2.
    const int C = ncav, F = nfac;
    const int extra = F > C ? F - C : 0;
    int base = 0, ok = 1;
    if (lane == 0 && extra > 0) {
        base = atomicAdd(T.tet_count, extra);
        if (base + extra > T.cap) {
            report(st, ST_TET_CAPACITY);
            ok = 0;
        }
    }
    base = __shfl_sync(kFull, base, 0);
    ok = __shfl_sync(kFull, ok, 0);
    int4* sv = W.st_v + int64_t(slot) * W.fac_cap;
    int4* sn = W.st_n + int64_t(slot) * W.fac_cap;
    // A fresh slot is locked from the start (no tet was ever in it), so whoever
    // reads its tet reads it after this warp's release.
    if (ok) {
        // New tet k (on boundary facet (c, i), vertex i of c replaced by v) keeps
        // c's outside neighbour across facet i.  Its facet j != i is v plus the
        // edge of c's vertices at the other two positions; that edge lies on
        // exactly one other boundary facet k2, where it is the edge of some
        // facet j2 of new tet k2: the two new tets meet there, k2 facing back
        // through j2.  Matching edge keys gives the same adjacency as turning
        // round the edge inside the region (reference src/tds.h:160-221)
        // without reading the mesh again.  The keys go through the warp's key
        // scratch, which stays in L1 (a shared-memory hash table per warp was
        // slower: the shared memory it takes comes out of L1).
        unsigned long long* keys = A.ekey + int64_t(slot) * 3 * W.fac_cap;
        for (int k = lane; k < F; k += 32) {
            const int c = fac[k] >> 2, i = fac[k] & 3;
            const int4 cv = ld4(&T.tv(c));
            int4 nv = cv;
            set_at(nv, i, v);
            sv[k] = nv;
            sn[k] = ld4(&T.tn(c));
            facet_edge_keys(cv, i, keys[3 * k], keys[3 * k + 1], keys[3 * k + 2]);
        }
        __syncwarp();
        bool bad = false;
        for (int k = lane; k < F; k += 32) {
            // One pass over the keys of every other facet finds the partners of
            // all three edges (key m of facet k2 is its edge m: each edge key
            // must occur on exactly one other facet).  The lanes walk the keys
            // in step, so every load is a broadcast.
            const unsigned long long e0 = keys[3 * k], e1 = keys[3 * k + 1], e2 = keys[3 * k + 2];
            int f0 = -1, f1 = -1, f2 = -1, n0 = 0, n1 = 0, n2 = 0;
            for (int o = 0; o < F; ++o) {
                const bool other = o != k;
#pragma unroll
                for (int m2 = 0; m2 < 3; ++m2) {
                    const unsigned long long key = keys[3 * o + m2];
                    const int q = 3 * o + m2;
                    if (other && key == e0) { f0 = q; ++n0; }
                    if (other && key == e1) { f1 = q; ++n1; }
                    if (other && key == e2) { f2 = q; ++n2; }
                }
            }
            const int i = fac[k] & 3;
            int4 nn = sn[k];
            // Facet j of new tet k (j != i, increasing) carries edge key m = 0, 1, 2.
            auto link = [&](int j, int found, int count) {
                if (count != 1) {
                    bad = true;
                    return;
                }
                const int k2 = found / 3, m2 = found - 3 * k2, i2 = fac[k2] & 3;
                const int j2 = m2 + (m2 >= i2 ? 1 : 0);
                set_at(nn, j, (k2 < C ? cav[k2] : base + (k2 - C)) * 4 + j2);
            };
            link(i == 0 ? 1 : 0, f0, n0);
            link(i <= 1 ? 2 : 1, f1, n1);
            link(i <= 2 ? 3 : 2, f2, n2);
            sn[k] = nn;
        }
        if (__any_sync(kFull, bad)) {
            if (lane == 0) report(st, ST_INTERNAL);
            ok = 0;
        }
        __syncwarp();
    }
    if (ok) {
        for (int k = lane; k < F; k += 32) {
            const int id = k < C ? cav[k] : base + (k - C);
            const int4 nv = sv[k], nn = sn[k];
            const int i = fac[k] & 3;
            T.tv(id) = nv;
            T.tn(id) = nn;
            const int enc = at(nn, i);
            T.link(enc) = id * 4 + i;
            if (nv.x != kInf) T.vert_tet[nv.x] = id;
            if (nv.y != kInf) T.vert_tet[nv.y] = id;
            if (nv.z != kInf) T.vert_tet[nv.z] = id;
            if (nv.w != kInf) T.vert_tet[nv.w] = id;
        }
        for (int k = F + lane; k < C; k += 32) T.kill(cav[k]);
    }
    // Publish, then give the locks back (ring tets first: their neighbour
    // entries now point at the new tets).
    __threadfence();
    __syncwarp();
    for (int k = lane; k < F; k += 32) {
        const int f = fac[k];
        const int c = f >> 2, i = f & 3;
        // The outside tet across facet (c, i): read from the staged neighbours,
        // since slot c may now hold a new tet.
        const int outside = ok ? (at(sn[k], i) >> 2) : (at(ld4(&T.tn(c)), i) >> 2);
        unlock_if(A.lock, outside, ring);
    }
    __syncwarp();
    for (int k = lane; k < C; k += 32) unlock_if(A.lock, cav[k], region);
    if (ok)
        for (int k = C + lane; k < F; k += 32) unlock_if(A.lock, base + (k - C), -1);
    if (lane == 0) {
        *nC += (unsigned long long)C;
        *nF += (unsigned long long)F;
    }
    if (ok && lane == 0) ctr.region(C);
    return ok ? AI_DONE : AI_LEAVE;
}

/// The full variant: persistent warps over the points k_insert_groups left, one
/// worker each (k_setup_list).
__global__ void __launch_bounds__(128, 8) k_insert_full(Tables T, Workers W, AsyncCtx A, Round R,
                                                      const double* __restrict__ vx, int nslots) {
    const int lane = threadIdx.x & 31;
    const int slot = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (slot >= nslots) return;   // the grid is rounded up to whole blocks; scratch has nslots slots
    unsigned long long won = 0, tries = 0, nC = 0, nF = 0;
    D3G_SHARED_COUNTERS(ctr);
    __shared__ int4 handed_tn[4][kHandedTn];   // per warp of the block
    for (;;) {
        int q = 0;
        if (lane == 0) q = atomicAdd(A.next, 1);
        q = __shfl_sync(kFull, q, 0);
        if (q >= A.nw) break;
        const int w = int((int64_t(q) * A.stride) % A.nw);
        const bool ex = (W.set_exact[W.wset[w]] & EX_BOTH) == EX_BOTH;
        const int v = W.cur[w];
        if (v < 0) continue;
        int outcome = AI_RETRY;
        for (int attempt = 0; attempt < kAsyncRetries && outcome == AI_RETRY; ++attempt) {
            if (attempt > 0) __nanosleep(200u << min(attempt, 6));
            outcome = insert_full(v, __ldcg(T.vert_tet + W.guide[w]), T, W, A, vx, ex, R.status, slot, lane, &nC, &nF,
                                  ctr, handed_tn[threadIdx.x >> 5]);
            ++tries;
            if (__ldcg(R.status) != 0) outcome = AI_LEAVE;
        }
        if (outcome == AI_DONE) {
            ++won;
        } else if (lane == 0) {
            A.leftover[atomicAdd(A.n_leftover, 1)] = v;
            atomicAdd(A.stats + 4, 1ull);
        }
        if (__ldcg(R.status) != 0) break;
    }
    if (lane == 0) {
        atomicAdd(R.totals, won);
        atomicAdd(R.totals + 1, tries);
        atomicAdd(R.sums, nC);
        atomicAdd(R.sums + 1, nF);
    }
    flush_counters(ctr, R);
}

// ---- structural self-check (the reference's Tds::validate, src/tds.h:483-530) ----

/// Codes of the first broken invariant k_validate finds.
enum : int {
    VF_VERTEX = 1,      // a vertex out of range, or repeated in a tet, or two infinite
    VF_NEIGHBOUR = 2,   // a neighbour out of range or dead
    VF_BACK = 3,        // a neighbour that does not point back through the same facet
    VF_FACET = 4,       // two neighbours whose shared facets have different vertices
    VF_LOCK = 5,        // a tet still locked after the asynchronous passes
    VF_VERT_TET = 6,    // an inserted vertex whose tet is dead or does not contain it
    VF_SET = 7,         // a tet whose vertices belong to different point sets
};

/// One thread per tet slot, then one per vertex: checks what the reference's
/// validate() checks - distinct vertices, live neighbours that point back, no
/// mark left behind (here: no lock held), every vertex's cached tet alive and
/// containing it - and, beyond it, that each pair of neighbours shares the
/// same three vertices.  Every index is range-checked before it is followed.
/// The first failure (lowest code, then lowest slot) is recorded in `fail` =
/// code << 60 | tet or vertex << 30 | detail, and ST_INTERNAL is reported;
/// nothing traps.
__global__ void k_validate(Tables T, const int* __restrict__ lock, int ntet, int nv, uint32_t* status,
                           unsigned long long* fail) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    int code = 0, where = 0, detail = 0;
    if (i < ntet) {
        const int c = int(i);
        if (T.alive(c)) {
            const int4 tv = T.tv(c), tn = T.tn(c);
            int ninf = 0;
            for (int k = 0; k < 4 && !code; ++k) {
                const int v = at(tv, k);
                if (v < -1 || v >= nv) code = VF_VERTEX;
                ninf += v == kInf;
                for (int m = k + 1; m < 4; ++m)
                    if (v == at(tv, m)) code = VF_VERTEX;
                detail = k;
            }
            if (!code && ninf > 1) code = VF_VERTEX;
            if (!code) {
                const int s0 = T.vset[tv.x != kInf ? tv.x : tv.y];
                for (int k = 0; k < 4; ++k)
                    if (at(tv, k) != kInf && T.vset[at(tv, k)] != s0) code = VF_SET;
            }
            for (int k = 0; k < 4 && !code; ++k) {
                detail = k;
                const int e = at(tn, k);
                const int n = e >> 2, f = e & 3;
                if (e < 0 || n >= ntet || !T.alive(n)) {
                    code = VF_NEIGHBOUR;
                    break;
                }
                if (at(T.tn(n), f) != c * 4 + k) {
                    code = VF_BACK;
                    break;
                }
                // The facet of c opposite k and the facet of n opposite f: the same
                // three vertices (in any order).
                const int4 nvx = T.tv(n);
                for (int m = 0; m < 4 && !code; ++m) {
                    if (m == k) continue;
                    const int v = at(tv, m);
                    bool found = false;
                    for (int q = 0; q < 4; ++q) found = found || (q != f && at(nvx, q) == v);
                    if (!found) code = VF_FACET;
                }
            }
            if (!code && lock && lock[c] != 0) {
                code = VF_LOCK;
                detail = lock[c];
            }
        }
        where = c;
    } else if (i < int64_t(ntet) + nv) {
        const int v = int(i - ntet);
        const int c = T.vert_tet[v];
        if (c >= 0) {   // -1: not inserted yet
            if (c >= ntet || !T.alive(c)) code = VF_VERT_TET;
            else if (pos_of(T.tv(c), v) == 3 && T.tv(c).w != v) code = VF_VERT_TET;
            detail = c;
        }
        where = v;
    }
    if (code) {
        report(status, ST_INTERNAL);
        const unsigned long long rec = (unsigned long long)(uint32_t(code)) << 60 |
                                       (unsigned long long)(uint32_t(where) & 0x3FFFFFFFu) << 30 |
                                       (unsigned long long)(uint32_t(detail) & 0x3FFFFFFFu);
        atomicMin(fail, rec);
    }
}

/// Workers for the points the asynchronous pass left: one point each, its walk
/// starting from the nearest earlier inserted vertex of its set.
__global__ void k_setup_list(Workers W, const int* __restrict__ list, int n, const int32_t* __restrict__ vset,
                             const int32_t* __restrict__ voff, const int* __restrict__ vert_tet) {
    const int w = int(blockIdx.x) * blockDim.x + threadIdx.x;
    if (w >= n) return;
    const int v = list[w];
    const int set = vset[v];
    W.beg[w] = v;
    W.end[w] = v + 1;
    W.pos[w] = 0;
    W.left[w] = 1;
    W.nwon[w] = 0;
    W.parked[w] = 0;
    W.last[w] = -1;
    W.wset[w] = set;
    next_point(W, w);
    int g = W.skips[set].x;
    for (int u = v - 1, k = 0; u >= voff[set] && k < 4096; --u, ++k)
        if (__ldcg(vert_tet + u) >= 0) {
            g = u;
            break;
        }
    W.guide[w] = g;
    W.state[w] = WS_DONE;
}

/// What a set's coordinates say of its filters.  All are multiples of grid = 2^emin
/// and lie in a box of longest side D grid steps, so every difference a filter
/// takes is a whole number of steps, at most D: exact in double, and with it
/// every product and sum of the determinants while these stay below 2^53.
/// orient3d sums 6 products of 3 differences (6 D^3), in_sphere 72 of 5 (72 D^5).
/// Bit 0: orient3d's filter value is exact for any points of the set, bit 1:
/// in_sphere's; bit 2: a grid of few enough steps that its points often are
/// cospherical, but too many for bit 1.  `inv_grid` is 1 / grid, for the tests whose five points are near
/// enough to be exact in 64 bits by themselves (in_sphere_near); 0 where the
/// scale leaves the range in which nothing can over- or underflow.
constexpr double kGridSteps = 1048576.0;
__global__ void k_set_exact(const int* __restrict__ span, const unsigned long long* __restrict__ box, int nsets,
                            uint8_t* __restrict__ ex, double* __restrict__ inv_grid) {
    const int s = int(blockIdx.x) * blockDim.x + threadIdx.x;
    if (s >= nsets) return;
    const int emin = span[s], top = span[nsets + s];
    int r = 0;
    double inv = 0.0;
    if (top < emin) {   // no coordinate but zeros
        r = EX_ORIENT | EX_SPHERE;
    } else if (emin >= -200 && emin <= 190) {
        inv = scalbn(1.0, -emin);
        double side = 0.0;
        for (int k = 0; k < 3; ++k)
            side = fmax(side, dbl_from_order_key(box[6 * int64_t(s) + 3 + k]) - dbl_from_order_key(box[6 * int64_t(s) + k]));
        const double steps = side * inv;
        r = (steps <= 110000.0 ? EX_ORIENT : 0) | (steps <= 659.0 ? EX_SPHERE : (steps <= kGridSteps ? EX_GRID : 0));
    }
    ex[s] = uint8_t(r);
    inv_grid[s] = inv;
}

/// Puts every vertex but the first tets' in its level's list (items), and gives
/// it the vertex its walk starts from: the nearest along the curve of the level
/// before (`keys` sorted, the curve in their low bits; null: the one at the same
/// fraction of that level), or in the first level its neighbour before it.
__global__ void __launch_bounds__(256) k_level_items(const int32_t* __restrict__ vset, const int4* __restrict__ skips,
                                                     const int* __restrict__ starts, int stride,
                                                     const int* __restrict__ base, int nsets,
                                                     const unsigned long long* __restrict__ keys, int curve_bits,
                                                     const double* __restrict__ vx, int nv,
                                                     int* __restrict__ items, int* __restrict__ guide) {
    const unsigned long long mask = (1ull << curve_bits) - 1;
    for (int v = int(blockIdx.x) * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        const int set = vset[v];
        const int4 sk = skips[set];
        if (sk.x < 0) continue;   // a flat set has no cells
        const int* b = starts + int64_t(set) * stride;
        int lev = stride - 1;
        while (b[lev] > v) --lev;
        const bool first_tet = v == sk.x || v == sk.y || v == sk.z || v == sk.w;
        const int to = base[int64_t(lev) * nsets + set];   // < 0: k_coarse inserts the level
        if (to >= 0) items[to + (v - b[lev])] = first_tet ? -1 : v;
        int lo = lev, hi = b[lev];
        while (lo > 0 && b[lo] == hi) --lo;   // the level before that has points: [b[lo], hi)
        int g;
        if (b[lo] == hi) {
            g = v > hi ? v - 1 : -1;
        } else if (keys) {
            const unsigned long long k = keys[v] & mask;
            int x = b[lo], y = hi;            // the first of [x, y) with key >= k
            while (x < y) {
                const int m = (x + y) >> 1;
                if ((keys[m] & mask) < k) x = m + 1;
                else y = m;
            }
            // Where many vertices there share the key (a cell with far more points than
            // others, see order.cu), the place at the same fraction of them.
            const int far = 2 * kGuideReach;
            if (x + far < hi && (keys[x + far] & mask) == k) {
                auto bound = [&](int from, int to, bool upper) {   // of k among the keys [from, to)
                    while (from < to) {
                        const int m = (from + to) >> 1;
                        const unsigned long long q = keys[m] & mask;
                        if (q < k || (upper && q == k)) from = m + 1;
                        else to = m;
                    }
                    return from;
                };
                const int own0 = bound(hi, v, false), own1 = bound(v, b[lev + 1], true);   // (the last level's end
                                                                                             // is the next set's start)
                x += int(double(v - own0) / double(own1 - own0) * double(bound(x, hi, true) - x));
            }
            // The nearest of the kGuideReach vertices before and after it there.
            const Pt p = vpt(vx, v);
            double best = 1e300;
            g = min(x, hi - 1);
            for (int u = max(b[lo], x - kGuideReach); u < min(hi, x + kGuideReach); ++u) {
                const Pt w = vpt(vx, u);
                const double dx = w.x - p.x, dy = w.y - p.y, dz = w.z - p.z, d = dx * dx + dy * dy + dz * dz;
                if (d < best) {
                    best = d;
                    g = u;
                }
            }
        } else {
            const int end = lev + 1 < stride ? b[lev + 1] : v + 1;
            g = b[lo] + int(double(v - hi) / double(max(end - hi, 1)) * double(hi - b[lo]));
            g = min(g, hi - 1);
        }
        guide[v] = g;
    }
}

/// Launches one insertion kernel (0: k_cavity, 1: k_check, 2: k_restar) over
/// `n` worker slots with G lanes per worker.
template <int G>
void launch_insertion_t(int which, const Tables& T, const Workers& W, const Round& R, const double* vx, int n,
                        cudaStream_t s) {
    const unsigned grid = unsigned((int64_t(n) * G + 127) / 128);
    if (which == 0) k_cavity<G><<<grid, 128, 0, s>>>(T, W, R, vx, 0);
    else if (which == 1) k_check<G><<<grid, 128, 0, s>>>(T, W, R, 0);
    else k_restar<G><<<grid, 128, 0, s>>>(T, W, R, 0);
}

void launch_insertion(int lanes, int which, const Tables& T, const Workers& W, const Round& R, const double* vx,
                      cudaStream_t s) {
    switch (lanes) {
        case 4: launch_insertion_t<4>(which, T, W, R, vx, W.n, s); break;
        case 8: launch_insertion_t<8>(which, T, W, R, vx, W.n, s); break;
        case 16: launch_insertion_t<16>(which, T, W, R, vx, W.n, s); break;
        default: launch_insertion_t<32>(which, T, W, R, vx, W.n, s); break;
    }
}


/// Lists the parked workers (for the big rounds).
__global__ void k_collect_parked(Workers W, int* list, int* count) {
    const int w = int(blockIdx.x) * blockDim.x + threadIdx.x;
    if (w >= W.n) return;
    if (W.parked[w] && W.cur[w] >= 0) list[atomicAdd(count, 1)] = w;
}

/// One set's share of a level: vertices [lb, le) (global ids) inserted by
/// workers [w0, w0 + count) with chunks of `chunk`; [plb, ple) is the set's
/// previous level.
struct LevelDesc {
    int set, lb, le, chunk, plb, ple, w0;
};

/// Workers of one level, one chunk each.  Each starts at a scattered offset
/// inside its chunk: chunks that are neighbours along the curve are mirror
/// images of each other, and workers walking them in step would reach their
/// common boundary together and keep colliding.
__global__ void k_setup_level(Workers W, const LevelDesc* __restrict__ ds, int nds) {
    const int w = int(blockIdx.x) * blockDim.x + threadIdx.x;
    if (w >= W.n) return;
    int lo = 0, hi = nds - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (ds[mid].w0 <= w) lo = mid;
        else hi = mid - 1;
    }
    const LevelDesc d = ds[lo];
    const int lw = w - d.w0;
    const int b = d.lb + lw * d.chunk;
    const int e = min(d.le, b + d.chunk);
    const int len = e - b;
    const int off = len > 0 ? int((uint32_t(lw) * 2654435761u >> 7) % uint32_t(len)) : 0;
    W.beg[w] = b;
    W.end[w] = e;
    W.pos[w] = off;
    W.left[w] = len;
    W.nwon[w] = 0;
    W.parked[w] = 0;
    W.last[w] = -1;
    W.wset[w] = d.set;
    next_point(W, w);
    // The previous level is ordered along the same curve: the same fraction
    // along it lands near this worker's first point.
    int g = W.skips[d.set].x;
    if (d.ple > d.plb) {
        const double frac = (double(lw) * d.chunk + off) / double(d.le - d.lb);
        g = d.plb + int(frac * double(d.ple - d.plb));
        if (g >= d.ple) g = d.ple - 1;
    }
    W.guide[w] = g;
    W.state[w] = WS_DONE;
}

// ---- growing the worker pool within a level ------------------------------------------
//
// A level's workers are sized for the points its set had when the level began;
// by its end the set has 8 times as many.  Once a set's inserted points call
// for twice its current workers, every worker of that set with enough of its
// chunk left hands the second half of what remains to a new worker.

struct SplitState {
    int* set_p0;     // per set: points inserted before the level
    int* set_ins;    // per set: points inserted so far in the level
    int* set_w;      // per set: current workers
    int* set_split;  // per set: split this time
    int* nworkers;   // the pool size (device copy of W.n)
    int cap;         // worker slots allocated
};

__global__ void k_count_wins(Workers W, SplitState S) {
    const int w = int(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool ok = w < W.n;
    const int set = ok ? W.wset[w] : -1;
    const int c = ok ? W.nwon[w] : 0;
    // Lanes of one set add once per warp.
    const unsigned m = __match_any_sync(__activemask(), set);
    const int sum = int(__reduce_add_sync(m, unsigned(c)));
    if (ok && (threadIdx.x & 31) == __ffs(int(m)) - 1 && sum) atomicAdd(S.set_ins + set, sum);
}

__global__ void k_plan_split(SplitState S, int nsets, double alpha) {
    for (int s = int(blockIdx.x) * blockDim.x + threadIdx.x; s < nsets; s += gridDim.x * blockDim.x) {
        const double p = double(S.set_p0[s]) + double(S.set_ins[s]);
        S.set_split[s] = (S.set_w[s] > 0 && p / alpha >= 2.0 * S.set_w[s]) ? 1 : 0;
        S.set_ins[s] = 0;
    }
}

__global__ void k_split(Workers W, SplitState S, int n_before) {
    const int w = int(blockIdx.x) * blockDim.x + threadIdx.x;
    if (w >= n_before) return;
    const int set = W.wset[w];
    if (!S.set_split[set] || W.cur[w] < 0 || W.parked[w] || W.left[w] < 2 * 16) return;
    const int slot = atomicAdd(S.nworkers, 1);
    if (slot >= S.cap) return;
    const int len = W.end[w] - W.beg[w];
    const int left = W.left[w];
    const int give = left - left / 2;
    W.beg[slot] = W.beg[w];
    W.end[slot] = W.end[w];
    W.pos[slot] = (W.pos[w] + left / 2) % len;
    W.left[slot] = give;
    W.left[w] = left / 2;
    W.nwon[slot] = 0;
    W.parked[slot] = 0;
    W.last[slot] = W.last[w];
    W.guide[slot] = W.guide[w];
    W.wset[slot] = set;
    W.state[slot] = WS_DONE;
    next_point(W, slot);
    atomicAdd(S.set_w + set, 1);
}

// ---- set-up: validation, duplicates, initial tet ----------------------------------

/// The set holding position g: off[s] <= g < off[s+1].
__device__ __forceinline__ int set_of(const int64_t* __restrict__ off, int nsets, int64_t g) {
    int lo = 0, hi = nsets - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

/// Global index of the input point at rank r (position r of its set's order).
__device__ __forceinline__ int64_t point_at(const int32_t* __restrict__ order, const int64_t* __restrict__ off,
                                            int nsets, int64_t r) {
    return off[set_of(off, nsets, r)] + order[r];
}

/// Coordinate bit patterns (with -0.0 folded onto +0.0, which compare equal)
/// of the point at each rank, for the duplicate grouping; axis 3 = the set.
__global__ void k_coord_keys(const double* __restrict__ xyz, const int32_t* __restrict__ order,
                             const int64_t* __restrict__ off, int nsets, int64_t n, int axis,
                             unsigned long long* __restrict__ keys, const int32_t* __restrict__ ranks) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * blockDim.x) {
        if (axis == 3) {
            keys[i] = (unsigned long long)set_of(off, nsets, ranks[i]);
            continue;
        }
        const double x = xyz[3 * point_at(order, off, nsets, ranks[i]) + axis];
        keys[i] = x == 0.0 ? 0ull : (unsigned long long)__double_as_longlong(x);
    }
}

__device__ __forceinline__ bool same_point(const double* xyz, int64_t i, int64_t j) {
    const double* a = xyz + 3 * i;
    const double* b = xyz + 3 * j;
    return a[0] == b[0] && a[1] == b[1] && a[2] == b[2];
}

/// Over ranks sorted by (set, coordinates), ties by rank: flags the first rank
/// of each group of equal points of one set and records the group's
/// representative, the point with the LAST rank (src/triangulation.cpp:77-81),
/// as an index local to its set.
__global__ void k_groups(const double* __restrict__ xyz, const int32_t* __restrict__ order,
                         const int64_t* __restrict__ off, int nsets, const int32_t* __restrict__ sranks,
                         int64_t n, int32_t* __restrict__ first, int32_t* __restrict__ rep_at_first,
                         int* ndup) {
    for (int64_t s = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; s < n;
         s += int64_t(gridDim.x) * blockDim.x) {
        const int32_t r = sranks[s];
        const int set = set_of(off, nsets, r);
        const int64_t pr = off[set] + order[r];
        auto same = [&](int64_t t) {
            const int32_t rt = sranks[t];
            const int st = set_of(off, nsets, rt);
            return st == set && same_point(xyz, off[st] + order[rt], pr);
        };
        if (s > 0 && same(s - 1)) {
            first[r] = 0;
            atomicAdd(ndup, 1);
            continue;
        }
        int64_t e = s;
        while (e + 1 < n && same(e + 1)) ++e;
        first[r] = 1;
        rep_at_first[r] = order[sranks[e]];
    }
}

/// Vertex records: coordinates, the input index (local to the set) the vertex
/// stands for, and its set.
__global__ void k_vertices(const double* __restrict__ xyz, const int32_t* __restrict__ order,
                           const int64_t* __restrict__ off, int nsets,
                           const int32_t* __restrict__ first, const int32_t* __restrict__ vid_of_rank,
                           const int32_t* __restrict__ rep_at_first, int64_t n, bool dups,
                           double* __restrict__ vx, int32_t* __restrict__ vert_point,
                           int32_t* __restrict__ vset) {
    for (int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; r < n;
         r += int64_t(gridDim.x) * blockDim.x) {
        if (dups && !first[r]) continue;
        const int32_t v = dups ? vid_of_rank[r] : int32_t(r);
        const int set = set_of(off, nsets, r);
        const int64_t i = off[set] + order[r];
        reinterpret_cast<double2*>(vx)[2 * int64_t(v)] = make_double2(xyz[3 * i], xyz[3 * i + 1]);
        reinterpret_cast<double2*>(vx)[2 * int64_t(v) + 1] = make_double2(xyz[3 * i + 2], 0.0);
        vert_point[v] = dups ? rep_at_first[r] : order[r];
        vset[v] = set;
    }
}

/// Vertex records in the build's own order (own_order_sets): as k_vertices.
__global__ void k_own_vertices(const double* __restrict__ xyz, const int32_t* __restrict__ vert,
                               const int32_t* __restrict__ rep, const int64_t* __restrict__ off, int nsets,
                               int64_t nv, double* __restrict__ vx, int32_t* __restrict__ vert_point,
                               int32_t* __restrict__ vset) {
    for (int64_t v = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; v < nv; v += int64_t(gridDim.x) * blockDim.x) {
        const int64_t g = vert[v];
        const int set = nsets > 1 ? set_of(off, nsets, g) : 0;
        reinterpret_cast<double2*>(vx)[2 * v] = make_double2(xyz[3 * g], xyz[3 * g + 1]);
        reinterpret_cast<double2*>(vx)[2 * v + 1] = make_double2(xyz[3 * g + 2], 0.0);
        vert_point[v] = rep ? rep[v] : int32_t(g - off[set]);
        vset[v] = set;
    }
}

/// voff[s] = the first vertex of set s, from the starts of its levels.
__global__ void k_own_voff(const int32_t* __restrict__ level_start, int nsets, int levels,
                           int32_t* __restrict__ voff) {
    for (int s = int(blockIdx.x) * blockDim.x + threadIdx.x; s <= nsets; s += gridDim.x * blockDim.x)
        voff[s] = level_start[int64_t(s) * levels];
}

/// Per set, one warp: the first vertex (in insertion order) not collinear with its
/// first two, and then the first not coplanar with those three, looked for among
/// its first kFirstLook vertices, where nearly every set has them; raises `more`
/// for a set that has not (the next two kernels, one thread per vertex, then look
/// through all; they took 574 us for 256 sets of 1.9 M points).
constexpr int kFirstLook = 1024;
__global__ void __launch_bounds__(128) k_first_four(const double* __restrict__ vx, const int32_t* __restrict__ voff,
                                                    int nsets, int* found2, int* found3, int* more, uint32_t* st) {
    const int set = int((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = int(threadIdx.x & 31u);
    if (set >= nsets) return;
    const int base = voff[set], end = voff[set + 1], last = min(end, base + kFirstLook);
    int v2 = INT_MAX, v3 = INT_MAX;
    for (int v0 = base + 2; v0 < last && v2 == INT_MAX; v0 += 32) {
        const int v = v0 + lane;
        const bool hit = v < last && !collinear(vpt(vx, base), vpt(vx, base + 1), vpt(vx, v), st);
        const unsigned m = __ballot_sync(kFull, hit);
        if (m) v2 = v0 + __ffs(int(m)) - 1;
    }
    for (int v0 = base + 2; v0 < last && v2 != INT_MAX && v3 == INT_MAX; v0 += 32) {
        const int v = v0 + lane;
        const bool hit = v < last && v != v2 &&
                         orient3d(vpt(vx, base), vpt(vx, base + 1), vpt(vx, v2), vpt(vx, v), st) != 0;
        const unsigned m = __ballot_sync(kFull, hit);
        if (m) v3 = v0 + __ffs(int(m)) - 1;
    }
    if (lane == 0) {
        if (v2 != INT_MAX) found2[set] = v2;
        if (v3 != INT_MAX) found3[set] = v3;
        if (v3 == INT_MAX && end > last) atomicOr(more, 1);
    }
}

/// The same over all vertices, for the sets k_first_four has not settled.
__global__ void k_find_noncollinear(const double* __restrict__ vx, int nv, const int32_t* __restrict__ vset,
                                    const int32_t* __restrict__ voff, int* found, const int* __restrict__ more,
                                    uint32_t* st) {
    if (*more == 0) return;
    for (int v = int(blockIdx.x) * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        const int set = vset[v], base = voff[set];
        if (v - base < 2 || v > found[set]) continue;
        if (!collinear(vpt(vx, base), vpt(vx, base + 1), vpt(vx, v), st)) atomicMin(found + set, v);
    }
}

__global__ void k_find_noncoplanar(const double* __restrict__ vx, int nv, const int32_t* __restrict__ vset,
                                   const int32_t* __restrict__ voff, const int* found2, int* found3,
                                   const int* __restrict__ more, uint32_t* st) {
    if (*more == 0) return;
    for (int v = int(blockIdx.x) * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        const int set = vset[v], base = voff[set], v2 = found2[set];
        if (v2 >= voff[set + 1] || v - base < 2 || v == v2 || v > found3[set]) continue;
        if (orient3d(vpt(vx, base), vpt(vx, base + 1), vpt(vx, v2), vpt(vx, v), st) != 0)
            atomicMin(found3 + set, v);
    }
}

/// Per set: its first four vertices (or -1s when the set is flat: no cells,
/// src/triangulation.cpp:943-949).
__global__ void k_set_skips(const int32_t* __restrict__ voff, const int* found2, const int* found3,
                            int nsets, int4* __restrict__ skips) {
    for (int s = int(blockIdx.x) * blockDim.x + threadIdx.x; s < nsets; s += gridDim.x * blockDim.x) {
        const int base = voff[s], end = voff[s + 1];
        if (end - base >= 4 && found2[s] < end && found3[s] < end)
            skips[s] = make_int4(base, base + 1, found2[s], found3[s]);
        else
            skips[s] = make_int4(-1, -1, -1, -1);
    }
}

/// One thread per set: the first tet and its four infinite neighbours, in
/// slots 5s .. 5s+4.
__global__ void k_init_tets(Tables T, const double* __restrict__ vx, const int4* __restrict__ skips,
                            int nsets, uint32_t* st) {
    for (int set = int(blockIdx.x) * blockDim.x + threadIdx.x; set < nsets; set += gridDim.x * blockDim.x) {
        const int4 sk = skips[set];
        if (sk.x < 0) continue;
        int v0 = sk.x, v1 = sk.y;
        const int v2 = sk.z, v3 = sk.w;
        if (orient3d(vpt(vx, v0), vpt(vx, v1), vpt(vx, v2), vpt(vx, v3), st) < 0) {
            const int t = v0;
            v0 = v1;
            v1 = t;
        }
        int4 tv[5];
        tv[0] = make_int4(v0, v1, v2, v3);
        for (int i = 0; i < 4; ++i) {
            // Facet i of the first tet, capped by the infinite vertex in slot i
            // and two other slots swapped, so the cap is positively oriented.
            int4 c = tv[0];
            set_at(c, i, kInf);
            const int a = (i + 1) & 3, b = (i + 2) & 3;
            const int x = at(c, a);
            set_at(c, a, at(c, b));
            set_at(c, b, x);
            tv[1 + i] = c;
        }
        const int base = 5 * set;
        int4 tn[5];
        for (int t = 0; t < 5; ++t)
            for (int f = 0; f < 4; ++f) {
                int fv[3], w = 0;
                for (int m = 0; m < 4; ++m)
                    if (m != f) fv[w++] = at(tv[t], m);
                for (int u = 0; u < 5; ++u) {
                    if (u == t) continue;
                    for (int g = 0; g < 4; ++g) {
                        int hits = 0;
                        for (int m = 0; m < 4; ++m) {
                            if (m == g) continue;
                            const int x = at(tv[u], m);
                            hits += (x == fv[0]) + (x == fv[1]) + (x == fv[2]);
                        }
                        if (hits == 3) set_at(tn[t], f, (base + u) * 4 + g);
                    }
                }
            }
        for (int t = 0; t < 5; ++t) {
            T.tv(base + t) = tv[t];
            T.tn(base + t) = tn[t];
            if (T.lock) T.lock[base + t] = 0;
        }
        T.vert_tet[v0] = base;
        T.vert_tet[v1] = base;
        T.vert_tet[v2] = base;
        T.vert_tet[v3] = base;
    }
}

// ---- output -----------------------------------------------------------------------

/// Even permutation bringing the smallest index to slot 0, then the cyclic
/// rotation of the other three that puts their smallest first.
__device__ __forceinline__ int4 canonical(int4 t) {
    int m = 0;
    int mv = t.x;
    if (t.y < mv) { m = 1; mv = t.y; }
    if (t.z < mv) { m = 2; mv = t.z; }
    if (t.w < mv) { m = 3; mv = t.w; }
    if (m == 1) t = make_int4(t.y, t.x, t.w, t.z);
    else if (m == 2) t = make_int4(t.z, t.w, t.x, t.y);
    else if (m == 3) t = make_int4(t.w, t.z, t.y, t.x);
    if (t.z < t.y && t.z < t.w) t = make_int4(t.x, t.z, t.w, t.y);
    else if (t.w < t.y && t.w < t.z) t = make_int4(t.x, t.w, t.y, t.z);
    return t;
}

__global__ void k_cell_flags(const int4* __restrict__ rec, int ntet,
                             bool with_infinite, int32_t* __restrict__ flag) {
    for (int t = int(blockIdx.x) * blockDim.x + threadIdx.x; t < ntet; t += gridDim.x * blockDim.x) {
        const int4 c = rec[2 * int64_t(t)];
        flag[t] = c.x != c.y && (with_infinite || inf_pos(c) < 0) ? 1 : 0;
    }
}

/// Writes the flagged tets, mapped to input point indices and canonicalised,
/// plus their sort keys (shifted by one so the infinite vertex, -1,
/// is 0).
__global__ void k_cells_out(const int4* __restrict__ rec, const int32_t* __restrict__ flag,
                            const int32_t* __restrict__ pos, int ntet,
                            const int32_t* __restrict__ vert_point, const int32_t* __restrict__ vset,
                            int kbits, int4* __restrict__ cells,
                            unsigned long long* __restrict__ khi, unsigned long long* __restrict__ klo,
                            int32_t* __restrict__ idx, int32_t* __restrict__ cset) {
    for (int t = int(blockIdx.x) * blockDim.x + threadIdx.x; t < ntet; t += gridDim.x * blockDim.x) {
        if (!flag[t]) continue;
        const int4 c = rec[2 * int64_t(t)];
        if (cset) cset[pos[t]] = vset[c.x != kInf ? c.x : c.y];
        int4 q;
        q.x = c.x == kInf ? -1 : vert_point[c.x];
        q.y = c.y == kInf ? -1 : vert_point[c.y];
        q.z = c.z == kInf ? -1 : vert_point[c.z];
        q.w = c.w == kInf ? -1 : vert_point[c.w];
        q = canonical(q);
        const int o = pos[t];
        cells[o] = q;
        khi[o] = ((unsigned long long)(uint32_t(q.x + 1)) << kbits) | uint32_t(q.y + 1);
        klo[o] = ((unsigned long long)(uint32_t(q.z + 1)) << kbits) | uint32_t(q.w + 1);
        idx[o] = o;
    }
}

// ---- canonical order of the finite cells by buckets ---------------------------------
//
// A canonical cell leads with its smallest vertex, so the lexicographic order
// is: by that vertex, then by the other three.  The cells are bucketed by the
// global index of their first vertex (set offset + local index; the sets are
// contiguous, so this also orders them by set) with a counting sort, then each
// bucket - the few cells whose smallest vertex is that point - is sorted by its
// other three vertices.

/// Buckets of up to kBucketThread cells are sorted many to a block, one block sorts one of up
/// to kBucketBlock; a larger bucket leaves the whole output to the radix sort.
constexpr int kBucketThread = 32;
constexpr int kBucketBlock = 2048;

/// The finite cells, mapped to input indices and canonicalised, in any order, with
/// their buckets, which it also counts.  Each block packs the cells of
/// kEmitTets tet slots behind one another (one atomic for their place), so the
/// slots are read once and no flags or scan over them are needed.  Bound by the
/// gathers of the vertices' input indices and the bucket counts, one atomic a cell.
constexpr int kEmitThreads = 256, kEmitItems = 8, kEmitTets = kEmitThreads * kEmitItems;
__global__ void __launch_bounds__(kEmitThreads) k_cells_emit(const int4* __restrict__ rec, int ntet,
                                                             const int32_t* __restrict__ vert_point,
                                                             const int32_t* __restrict__ vset,
                                                             const int64_t* __restrict__ off, bool sets,
                                                             int4* __restrict__ cells, int* __restrict__ bucket,
                                                             int* __restrict__ count, int* total) {
    typedef cub::BlockScan<int, kEmitThreads> BlockScan;
    __shared__ typename BlockScan::TempStorage tmp;
    __shared__ int base;
    int4 q[kEmitItems];
    unsigned mask = 0;
    const int first = int(blockIdx.x) * kEmitTets + int(threadIdx.x);
#pragma unroll
    for (int k = 0; k < kEmitItems; ++k) {
        const int t = first + k * kEmitThreads;
        q[k] = t < ntet ? rec[2 * int64_t(t)] : make_int4(0, 0, 0, 0);
        if (q[k].x != q[k].y && inf_pos(q[k]) < 0) mask |= 1u << k;
    }
    int at_ = 0, sum = 0;
    BlockScan(tmp).ExclusiveSum(__popc(mask), at_, sum);
    if (threadIdx.x == 0) base = atomicAdd(total, sum);
    __syncthreads();
    int o = base + at_;
#pragma unroll
    for (int k = 0; k < kEmitItems; ++k) {
        if (!(mask >> k & 1u)) continue;
        const int4 c = q[k];
        const int4 w = canonical(make_int4(vert_point[c.x], vert_point[c.y], vert_point[c.z], vert_point[c.w]));
        const int b = (sets ? int(off[vset[c.x]]) : 0) + w.x;
        cells[o] = w;
        bucket[o] = b;
        atomicAdd(count + b, 1);
        ++o;
    }
}

/// Puts every cell in its bucket; `count` runs down to zero again.
__global__ void k_bucket_place(const int4* __restrict__ cells, const int* __restrict__ bucket,
                               const int* __restrict__ total, const int* __restrict__ start, int* __restrict__ count,
                               int4* __restrict__ out) {
    const int n = *total;
    for (int i = int(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int b = bucket[i];
        out[start[b] + atomicSub(count + b, 1) - 1] = cells[i];
    }
}

__device__ __forceinline__ bool cell_tail_less(const int4& a, const int4& b) {
    if (a.y != b.y) return a.y < b.y;
    if (a.z != b.z) return a.z < b.z;
    return a.w < b.w;
}

/// Sorts the buckets of up to kBucketThread cells by the last three vertices, 128
/// buckets a block: the block loads their cells in order into shared memory, and
/// each cell, one thread each, counts the cells of its bucket that come before it
/// and goes to that place.  All cells do about the same work, where a thread that
/// sorts a bucket by itself keeps its warp waiting for the largest (664 us in
/// place in device memory for 11.4 M cells, 1056 us in shared memory).  A bucket of
/// more cells is listed in `mid` for k_bucket_sort_block, one of more than
/// kBucketBlock only raises `big`.
constexpr int kBucketStage = 1024;
__global__ void __launch_bounds__(128) k_bucket_sort(int4* __restrict__ cells, const int* __restrict__ start, int nb,
                                                     int* __restrict__ mid, int* __restrict__ nmid,
                                                     int* __restrict__ big) {
    __shared__ int4 stage[kBucketStage];
    __shared__ int lo_of[129];
    __shared__ uint8_t owner[kBucketStage];
    const int b0 = int(blockIdx.x) * 128, nbuckets = min(128, nb - b0);
    for (int k = int(threadIdx.x); k <= nbuckets; k += 128) lo_of[k] = start[b0 + k];
    __syncthreads();
    if (int(threadIdx.x) < nbuckets) {
        const int n = lo_of[threadIdx.x + 1] - lo_of[threadIdx.x];
        if (n > kBucketBlock) *big = 1;
        else if (n > kBucketThread) mid[atomicAdd(nmid, 1)] = b0 + int(threadIdx.x);
    }
    // Whole buckets, as many as fit the stage, at a time.
    for (int k0 = 0; k0 < nbuckets;) {
        int k1 = k0;
        while (k1 < nbuckets && lo_of[k1 + 1] - lo_of[k0] <= kBucketStage) ++k1;
        if (k1 == k0) {          // one bucket beyond the stage: listed above
            ++k0;
            continue;
        }
        const int first = lo_of[k0], n = lo_of[k1] - first;
        for (int i = int(threadIdx.x); i < n; i += 128) stage[i] = cells[first + i];
        if (int(threadIdx.x) >= k0 && int(threadIdx.x) < k1)
            for (int i = lo_of[threadIdx.x] - first; i < lo_of[threadIdx.x + 1] - first; ++i)
                owner[i] = uint8_t(threadIdx.x);
        __syncthreads();
        for (int i = int(threadIdx.x); i < n; i += 128) {
            const int k = owner[i], lo = lo_of[k] - first, hi = lo_of[k + 1] - first;
            if (hi - lo < 2 || hi - lo > kBucketThread) continue;
            const int4 x = stage[i];
            int rank = lo;
            for (int j = lo; j < hi; ++j) rank += cell_tail_less(stage[j], x) ? 1 : 0;
            cells[first + rank] = x;
        }
        __syncthreads();
        k0 = k1;
    }
}

/// One block per listed bucket: a bitonic sort by the last three vertices in
/// shared memory (padded to a power of two with cells that sort last).
__global__ void __launch_bounds__(512) k_bucket_sort_block(int4* __restrict__ cells, const int* __restrict__ start,
                                                           const int* __restrict__ mid) {
    __shared__ int4 sh[kBucketBlock];
    const int b = mid[blockIdx.x];
    const int lo = start[b], n = start[b + 1] - lo;
    int m = 1;
    while (m < n) m <<= 1;
    const int4 pad = make_int4(INT_MAX, INT_MAX, INT_MAX, INT_MAX);
    for (int i = int(threadIdx.x); i < m; i += blockDim.x) sh[i] = i < n ? cells[lo + i] : pad;
    __syncthreads();
    for (int k = 2; k <= m; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = int(threadIdx.x); i < m; i += blockDim.x) {
                const int l = i ^ j;
                if (l > i) {
                    const bool up = (i & k) == 0;
                    const int4 a = sh[i], c = sh[l];
                    if (cell_tail_less(c, a) == up) {
                        sh[i] = c;
                        sh[l] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
    for (int i = int(threadIdx.x); i < n; i += blockDim.x) cells[lo + i] = sh[i];
}

/// cell_off[s] = the first bucket of set s.
__global__ void k_cell_off(const int* __restrict__ start, const int64_t* __restrict__ off, int nsets,
                           int64_t* __restrict__ cell_off) {
    for (int s = int(blockIdx.x) * blockDim.x + threadIdx.x; s <= nsets; s += gridDim.x * blockDim.x)
        cell_off[s] = start[off[s]];
}

__global__ void k_gather_cells(const int4* __restrict__ in, const int32_t* __restrict__ idx, int64_t n,
                               int4* __restrict__ out) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * blockDim.x)
        out[i] = in[idx[i]];
}

__global__ void k_incident_pairs(const int4* __restrict__ cells, int64_t nc, int32_t* __restrict__ pt,
                                 int32_t* __restrict__ cell, int32_t* __restrict__ count) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < nc;
         i += int64_t(gridDim.x) * blockDim.x) {
        const int4 c = cells[i];
        const int v[4] = {c.x, c.y, c.z, c.w};
        for (int k = 0; k < 4; ++k) {
            pt[4 * i + k] = v[k];
            cell[4 * i + k] = int32_t(i);
            atomicAdd(count + v[k], 1);
        }
    }
}

__global__ void k_set_int(int* p, int v) { *p = v; }

__global__ void k_gather_u64(const unsigned long long* __restrict__ in, const int32_t* __restrict__ ix,
                             int64_t m, unsigned long long* __restrict__ o) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < m;
         i += int64_t(gridDim.x) * blockDim.x)
        o[i] = in[ix[i]];
}

__global__ void k_gather_i32(const int32_t* __restrict__ in, const int32_t* __restrict__ ix, int64_t m,
                             int32_t* __restrict__ o) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < m;
         i += int64_t(gridDim.x) * blockDim.x)
        o[i] = in[ix[i]];
}

__global__ void k_iota32(int32_t* __restrict__ a, int64_t m) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < m;
         i += int64_t(gridDim.x) * blockDim.x)
        a[i] = int32_t(i);
}

__global__ void k_widen(const int32_t* __restrict__ a, int64_t m, int64_t* __restrict__ o) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < m;
         i += int64_t(gridDim.x) * blockDim.x)
        o[i] = a[i];
}

}  // namespace

namespace {

__global__ void k_voff(const int64_t* __restrict__ off, int nsets, const int32_t* __restrict__ vid, bool dups,
                       int64_t n, int nv, int32_t* __restrict__ voff) {
    for (int s = int(blockIdx.x) * blockDim.x + threadIdx.x; s <= nsets; s += gridDim.x * blockDim.x) {
        const int64_t o = off[s];
        voff[s] = o >= n ? nv : (dups ? vid[o] : int32_t(o));
    }
}

/// Sorts `n` canonical cells lexicographically - by set first when `cset` is
/// given - into `out` (keys prepared by k_cells_out).
int sort_cells(DevBuf<int4>& cells, DevBuf<unsigned long long>& khi, DevBuf<unsigned long long>& klo,
               DevBuf<int32_t>& idx, const int32_t* cset, int nsets, int64_t n, int kbits,
               DevBuf<int4>& out, cudaStream_t s) {
    D3G_TRY(out.alloc(size_t(n), s));
    if (n == 0) return D3G_OK;
    DevBuf<unsigned long long> k2, kg;
    DevBuf<int32_t> i2;
    D3G_TRY(k2.alloc(size_t(n), s));
    D3G_TRY(kg.alloc(size_t(n), s));
    D3G_TRY(i2.alloc(size_t(n), s));
    // LSD: low half, then the high half, then (several sets) the set - each stable.
    D3G_TRY(sort_pairs(klo.p, k2.p, idx.p, i2.p, n, 0, 2 * kbits, s));
    k_gather_u64<<<grid_for(n, 256), 256, 0, s>>>(khi.p, i2.p, n, kg.p);
    D3G_TRY(sort_pairs(kg.p, k2.p, i2.p, idx.p, n, 0, 2 * kbits, s));
    if (cset) {
        DevBuf<int32_t> sk, sk2;
        D3G_TRY(sk.alloc(size_t(n), s));
        D3G_TRY(sk2.alloc(size_t(n), s));
        k_gather_i32<<<grid_for(n, 256), 256, 0, s>>>(cset, idx.p, n, sk.p);
        D3G_TRY(sort_pairs(sk.p, sk2.p, idx.p, i2.p, n, 0, bits_for(uint64_t(nsets)), s));
        idx.swap(i2);
    }
    k_gather_cells<<<grid_for(n, 256), 256, 0, s>>>(cells.p, idx.p, n, out.p);
    D3G_CUDA(cudaGetLastError());
    return D3G_OK;
}

}  // namespace

int build_sets_impl(const double* d_xyz, const int64_t* h_off, int nsets, const d3g_options& opt,
                    cudaStream_t s, DeviceResult& R);

/// A non-blocking stream of the calling thread for the current device; it lives
/// as long as the thread, so buffers bound to it can be freed at any later time.
cudaStream_t internal_stream() {
    thread_local cudaStream_t streams[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (!streams[dev] && cudaStreamCreateWithFlags(&streams[dev], cudaStreamNonBlocking) != cudaSuccess)
        streams[dev] = nullptr;
    return streams[dev];
}

/// Runs the build on `s`, or - for the legacy default stream, which cannot be
/// captured into a graph - on the thread's internal stream, after the legacy
/// stream's prior work (the build synchronises its stream before returning).
int build_on_stream(const double* d_xyz, const int64_t* h_off, int nsets, const d3g_options& opt,
                    cudaStream_t s, DeviceResult& R) {
    D3G_TRY(prepare_device());
    if (s != nullptr && s != cudaStreamLegacy) return build_sets_impl(d_xyz, h_off, nsets, opt, s, R);
    cudaStream_t own = internal_stream();
    if (!own) {
        set_error("d3g_build: could not create a stream");
        return D3G_ERR_CUDA;
    }
    cudaEvent_t ev;
    D3G_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    cudaEventRecord(ev, cudaStreamLegacy);
    cudaStreamWaitEvent(own, ev, 0);
    cudaEventDestroy(ev);
    return build_sets_impl(d_xyz, h_off, nsets, opt, own, R);
}

int build_on_stream(const double* d_xyz, int64_t n, const d3g_options& opt, cudaStream_t s,
                    DeviceResult& R) {
    const int64_t h_off[2] = {0, n};
    return build_on_stream(d_xyz, h_off, 1, opt, s, R);
}

int build_sets_impl(const double* d_xyz, const int64_t* h_off, int nsets, const d3g_options& opt,
                    cudaStream_t s, DeviceResult& R) {
    R.reset();
    const int64_t n = h_off[nsets];
    int64_t max_n = 0;
    for (int i = 0; i < nsets; ++i) {
        if (h_off[i + 1] < h_off[i]) {
            set_error("d3g_build: set offsets must not decrease");
            return D3G_ERR_INVALID_ARGUMENT;
        }
        max_n = std::max<int64_t>(max_n, h_off[i + 1] - h_off[i]);
    }
    R.cell_off.assign(size_t(nsets) + 1, 0);
    R.set_nv.assign(size_t(nsets), 0);
    if (n == 0) return D3G_OK;
    if (n > (int64_t(1) << 27) || h_off[0] != 0) {
        set_error("d3g_build: at most 2^27 points per call, offsets starting at 0");
        return D3G_ERR_INVALID_ARGUMENT;
    }
    if (opt.level_growth != 0 && (opt.level_growth < 2 || opt.level_growth > 8)) {
        set_error("d3g_build: level_growth must be 0 or 2-8");
        return D3G_ERR_INVALID_ARGUMENT;
    }
    const bool single = nsets == 1;
    const int N = int(n);
    // Asynchronous insertion (k_insert_groups), or lockstep rounds only.
    const bool use_async = opt.schedule != 1 && !(opt.chunk <= 0 && opt.split != 0);
    DevBuf<uint32_t> status;
    DevBuf<int64_t> d_off;
    D3G_TRY(status.alloc(4, s));
    D3G_TRY(d_off.alloc(size_t(nsets) + 1, s));
    D3G_CUDA(cudaMemsetAsync(status.p, 0, 4 * sizeof(uint32_t), s));
    D3G_CUDA(cudaMemcpyAsync(d_off.p, h_off, sizeof(int64_t) * (size_t(nsets) + 1), cudaMemcpyHostToDevice, s));

    cudaEvent_t ph[4];
    for (auto& e : ph) cudaEventCreate(&e);
    struct PhGuard {
        cudaEvent_t* e;
        ~PhGuard() {
            for (int i = 0; i < 4; ++i) cudaEventDestroy(e[i]);
        }
    } ph_guard{ph};
    cudaEventRecord(ph[0], s);
    NvtxRange nvtx_build("d3g.build");
    std::optional<NvtxRange> nvtx_phase;
    nvtx_phase.emplace("d3g.order");
    // ---- insertion order and duplicate groups ----
    // BRIO levels of the build's own insertion order: each level `growth` times
    // the points before it.  Any order gives the same cells, so the build may
    // take more and shorter levels than the reference's 8: kGroupGrowth in an
    // asynchronous build; in one by rounds alone, 4 when a set's coordinates make
    // the filters exact (lattices and coarse grids, whose long levels collide
    // most) and for a build too small to fill the GPU (whose levels are inserted
    // chunk by chunk, so shorter ones finish sooner).
    int growth = opt.level_growth;
    SetScan scan;
    D3G_TRY(scan_sets(d_xyz, d_off.p, nsets, n, scan, status.p + 1, s));
    // Sets whose coordinates span few grid steps (integer lattices, coarse grids):
    // their filters are exact, so their degenerate queries skip the exact stage.
    DevBuf<uint8_t> set_exact;
    DevBuf<double> inv_grid;
    D3G_TRY(set_exact.alloc(size_t(nsets), s));
    D3G_TRY(inv_grid.alloc(size_t(nsets), s));
    k_set_exact<<<grid_for(nsets, 128), 128, 0, s>>>(scan.span.p, scan.box.p, nsets, set_exact.p, inv_grid.p);
    if (growth == 0 && use_async) growth = kGroupGrowth;
    if (growth == 0) {
        std::vector<uint8_t> hex(static_cast<size_t>(nsets));
        D3G_CUDA(cudaMemcpyAsync(hex.data(), set_exact.p, size_t(nsets), cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaStreamSynchronize(s));
        growth = n < kSmallBuildPoints ? kExactSetGrowth : 8;
        for (const uint8_t e : hex) growth = (e & EX_BOTH) == EX_BOTH ? kExactSetGrowth : growth;
    }
    DevBuf<double> vx;
    DevBuf<int32_t> vert_point, vset, voff;
    int nv = N;
    D3G_TRY(voff.alloc(size_t(nsets) + 1, s));
    // The own order, or - where its keys cannot tell the points apart - the
    // spatial sort with the sorts that find repeated points.
    OwnOrder own;
    D3G_TRY(own_order_sets(d_xyz, h_off, d_off.p, nsets, growth, scan, status.p + 1, own, s));
    std::vector<int32_t> hlevel;   // own order: first vertex of each (set, level)
    if (own.ok) {
        nv = int(own.nv);
        D3G_TRY(vx.alloc(size_t(4) * nv, s));
        D3G_TRY(vert_point.alloc(size_t(nv), s));
        D3G_TRY(vset.alloc(size_t(nv), s));
        k_own_vertices<<<grid_for(nv, 256), 256, 0, s>>>(d_xyz, own.vert.p, own.rep.p, d_off.p, nsets, nv, vx.p,
                                                         vert_point.p, vset.p);
        k_own_voff<<<grid_for(nsets + 1, 128), 128, 0, s>>>(own.level_start.p, nsets, own.levels, voff.p);
        hlevel.resize(size_t(nsets) * size_t(own.levels) + 1);
        D3G_CUDA(cudaMemcpyAsync(hlevel.data(), own.level_start.p, sizeof(int32_t) * hlevel.size(),
                                 cudaMemcpyDeviceToHost, s));
    }
    while (!own.ok) {
        DevBuf<int32_t> order;
        D3G_TRY(order.alloc(size_t(N), s));
        D3G_TRY(spatial_order_sets_device(d_xyz, h_off, d_off.p, nsets, order.p, s, 1.0 / double(growth)));
        DevBuf<int32_t> ranks, sranks, first, rep, vid;
        DevBuf<unsigned long long> keys, keys2;
        DevBuf<int> ndup;
        D3G_TRY(ranks.alloc(size_t(N), s));
        D3G_TRY(sranks.alloc(size_t(N), s));
        D3G_TRY(keys.alloc(size_t(N), s));
        D3G_TRY(keys2.alloc(size_t(N), s));
        D3G_TRY(ndup.alloc(1, s));
        D3G_CUDA(cudaMemsetAsync(ndup.p, 0, sizeof(int), s));
        k_iota32<<<grid_for(n, 256), 256, 0, s>>>(ranks.p, n);
        // LSD over z, y, x (and the set): ranks sorted by (set, coordinates),
        // ties kept in rank order.
        for (int axis = 2; axis >= (single ? 0 : -1); --axis) {
            const int key_axis = axis < 0 ? 3 : axis;
            k_coord_keys<<<grid_for(n, 256), 256, 0, s>>>(d_xyz, order.p, d_off.p, nsets, n, key_axis, keys.p,
                                                          ranks.p);
            D3G_TRY(sort_pairs(keys.p, keys2.p, ranks.p, sranks.p, n, 0,
                               key_axis == 3 ? bits_for(uint64_t(nsets)) : 64, s));
            ranks.swap(sranks);
        }
        D3G_TRY(first.alloc(size_t(N), s));
        D3G_TRY(rep.alloc(size_t(N), s));
        k_groups<<<grid_for(n, 256), 256, 0, s>>>(d_xyz, order.p, d_off.p, nsets, ranks.p, n, first.p, rep.p,
                                                  ndup.p);
        int hdup = 0;
        D3G_CUDA(cudaMemcpyAsync(&hdup, ndup.p, sizeof hdup, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaStreamSynchronize(s));
        if (hdup > 0 && growth != 8) {
            growth = 8;
            continue;
        }
        nv = N - hdup;
        D3G_TRY(vx.alloc(size_t(4) * nv, s));
        D3G_TRY(vert_point.alloc(size_t(nv), s));
        D3G_TRY(vset.alloc(size_t(nv), s));
        if (hdup > 0) {
            D3G_TRY(vid.alloc(size_t(N), s));
            D3G_TRY(exclusive_scan(first.p, vid.p, n, s));
        }
        k_vertices<<<grid_for(n, 256), 256, 0, s>>>(d_xyz, order.p, d_off.p, nsets, first.p, vid.p, rep.p, n,
                                                    hdup > 0, vx.p, vert_point.p, vset.p);
        k_voff<<<grid_for(nsets + 1, 128), 128, 0, s>>>(d_off.p, nsets, vid.p, hdup > 0, n, nv, voff.p);
        D3G_CUDA(cudaGetLastError());
        break;
    }
    const double level_ratio = 1.0 / double(growth);
    R.n_vertices = nv;
    std::vector<int32_t> hvoff(size_t(nsets) + 1);
    D3G_CUDA(cudaMemcpyAsync(hvoff.data(), voff.p, sizeof(int32_t) * hvoff.size(), cudaMemcpyDeviceToHost, s));

    std::vector<uint8_t> hexact(static_cast<size_t>(nsets));
    D3G_CUDA(cudaMemcpyAsync(hexact.data(), set_exact.p, size_t(nsets), cudaMemcpyDeviceToHost, s));
    uint32_t hst[2] = {0, 0};
    D3G_CUDA(cudaMemcpyAsync(hst, status.p, sizeof hst, cudaMemcpyDeviceToHost, s));
    D3G_CUDA(cudaStreamSynchronize(s));
    if (hst[1]) {
        set_error("d3g_build: non-finite coordinate");
        return D3G_ERR_INVALID_INPUT;
    }
    for (int i = 0; i < nsets; ++i) R.set_nv[size_t(i)] = hvoff[size_t(i) + 1] - hvoff[size_t(i)];

    cudaEventRecord(ph[1], s);
    nvtx_phase.reset();
    nvtx_phase.emplace("d3g.insert");
    // ---- each set's first tet: its first four affinely independent vertices ----
    DevBuf<int> found;
    DevBuf<int4> skips;
    D3G_TRY(found.alloc(2 * size_t(nsets) + 1, s));
    D3G_TRY(skips.alloc(size_t(nsets), s));
    D3G_CUDA(cudaMemsetAsync(found.p, 0x7F, 2 * sizeof(int) * size_t(nsets), s));
    int* more = found.p + 2 * size_t(nsets);
    D3G_CUDA(cudaMemsetAsync(more, 0, sizeof(int), s));
    k_first_four<<<unsigned((int64_t(nsets) * 32 + 127) / 128), 128, 0, s>>>(vx.p, voff.p, nsets, found.p,
                                                                            found.p + nsets, more, status.p);
    k_find_noncollinear<<<grid_for(nv, 256), 256, 0, s>>>(vx.p, nv, vset.p, voff.p, found.p, more, status.p);
    k_find_noncoplanar<<<grid_for(nv, 256), 256, 0, s>>>(vx.p, nv, vset.p, voff.p, found.p, found.p + nsets, more,
                                                         status.p);
    k_set_skips<<<grid_for(nsets, 128), 128, 0, s>>>(voff.p, found.p, found.p + nsets, nsets, skips.p);
    std::vector<int4> hskips(static_cast<size_t>(nsets));
    D3G_CUDA(cudaMemcpyAsync(hskips.data(), skips.p, sizeof(int4) * size_t(nsets), cudaMemcpyDeviceToHost, s));
    D3G_CUDA(cudaMemcpyAsync(hst, status.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    D3G_CUDA(cudaStreamSynchronize(s));
    {
        const int st = status_from_bits(hst[0]);
        if (st != D3G_OK) return st;
    }
    bool any_cells = false;
    for (const int4& k : hskips) any_cells = any_cells || k.x >= 0;
    if (!any_cells) {
        // Every set collinear or coplanar: no cells (src/triangulation.cpp:943-949).
        if (single && opt.want_incident) {
            D3G_TRY(R.inc_off.alloc(size_t(N) + 1, s));
            D3G_CUDA(cudaMemsetAsync(R.inc_off.p, 0, sizeof(int64_t) * (size_t(N) + 1), s));
        }
        D3G_CUDA(cudaStreamSynchronize(s));
        return D3G_OK;
    }

    // ---- tables ----
    Tables T;
    const int tets_per_vertex = opt.tet_capacity > 0 ? opt.tet_capacity : 8;
    // (beyond it, room for the slots groups hold without using them: two blocks of
    // kPoolSlots each, at most one group per kPoolSlots vertices)
    int64_t cap64 = int64_t(nv) * tets_per_vertex + 5 * int64_t(nsets) + 4096 +
                    (use_async ? 2 * std::min<int64_t>(nv, int64_t(kMaxGroups) * kPoolSlots) : 0);
    if (cap64 > (int64_t(1) << 29)) cap64 = int64_t(1) << 29;
    T.cap = int(cap64);
    T.walk_limit = opt.walk_limit > 0 ? opt.walk_limit : kWalkLimit;
    DevBuf<int4> rec;
    DevBuf<unsigned long long> claim;
    DevBuf<int> fnew, vert_tet, tet_count, alock;
    D3G_TRY(rec.alloc(2 * size_t(T.cap), s));
    D3G_TRY(vert_tet.alloc(size_t(nv), s));
    D3G_TRY(tet_count.alloc(1, s));
    if (use_async) {
        // A slot without a tet is locked until its first tet is written.
        D3G_TRY(alock.alloc(size_t(T.cap), s));
        D3G_CUDA(cudaMemsetAsync(alock.p, 0xFF, sizeof(int) * size_t(T.cap), s));
    }
    T.lock = alock.p;
    // Every slot holds in-range indices from the start (the asynchronous walk
    // may read a slot before its tet is written), and a vertex not inserted yet
    // has no tet.
    D3G_CUDA(cudaMemsetAsync(rec.p, 0, 2 * sizeof(int4) * size_t(T.cap), s));
    D3G_CUDA(cudaMemsetAsync(vert_tet.p, 0xFF, sizeof(int) * size_t(nv), s));
    T.rec = rec.p;
    T.claim = nullptr;
    T.fnew = nullptr;
    T.vert_tet = vert_tet.p;
    T.tet_count = tet_count.p;
    T.vset = vset.p;
    k_set_int<<<1, 1, 0, s>>>(tet_count.p, 5 * nsets);
    k_init_tets<<<grid_for(nsets, 64), 64, 0, s>>>(T, vx.p, skips.p, nsets, status.p);
    // ---- levels ----
    // A level of s points goes into a triangulation of p earlier points.  Two
    // insertions collide when their regions (about 20 tets and their ring)
    // meet, so the useful number of simultaneous insertions grows with p, not
    // with s: each level gets about p / alpha of them.  Several sets: their
    // levels are aligned from the coarsest and served together.
    const bool grow = opt.chunk <= 0 && opt.split != 0;   // the lockstep pool grows within levels
    const int alpha = opt.chunk < 0 ? -opt.chunk : 48;
    constexpr int kMinChunk = 16;
    // Below one latency wave of the GPU (about 4K resident warps), a level's time is
    // its depth: then a denser pool (down to one worker per kAlphaSmall earlier
    // points) trades more collisions for fewer insertions in a row.
    constexpr double kWaveWorkers = 4096.0;
    const double kAlphaSmall = opt.alpha_small > 0 ? double(opt.alpha_small) : double(alpha);
    auto level_chunk = [&](int64_t lb, int64_t le, double alpha_eff) -> int {
        if (opt.chunk > 0) return opt.chunk;
        const int64_t s_ = le - lb;
        int64_t w_ = std::max<int64_t>(1, int64_t(double(lb) / alpha_eff));
        w_ = std::min<int64_t>(w_, (s_ + kMinChunk - 1) / kMinChunk);
        return int((s_ + w_ - 1) / w_);
    };
    // levels[set] = bounds from the coarsest: [lev[k], lev[k+1]) local vertex ids.
    std::vector<std::vector<int>> levels(static_cast<size_t>(nsets));
    int nlev = 0;
    for (int st = 0; st < nsets; ++st) {
        if (hskips[size_t(st)].x < 0) continue;
        std::vector<int>& L = levels[size_t(st)];
        L.push_back(0);
        if (own.ok) {
            const int32_t* b = hlevel.data() + size_t(st) * size_t(own.levels);
            const int n_st = int(R.set_nv[size_t(st)]);
            for (int k = 1; k <= own.levels && L.back() < n_st; ++k) L.push_back(b[k] - b[0]);
        } else {
            int64_t hb[64];
            const int nb = multiscale_bounds(R.set_nv[size_t(st)], hb, 63, level_ratio);
            for (int k = nb - 1; k >= 0; --k) L.push_back(int(hb[k]));
        }
        nlev = std::max(nlev, int(L.size()) - 1);
    }
    // The effective alpha of a level: alpha, lowered (to kAlphaSmall at most)
    // while the whole pool would stay below one latency wave.
    auto level_alpha = [&](int lev) -> double {
        double w0 = 0;
        for (int st = 0; st < nsets; ++st) {
            const std::vector<int>& L = levels[size_t(st)];
            if (int(L.size()) - 1 <= lev) continue;
            w0 += std::max(1.0, double(L[size_t(lev)]) / alpha);
        }
        const double m = std::min(std::max(kWaveWorkers / std::max(w0, 1.0), 1.0), alpha / kAlphaSmall);
        return alpha / m;
    };
    auto level_descs = [&](int lev, double alpha_eff, std::vector<LevelDesc>& out) -> int {
        out.clear();
        int w = 0;
        for (int st = 0; st < nsets; ++st) {
            const std::vector<int>& L = levels[size_t(st)];
            if (int(L.size()) - 1 <= lev) continue;
            const int lb = L[size_t(lev)], le = L[size_t(lev) + 1];
            if (le <= lb) continue;
            const int plb = lev > 0 ? L[size_t(lev) - 1] : 0, ple = lb;
            const int ch = level_chunk(lb, le, alpha_eff);
            const int base = hvoff[size_t(st)];
            out.push_back(LevelDesc{st, base + lb, base + le, ch, base + plb, base + ple, w});
            w += (le - lb + ch - 1) / ch;
        }
        return w;
    };
    // ---- counters and status ----
    Round Rd;
    DevBuf<int> counters;
    DevBuf<unsigned long long> sums, totals, steps, pstats, astats;
    DevBuf<unsigned> dround;
    D3G_TRY(counters.alloc(4, s));
    D3G_TRY(sums.alloc(2, s));
    D3G_TRY(steps.alloc(2, s));
    D3G_TRY(totals.alloc(6, s));
    D3G_TRY(pstats.alloc(4, s));
    D3G_TRY(astats.alloc(6, s));
    D3G_TRY(dround.alloc(1, s));
    D3G_CUDA(cudaMemsetAsync(steps.p, 0, 2 * sizeof(unsigned long long), s));
    D3G_CUDA(cudaMemsetAsync(sums.p, 0, 2 * sizeof(unsigned long long), s));
    D3G_CUDA(cudaMemsetAsync(totals.p, 0, 6 * sizeof(unsigned long long), s));
    D3G_CUDA(cudaMemsetAsync(pstats.p, 0, 4 * sizeof(unsigned long long), s));
    D3G_CUDA(cudaMemsetAsync(astats.p, 0, 6 * sizeof(unsigned long long), s));
    D3G_CUDA(cudaMemsetAsync(dround.p, 0, sizeof(unsigned), s));
    Rd.counters = counters.p;
    Rd.sums = sums.p;
    Rd.totals = totals.p;
    Rd.steps = opt.timing ? steps.p : nullptr;
    Rd.round = dround.p;
    Rd.status = status.p;
    Rd.pstats = pstats.p;
    const int max_rounds = opt.max_rounds > 0 ? opt.max_rounds : (1 << 20);
    int round = 0;
    long long to_rounds = 0;   // points the asynchronous passes left to the rounds
    // Structural self-check after each level (opt.validate): k_validate over
    // every tet slot and vertex; the first broken invariant ends the build.
    DevBuf<unsigned long long> vfail;
    auto validate_tables = [&](const char* when, int lev) -> int {
        if (!vfail.p) D3G_TRY(vfail.alloc(1, s));
        D3G_CUDA(cudaMemsetAsync(vfail.p, 0xFF, sizeof(unsigned long long), s));
        int ntet_now = 0;
        D3G_CUDA(cudaMemcpyAsync(&ntet_now, tet_count.p, sizeof ntet_now, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaStreamSynchronize(s));
        const int64_t threads = int64_t(ntet_now) + nv;
        k_validate<<<grid_for(threads, 256, 1 << 30), 256, 0, s>>>(T, alock.p, ntet_now, nv,
                                                                   status.p, vfail.p);
        D3G_CUDA(cudaGetLastError());
        unsigned long long rec = ~0ull;
        D3G_CUDA(cudaMemcpyAsync(&rec, vfail.p, sizeof rec, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaStreamSynchronize(s));
        if (rec == ~0ull) return D3G_OK;
        static const char* what[] = {"", "bad vertex", "bad neighbour", "neighbour does not point back",
                                     "neighbours' shared facets differ", "lock held", "vertex's tet",
                                     "vertices of different sets"};
        const int code = int(rec >> 60);
        char msg[200];
        std::snprintf(msg, sizeof msg, "d3g_build: validate %s level %d: %s (%s %lld, %lld)", when, lev,
                      what[code > 0 && code < 8 ? code : 0], code == VF_VERT_TET ? "vertex" : "tet",
                      (long long)((rec >> 30) & 0x3FFFFFFFull), (long long)(rec & 0x3FFFFFFFull));
        set_error(msg);
        return D3G_ERR_INTERNAL;
    };
    const bool trace = getenv("D3G_TRACE") != nullptr;
    cudaEvent_t kev[4] = {nullptr, nullptr, nullptr, nullptr};
    if (opt.timing)
        for (auto& e : kev) cudaEventCreate(&e);
    struct EvGuard {
        cudaEvent_t* e;
        ~EvGuard() {
            for (int i = 0; i < 4; ++i)
                if (e[i]) cudaEventDestroy(e[i]);
        }
    } ev_guard{kev};
    // ---- workers of the lockstep rounds and of the full variant ----
    // Allocated when first needed: a build whose points all go in through
    // k_insert_groups has none.
    constexpr int kAsyncWarps = kNumSMs * 32;   // resident at 64 registers a thread
    Workers W{};
    Workers WB{};
    // Conflict-region scratch per worker (normal rounds and the full variant) and
    // per big-round slot; a caller's cavity_capacity lowers both.
    const int cav_normal = opt.cavity_capacity > 0 ? std::min(kCavCap, int(opt.cavity_capacity)) : kCavCap;
    const int cav_big = opt.cavity_capacity > 0 ? std::min(kBigCav, int(opt.cavity_capacity)) : kBigCav;
    int maxw = 0, wcap = 0, wslots = 0;
    DevBuf<int> wcur, wbeg, wend, wpos, wleft, wnwon, wlast, wguide, wstate, wncav, wnfac, wcav, wfac, wparked, wset;
    DevBuf<int4> wsv, wsn;
    DevBuf<unsigned long long> aekey;
    // Records for `cap` workers; per-slot scratch for `slots` of them at a time.
    auto alloc_workers = [&](int cap, int slots) -> int {
        if (cap <= wcap && slots <= wslots) return D3G_OK;
        wcap = std::max(wcap, cap);
        wslots = std::max(wslots, slots);
        W.cav_cap = cav_normal;
        W.fac_cap = 2 * cav_normal;
        DevBuf<int>* per_worker[] = {&wcur, &wbeg, &wend, &wpos, &wleft, &wnwon, &wlast, &wguide,
                                     &wstate, &wncav, &wnfac, &wparked, &wset};
        for (DevBuf<int>* d : per_worker) D3G_TRY(d->alloc(size_t(wcap), s));
        D3G_TRY(wcav.alloc(size_t(wslots) * W.cav_cap, s));
        D3G_TRY(wfac.alloc(size_t(wslots) * W.fac_cap, s));
        D3G_TRY(wsv.alloc(size_t(wslots) * W.fac_cap, s));
        D3G_TRY(wsn.alloc(size_t(wslots) * W.fac_cap, s));
        if (use_async) D3G_TRY(aekey.alloc(size_t(std::min(wslots, kAsyncWarps)) * 3 * size_t(W.fac_cap), s));
        W.cur = wcur.p;
        W.end = wend.p;
        W.beg = wbeg.p;
        W.list = nullptr;
        W.parked = wparked.p;
        W.wset = wset.p;
        W.skips = skips.p;
        W.set_exact = set_exact.p;
        W.pos = wpos.p;
        W.left = wleft.p;
        W.nwon = wnwon.p;
        W.last = wlast.p;
        W.guide = wguide.p;
        W.state = wstate.p;
        W.ncav = wncav.p;
        W.nfac = wnfac.p;
        W.cav = wcav.p;
        W.fac = wfac.p;
        W.st_v = wsv.p;
        W.st_n = wsn.p;
        return D3G_OK;
    };
    // The rounds' claims and restar scratch, likewise.
    auto alloc_rounds = [&]() -> int {
        if (claim.p) return D3G_OK;
        D3G_TRY(claim.alloc(size_t(T.cap), s));
        D3G_TRY(fnew.alloc(size_t(T.cap) * 4, s));
        D3G_CUDA(cudaMemsetAsync(claim.p, 0xFF, sizeof(unsigned long long) * size_t(T.cap), s));
        T.claim = claim.p;
        T.fnew = fnew.p;
        return D3G_OK;
    };
    DevBuf<int> set_p0, set_ins, set_w, set_split, nworkers;
    SplitState SS{};
    DevBuf<int> blist, bcount, bcav, bfac;
    DevBuf<int4> bsv, bsn;
    // Big rounds: workers whose conflict region outgrew the normal scratch.
    auto big_rounds = [&]() -> int {
        if (blist.n < size_t(wcap)) D3G_TRY(blist.alloc(size_t(wcap), s));
        if (!bcount.p) {
            D3G_TRY(bcount.alloc(1, s));
            D3G_TRY(bcav.alloc(size_t(kBigSlots) * cav_big, s));
            D3G_TRY(bfac.alloc(size_t(kBigSlots) * 2 * cav_big, s));
            D3G_TRY(bsv.alloc(size_t(kBigSlots) * 2 * cav_big, s));
            D3G_TRY(bsn.alloc(size_t(kBigSlots) * 2 * cav_big, s));
        }
        for (;;) {
            D3G_CUDA(cudaMemsetAsync(bcount.p, 0, sizeof(int), s));
            k_collect_parked<<<grid_for(W.n, 128, 1 << 30), 128, 0, s>>>(W, blist.p, bcount.p);
            int nparked = 0;
            D3G_CUDA(cudaMemcpyAsync(&nparked, bcount.p, sizeof nparked, cudaMemcpyDeviceToHost, s));
            D3G_CUDA(cudaStreamSynchronize(s));
            if (nparked == 0) return D3G_OK;
            WB = W;
            WB.list = blist.p;
            WB.n = std::min(nparked, kBigSlots);
            WB.cav = bcav.p;
            WB.fac = bfac.p;
            WB.st_v = bsv.p;
            WB.st_n = bsn.p;
            WB.cav_cap = cav_big;
            WB.fac_cap = 2 * cav_big;
            for (;;) {
                if (++round > max_rounds) {
                    set_error("d3g_build: insertion round limit reached");
                    return D3G_ERR_ROUND_LIMIT;
                }
                unsigned long long before = 0;
                D3G_CUDA(cudaMemcpyAsync(&before, totals.p, sizeof before, cudaMemcpyDeviceToHost, s));
                k_round_begin<<<1, 1, 0, s>>>(Rd);
                launch_insertion(32, 0, T, WB, Rd, vx.p, s);
                launch_insertion(32, 1, T, WB, Rd, vx.p, s);
                launch_insertion(32, 2, T, WB, Rd, vx.p, s);
                k_round_end<<<1, 1, 0, s>>>(Rd);
                unsigned long long ht[6];
                uint32_t hs = 0;
                D3G_CUDA(cudaMemcpyAsync(ht, totals.p, sizeof ht, cudaMemcpyDeviceToHost, s));
                D3G_CUDA(cudaMemcpyAsync(&hs, status.p, sizeof hs, cudaMemcpyDeviceToHost, s));
                D3G_CUDA(cudaStreamSynchronize(s));
                if (hs != 0) {
                    const int st = status_from_bits(hs);
                    if (st == D3G_ERR_CAVITY_CAPACITY)
                        set_error("d3g_build: a conflict region exceeded the big-round scratch");
                    return st;
                }
                if (ht[3] == 0) break;           // every listed worker got its point in
                if (ht[0] == before) {           // the earliest parked point must win
                    set_error("d3g_build: a big round made no progress");
                    return D3G_ERR_INTERNAL;
                }
            }
        }
    };
    double split_alpha = alpha;
    int lanes = opt.lanes > 0 ? opt.lanes : 32;
    auto one_round = [&](bool timed) {
        k_round_begin<<<1, 1, 0, s>>>(Rd);
        if (timed) cudaEventRecord(kev[0], s);
        launch_insertion(lanes, 0, T, W, Rd, vx.p, s);
        if (timed) cudaEventRecord(kev[1], s);
        launch_insertion(lanes, 1, T, W, Rd, vx.p, s);
        if (timed) cudaEventRecord(kev[2], s);
        launch_insertion(lanes, 2, T, W, Rd, vx.p, s);
        if (timed) cudaEventRecord(kev[3], s);
        k_round_end<<<1, 1, 0, s>>>(Rd);
    };
    // Rounds go out in batches captured as one CUDA graph; the host looks at
    // the counters once per batch.  Rounds after the level is done find no
    // active worker and return at once.
    cudaGraphExec_t gexec = nullptr;
    struct GraphGuard {
        cudaGraphExec_t* g;
        ~GraphGuard() {
            if (*g) cudaGraphExecDestroy(*g);
        }
    } graph_guard{&gexec};
    auto capture = [&]() -> int {
        if (gexec) cudaGraphExecDestroy(gexec);
        gexec = nullptr;
        if (opt.timing) return D3G_OK;
        cudaGraph_t graph = nullptr;
        D3G_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        for (int r = 0; r < kRoundsPerBatch; ++r) one_round(false);
        D3G_CUDA(cudaStreamEndCapture(s, &graph));
        const cudaError_t ge = cudaGraphInstantiate(&gexec, graph, 0);
        cudaGraphDestroy(graph);
        if (ge != cudaSuccess) {
            set_error(std::string("cudaGraphInstantiate: ") + cudaGetErrorString(ge));
            return D3G_ERR_CUDA;
        }
        return D3G_OK;
    };
    auto run_rounds = [&]() -> int {
    D3G_TRY(capture());
    for (;;) {
        const int batch = opt.timing ? 1 : kRoundsPerBatch;
        round += batch;
        if (round > max_rounds) {
            set_error("d3g_build: insertion round limit reached");
            return D3G_ERR_ROUND_LIMIT;
        }
        if (opt.timing) one_round(true);
        else D3G_CUDA(cudaGraphLaunch(gexec, s));
        if (grow) {
            D3G_CUDA(cudaMemsetAsync(set_ins.p, 0, sizeof(int) * size_t(nsets), s));
            k_count_wins<<<grid_for(W.n, 128, 1 << 30), 128, 0, s>>>(W, SS);
            k_plan_split<<<grid_for(nsets, 128), 128, 0, s>>>(SS, nsets, split_alpha);
            k_split<<<grid_for(W.n, 128, 1 << 30), 128, 0, s>>>(W, SS, W.n);
        }
        unsigned long long ht[6];
        uint32_t hs = 0;
        int hn = W.n;
        D3G_CUDA(cudaMemcpyAsync(ht, totals.p, sizeof ht, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaMemcpyAsync(&hs, status.p, sizeof hs, cudaMemcpyDeviceToHost, s));
        if (grow) D3G_CUDA(cudaMemcpyAsync(&hn, nworkers.p, sizeof hn, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaStreamSynchronize(s));
        hn = std::min(hn, maxw);
        if (hn != W.n) {
            // The pool grew: the next batches serve the new workers too.
            W.n = hn;
            k_set_int<<<1, 1, 0, s>>>(nworkers.p, W.n);
            D3G_TRY(capture());
        }
        if (hs != 0) {
            const int st = status_from_bits(hs);
            if (st == D3G_ERR_OOM) set_error("d3g_build: tet table full");
            return st;
        }
        if (ht[4]) {
            set_error("d3g_build: an insertion round made no progress");
            return D3G_ERR_INTERNAL;
        }
        if (opt.timing) {
            float a = 0.f, b2 = 0.f, c = 0.f;
            cudaEventElapsedTime(&a, kev[0], kev[1]);
            cudaEventElapsedTime(&b2, kev[1], kev[2]);
            cudaEventElapsedTime(&c, kev[2], kev[3]);
            R.stats.ms_cavity += a;
            R.stats.ms_check += b2;
            R.stats.ms_restar += c;
            R.stats.launches_cavity += 1;
        }
        if (ht[5] != 0) continue;
        if (ht[3] == 0) break;
        // Only parked workers are left: serve them in big rounds, up to
        // kBigSlots at a time, each until its point is in.
        D3G_TRY(big_rounds());
    }
    return D3G_OK;
    };
    // Lockstep rounds over every level (schedule = 1, or a pool that grows within
    // levels).
    auto run_lockstep = [&]() -> int {
        std::vector<LevelDesc> descs;
        maxw = 1;
        for (int lev = 0; lev < nlev; ++lev) maxw = std::max(maxw, level_descs(lev, level_alpha(lev), descs));
        // Room for the pool to grow within levels (at most one worker per 16 points).
        if (grow) maxw = std::max<int>(maxw, int(std::min<int64_t>(int64_t(nv) / 16, int64_t(1) << 18)));
        D3G_TRY(alloc_workers(maxw, maxw));
        D3G_TRY(alloc_rounds());
        D3G_TRY(set_p0.alloc(size_t(nsets), s));
        D3G_TRY(set_ins.alloc(size_t(nsets), s));
        D3G_TRY(set_w.alloc(size_t(nsets), s));
        D3G_TRY(set_split.alloc(size_t(nsets), s));
        D3G_TRY(nworkers.alloc(1, s));
        D3G_CUDA(cudaMemsetAsync(set_ins.p, 0, sizeof(int) * size_t(nsets), s));
        SS = SplitState{set_p0.p, set_ins.p, set_w.p, set_split.p, nworkers.p, maxw};
        std::vector<int> hp0(static_cast<size_t>(nsets)), hw(static_cast<size_t>(nsets));
        for (int lev = 0; lev < nlev; ++lev) {
            split_alpha = level_alpha(lev);
            W.n = level_descs(lev, split_alpha, descs);
            if (W.n == 0) continue;
            char level_name[32];
            std::snprintf(level_name, sizeof level_name, "d3g.level %d", lev);
            NvtxRange nvtx_level(level_name);
            std::fill(hp0.begin(), hp0.end(), 0);
            std::fill(hw.begin(), hw.end(), 0);
            for (size_t i = 0; i < descs.size(); ++i) {
                const LevelDesc& d = descs[i];
                hp0[size_t(d.set)] = d.lb - hvoff[size_t(d.set)];
                hw[size_t(d.set)] = (i + 1 < descs.size() ? descs[i + 1].w0 : W.n) - d.w0;
            }
            D3G_CUDA(cudaMemcpyAsync(set_p0.p, hp0.data(), sizeof(int) * size_t(nsets), cudaMemcpyHostToDevice, s));
            D3G_CUDA(cudaMemcpyAsync(set_w.p, hw.data(), sizeof(int) * size_t(nsets), cudaMemcpyHostToDevice, s));
            k_set_int<<<1, 1, 0, s>>>(nworkers.p, W.n);
            DevBuf<LevelDesc> ddesc;
            D3G_TRY(ddesc.alloc(descs.size(), s));
            D3G_CUDA(cudaMemcpyAsync(ddesc.p, descs.data(), sizeof(LevelDesc) * descs.size(),
                                     cudaMemcpyHostToDevice, s));
            k_setup_level<<<grid_for(W.n, 128, 1 << 30), 128, 0, s>>>(W, ddesc.p, int(descs.size()));
            D3G_TRY(run_rounds());
            if (opt.validate) D3G_TRY(validate_tables("after", lev));
            if (trace) fprintf(stderr, "d3g level %d sets %zu workers %d rounds so far %d\n", lev, descs.size(), W.n, round);
        }
        return D3G_OK;
    };
    // The points k_insert_groups left (regions beyond its scratch, persistent
    // conflicts) through the full variant, one worker per point, all of them at once,
    // again while a pass inserts at least a quarter of its points; what that leaves
    // through the rounds.
    DevBuf<int> aleft, aleft2, actl;
    auto finish_points = [&](int* list, int count) -> int {
        if (count <= 0) return D3G_OK;
        D3G_TRY(alloc_workers(std::min(count, 1 << 20), std::min(count, kAsyncWarps)));
        if (!aleft.p) {
            D3G_TRY(aleft.alloc(size_t(nv), s));
            D3G_TRY(aleft2.alloc(size_t(nv), s));
            D3G_TRY(actl.alloc(2, s));
        }
        int* cur = list;
        int* nxt = aleft.p;
        int ncur = count;
        for (int pass = 0; ncur > 0 && pass < kLeftPasses; ++pass) {
            int nnext = 0;
            D3G_CUDA(cudaMemsetAsync(actl.p + 1, 0, sizeof(int), s));
            for (int off = 0; off < ncur; off += wcap) {
                W.n = std::min(wcap, ncur - off);
                k_setup_list<<<grid_for(W.n, 128, 1 << 30), 128, 0, s>>>(W, cur + off, W.n, vset.p, voff.p, T.vert_tet);
                // Workers go out in a scattered order (stride coprime with their count,
                // near its golden ratio), so that those taken at the same time lie far
                // apart along the curve.
                int64_t stride = std::max<int64_t>(1, int64_t(double(W.n) * 0.6180339887));
                while (std::gcd(stride, int64_t(W.n)) != 1) ++stride;
                D3G_CUDA(cudaMemsetAsync(actl.p, 0, sizeof(int), s));
                const int warps = std::min(W.n, kAsyncWarps);
                if (warps > wslots) {
                    set_error("d3g_build: asynchronous pass wider than its scratch");
                    return D3G_ERR_INTERNAL;
                }
                AsyncCtx A{alock.p, actl.p, nxt, actl.p + 1, stride, W.n, aekey.p, astats.p};
                k_insert_full<<<unsigned((int64_t(warps) * 32 + 127) / 128), 128, 0, s>>>(T, W, A, Rd, vx.p, warps);
                D3G_CUDA(cudaGetLastError());
                R.stats.launches_async += 1;
            }
            uint32_t hs = 0;
            D3G_CUDA(cudaMemcpyAsync(&nnext, actl.p + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
            D3G_CUDA(cudaMemcpyAsync(&hs, status.p, sizeof hs, cudaMemcpyDeviceToHost, s));
            D3G_CUDA(cudaStreamSynchronize(s));
            if (trace) fprintf(stderr, "d3g full pass over %d points left %d\n", ncur, nnext);
            if (hs != 0) {
                const int st = status_from_bits(hs);
                if (st == D3G_ERR_OOM) set_error("d3g_build: tet table full");
                return st;
            }
            const bool slow = int64_t(ncur - nnext) * 4 < int64_t(ncur);
            cur = nxt;
            nxt = cur == aleft.p ? aleft2.p : aleft.p;
            ncur = nnext;
            if (slow) break;
        }
        if (ncur > 0) D3G_TRY(alloc_rounds());
        to_rounds += ncur;
        for (int off = 0; off < ncur; off += wslots) {
            maxw = W.n = std::min(wslots, ncur - off);
            k_setup_list<<<grid_for(W.n, 128, 1 << 30), 128, 0, s>>>(W, cur + off, W.n, vset.p, voff.p, T.vert_tet);
            D3G_TRY(run_rounds());
        }
        return D3G_OK;
    };
    // Every level through k_insert_groups, launched one after another with no
    // look at the results in between: what a level leaves goes in at the end (the
    // order of insertions does not matter).
    auto run_async = [&]() -> int {
        // Items: level by level, each set's vertices of the level together.
        std::vector<int> ctl(size_t(2) * size_t(nlev) + size_t(nlev) * size_t(nsets) + size_t(nsets), 0);
        int* m_of = ctl.data();
        int* first_of = ctl.data() + nlev;
        int* base = ctl.data() + 2 * nlev;
        int* coarse = base + size_t(nlev) * size_t(nsets);   // levels of each set that k_coarse inserts
        // (Not under a caller's limits, which are on the tables and on a group's scratch.)
        // Nor for more sets than the GPU has SMs: a block inserts slower than the GPU does
        // when other sets keep it busy (without it and with it, ms: 256 mixed sets 39.2 and
        // 41.8, 600 / 1000 / 2000 sets of 700 points 8.2 / 9.8 / 15.7 and 9.2 / 13.0 / 25.1,
        // 300 of them 6.2 and 5.7).
        const bool use_coarse = own.ok && nsets <= kNumSMs && opt.walk_limit <= 0 && opt.cavity_capacity <= 0 && opt.tet_capacity <= 0;
        for (int st = 0; use_coarse && st < nsets; ++st) {
            const std::vector<int>& L = levels[size_t(st)];
            int k = std::min(int(L.size()) - 1, coarse_levels(h_off[st + 1] - h_off[st], growth));
            while (k > 0 && L[size_t(k)] > kCoarseCap) --k;
            coarse[st] = k > 0 && L[size_t(k)] >= 8 ? k : 0;
        }
        int total = 0;
        std::vector<int64_t> groups_of(static_cast<size_t>(nlev), 0);
        std::vector<int> sets_of(static_cast<size_t>(nlev), 0);
        for (int lev = 0; lev < nlev; ++lev) {
            const double alpha_eff = level_alpha(lev);
            first_of[lev] = total;
            for (int st = 0; st < nsets; ++st) {
                const std::vector<int>& L = levels[size_t(st)];
                if (int(L.size()) - 1 <= lev) continue;
                if (lev < coarse[st]) {
                    base[size_t(lev) * size_t(nsets) + size_t(st)] = -1;
                    continue;
                }
                const int cnt = L[size_t(lev) + 1] - L[size_t(lev)];
                base[size_t(lev) * size_t(nsets) + size_t(st)] = total;
                total += cnt;
                if (cnt <= 0) continue;
                sets_of[size_t(lev)] += 1;
                const int64_t w = opt.chunk > 0 ? (cnt + opt.chunk - 1) / opt.chunk
                                                : std::max<int64_t>(1, int64_t(double(L[size_t(lev)]) / alpha_eff));
                groups_of[size_t(lev)] += std::min<int64_t>(w, cnt);
            }
            m_of[lev] = total - first_of[lev];
        }
        constexpr int kPassHeads = 256;    // queue heads of passes with the exact stage
        DevBuf<int> heads;
        int head = 0;
        DevBuf<int> dctl, items, guide, hint, lstart, defer[2], big, left[2], cnt;
        DevBuf<int4> pool;
        D3G_TRY(dctl.alloc(ctl.size(), s));
        D3G_TRY(items.alloc(size_t(std::max(total, 1)), s));
        D3G_TRY(guide.alloc(size_t(nv), s));
        D3G_TRY(hint.alloc(size_t(nv), s));
        D3G_CUDA(cudaMemsetAsync(hint.p, 0xFF, sizeof(int) * size_t(nv), s));
        for (auto& l : defer) D3G_TRY(l.alloc(size_t(nv), s));
        D3G_TRY(big.alloc(size_t(nv), s));
        for (auto& l : left) D3G_TRY(l.alloc(size_t(nv), s));
        D3G_TRY(pool.alloc(size_t(kMaxGroups), s));
        // Counters: four per list of points left, one per list of deferred ones (at most
        // one after each level and kExactPasses each time they are drained), seven more.
        const size_t nleft_lists = size_t(nlev) + kLastPasses + 1, ndefer_lists = size_t(nlev) * (kExactPasses + 1) + 2;
        D3G_TRY(cnt.alloc(4 * nleft_lists + ndefer_lists + 7, s));
        D3G_CUDA(cudaMemcpyAsync(dctl.p, ctl.data(), sizeof(int) * ctl.size(), cudaMemcpyHostToDevice, s));
        D3G_CUDA(cudaMemsetAsync(pool.p, 0, sizeof(int4) * size_t(kMaxGroups), s));
        D3G_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(int) * cnt.n, s));
        const int* starts = own.level_start.p;
        int start_stride = own.levels;
        std::vector<int> hstart;
        if (!own.ok) {
            start_stride = nlev;
            hstart.resize(size_t(nsets) * size_t(nlev) + 1);
            for (int st = 0; st < nsets; ++st)
                for (int lev = 0; lev < nlev; ++lev) {
                    const std::vector<int>& L = levels[size_t(st)];
                    const int k = std::min(lev, std::max(int(L.size()) - 1, 0));
                    hstart[size_t(st) * size_t(nlev) + size_t(lev)] = hvoff[size_t(st)] + (L.empty() ? 0 : L[size_t(k)]);
                }
            hstart.back() = nv;
            D3G_TRY(lstart.alloc(hstart.size(), s));
            D3G_CUDA(cudaMemcpyAsync(lstart.p, hstart.data(), sizeof(int) * hstart.size(), cudaMemcpyHostToDevice, s));
            starts = lstart.p;
        }
        k_level_items<<<grid_for(nv, 256), 256, 0, s>>>(vset.p, skips.p, starts, start_stride, dctl.p + 2 * nlev, nsets,
                                                        own.ok ? own.keys.p : nullptr, own.curve_bits, vx.p, nv,
                                                        items.p, guide.p);
        own.keys.release();
        // Lists of points left, and per list the head of the queue whose points it gets, how
        // many it has and the head of the pass over them.
        auto head_of = [&](int k) { return cnt.p + 4 * k; };
        auto n_left_of = [&](int k) { return cnt.p + 4 * k + 1; };
        auto left_of = [&](int k) { return left[k & 1].p; };
        // Likewise the lists of points with undecided tests.
        auto defer_of = [&](int k) { return defer[k & 1].p; };
        auto n_defer_of = [&](int k) { return cnt.p + 4 * nleft_lists + k; };
        int* const coarse_queue = cnt.p + (cnt.n - 7);
        int* const big_ctl = coarse_queue + 1;   // [0] points too big, [1], [3] and [5] queue heads, [2] and [4] left
        int list = 0, deferred = 0;
        GroupArgs A{};
        A.lock = alock.p;
        A.guide = guide.p;
        A.hint = hint.p;
        A.defer = defer_of(0);
        A.n_defer = n_defer_of(0);
        A.big = big.p;
        A.n_big = big_ctl;
        A.pool = pool.p;
        A.skips = skips.p;
        A.set_exact = set_exact.p;
        A.inv_grid = inv_grid.p;
        A.voff = voff.p;
        A.stats = astats.p;
        A.cavity = cav_normal;
        A.first = 0;
        A.most = INT_MAX;
        auto launch = [&](int G, int ngroups, int mode) {
            // At most one group per kPoolSlots vertices, so that the slots groups hold
            // without using them stay within the table's room for them.
            const int blocks = mode == kExact ? kExactBlocks : kGroupBlocks;
            A.ngroups = std::max(1, std::min({ngroups, kNumSMs * blocks * (kGroupThreads / G), nv / kPoolSlots}));
            const unsigned grid = unsigned((A.ngroups + kGroupThreads / G - 1) / (kGroupThreads / G));
            auto* kernel = mode == kExact ? k_insert_groups<32, kExact, 256, kGroupThreads>
                         : G == 8  ? (mode == kNear ? k_insert_groups<8, kNear, 64, kGroupThreads> : k_insert_groups<8, kFilter, 64, kGroupThreads>)
                         : G == 16 ? (mode == kNear ? k_insert_groups<16, kNear, 128, kGroupThreads> : k_insert_groups<16, kFilter, 128, kGroupThreads>)
                                   : (mode == kNear ? k_insert_groups<32, kNear, 256, kGroupThreads> : k_insert_groups<32, kFilter, 256, kGroupThreads>);
            const size_t scratch = G == 8 ? sizeof(GroupScratch<8, 64>) * 16
                                          : (G == 16 ? sizeof(GroupScratch<16, 128>) * 8 : sizeof(GroupScratch<32, 256>) * 4);
            kernel<<<grid, kGroupThreads, scratch, s>>>(T, A, Rd, vx.p);
            R.stats.launches_async += 1;
        };
        // The variant that settles undecided tests of near points in 64 bits needs more
        // registers (52 bytes of spills stored and 60 loaded at 96): 10^7 uniform points 107 -> 114 ms, 4096
        // mixed sets 410 -> 437, but the 10^6 sphere on a 2^-10 grid 79 -> 27.  So it takes
        // the levels of a build most of whose points lie on such grids, and elsewhere
        // only what the plain one leaves.
        int64_t on_grid = 0;
        for (int st = 0; st < nsets; ++st)
            if (hexact[size_t(st)] & EX_GRID) on_grid += R.set_nv[size_t(st)];
        const int main_mode = 2 * on_grid > nv ? kNear : kFilter;
        // A pass of the widest groups over the current list; what it leaves is the next.
        auto left_pass = [&](int ngroups, bool last = false) {
            A.items = left_of(list);
            A.n_items = n_left_of(list);
            A.next = head_of(list) + 2;
            ++list;
            A.left = last ? A.big : left_of(list);
            A.n_left = last ? A.n_big : n_left_of(list);
            launch(32, ngroups, kNear);
        };
        // The same with the exact stage, over the points with undecided tests: about `n` of
        // them, where `in` points are in.  Where that is more than are in, a part after
        // the other, each about as many points as are in, as levels do.
        auto exact_pass = [&](int64_t n, int64_t in, int ngroups) -> int {
            if (!heads.p) D3G_TRY(heads.alloc(kPassHeads, s));
            A.items = defer_of(deferred);
            A.n_items = n_defer_of(deferred);
            ++deferred;
            A.left = A.defer = defer_of(deferred);
            A.n_left = A.n_defer = n_defer_of(deferred);
            in = std::max<int64_t>(in, 16);
            for (int64_t k = 0; k >= 0;) {
                if (head == 0) D3G_CUDA(cudaMemsetAsync(heads.p, 0, sizeof(int) * kPassHeads, s));
                A.next = heads.p + head;
                head = (head + 1) % kPassHeads;
                const int64_t part = std::max<int64_t>(in, 64);
                A.first = int(k);
                A.most = k + part < n ? int(part) : INT_MAX;
                launch(32, int(std::min<int64_t>(std::max<int64_t>(in / alpha, 1), ngroups)), kExact);
                k = k + part < n ? k + part : -1;
                in += part;
            }
            A.first = 0;
            A.most = INT_MAX;
            return D3G_OK;
        };
        // What the levels' passes could not do, while the host looks on: points with
        // undecided tests, with fewer and fewer groups in the way of one another while at
        // least half of them go in; then these, regions beyond the widest groups' scratch and
        // points worn out by conflicts with room for kBigCapacity, by 16 groups, and - such
        // regions of one set overlap, and take longer than a group waits for another - by one
        // alone; the rest by k_insert_full.
        auto drain = [&]() -> int {
            int nd = 0, nb[6] = {0, 0, 0, 0, 0, 0};
            std::vector<int> seen(ndefer_lists + 7);
            auto look = [&]() -> int {
                uint32_t hs = 0;
                D3G_CUDA(cudaGetLastError());
                if (opt.timing) cudaEventRecord(kev[1], s);
                D3G_CUDA(cudaMemcpyAsync(seen.data(), n_defer_of(0), sizeof(int) * seen.size(), cudaMemcpyDeviceToHost, s));
                D3G_CUDA(cudaMemcpyAsync(&hs, status.p, sizeof hs, cudaMemcpyDeviceToHost, s));
                D3G_CUDA(cudaStreamSynchronize(s));
                nd = seen[size_t(deferred)];
                std::copy(seen.end() - 6, seen.end(), nb);
                if (opt.timing) {
                    float am = 0.f;
                    cudaEventElapsedTime(&am, kev[0], kev[1]);
                    R.stats.ms_async += am;
                    cudaEventRecord(kev[0], s);
                }
                if (trace) fprintf(stderr, "d3g drain: %d undecided, too big %d %d %d\n", nd, nb[0], nb[2], nb[4]);
                const int st = status_from_bits(hs);
                if (st == D3G_ERR_OOM) set_error("d3g_build: tet table full");
                return st;
            };
            D3G_TRY(look());
            for (int k = 0; nd > 4 * nb[0] && k < kExactPasses; ++k) {   // (else most regions are large)
                const int before = nd;
                D3G_TRY(exact_pass(nd, int64_t(nv) - nd, std::max(kNumSMs * kExactBlocks * (kGroupThreads / 32) >> (3 * k), 16)));
                D3G_TRY(look());
                if (2 * nd > before) break;        // (in each other's way, or of large regions)
            }
            if (nb[0] + nd > 0) {
                // (the exact stage's stack only where some point has needed it)
                auto* kernel = deferred > 0 || nd > 0 ? k_insert_groups<32, kExact, kBigCapacity, 32>
                                                      : k_insert_groups<32, kNear, kBigCapacity, 32>;
                D3G_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              int(sizeof(GroupScratch<32, kBigCapacity>))));
                int* const rest = defer_of(deferred + 1);      // (free here)
                GroupArgs B = A;
                B.cavity = opt.cavity_capacity > 0 ? cav_normal : kBigCapacity;
                auto pass = [&](int* items, const int* n, int most, int* next, int* out, int* n_out, int ngroups) {
                    B.items = items;
                    B.n_items = n;
                    B.most = most;
                    B.next = next;
                    B.left = B.big = B.defer = out;
                    B.n_left = B.n_big = B.n_defer = n_out;
                    B.ngroups = std::min(ngroups, std::max(1, nv / kPoolSlots));
                    kernel<<<unsigned(B.ngroups), 32, sizeof(GroupScratch<32, kBigCapacity>), s>>>(T, B, Rd, vx.p);
                    R.stats.launches_async += 1;
                };
                if (nb[0] > 0) pass(big.p, big_ctl, INT_MAX, big_ctl + 1, rest, big_ctl + 2, kBigGroups);
                if (nd > 0) pass(defer_of(deferred), n_defer_of(deferred), INT_MAX, big_ctl + 5, rest, big_ctl + 2, kBigGroups);
                D3G_TRY(look());
                const int left_over = nb[2];
                if (left_over > 0) {
                    pass(rest, big_ctl + 2, kLonePoints, big_ctl + 3, big.p, big_ctl + 4, 1);
                    D3G_TRY(look());
                }
                D3G_TRY(finish_points(rest + kLonePoints, left_over - kLonePoints));
                D3G_TRY(finish_points(big.p, nb[4]));
            }
            D3G_CUDA(cudaMemsetAsync(big_ctl, 0, 6 * sizeof(int), s));
            D3G_CUDA(cudaMemsetAsync(n_defer_of(deferred), 0, sizeof(int), s));
            return D3G_OK;
        };
        // The look behind a level is at the counts of the level before, which the device
        // has passed by then, so that it never waits for the host.
        const bool may_defer = std::any_of(hexact.begin(), hexact.end(), [](uint8_t e) { return (e & EX_BOTH) != EX_BOTH; });
        struct Look {
            int* n = nullptr;            // pinned
            cudaEvent_t ev = nullptr;
            int64_t points = 0;          // inserted or waiting when it was taken
            ~Look() {
                if (ev) cudaEventSynchronize(ev), cudaEventDestroy(ev);
                host_result_free(n);
            }
        } look;
        bool exact_levels = false;
        int64_t waiting = 0;
        auto look_behind = [&](int lev) -> int {
            if (!exact_levels && look.points > 0) {
                D3G_CUDA(cudaEventSynchronize(look.ev));
                exact_levels = int64_t(*look.n) * kUndecidedShare > look.points;
                waiting = int64_t(*look.n) + m_of[lev];        // the level just launched may leave all of its points
            }
            if (exact_levels) {
                const int64_t points = first_of[lev] + m_of[lev];
                const int64_t n = std::exchange(waiting, 0);   // later levels' are decided as they come
                return exact_pass(n, points - n, 1 << 24);
            }
            if (!look.ev) {
                look.n = static_cast<int*>(host_result_alloc(sizeof(int)));
                D3G_CUDA(cudaEventCreateWithFlags(&look.ev, cudaEventDisableTiming));
            }
            look.points = first_of[lev] + m_of[lev];
            D3G_CUDA(cudaMemcpyAsync(look.n, n_defer_of(deferred), sizeof(int), cudaMemcpyDeviceToHost, s));
            D3G_CUDA(cudaEventRecord(look.ev, s));
            return D3G_OK;
        };
        if (opt.timing) cudaEventRecord(kev[0], s);
        if (use_coarse) {
            NvtxRange nvtx_level("d3g.coarse");
            A.left = left_of(list);
            A.n_left = n_left_of(list);
            const CoarseArgs K{starts, start_stride, dctl.p + (coarse - ctl.data()), nsets, coarse_queue};
            auto* kernel = main_mode == kNear ? k_coarse<kNear> : k_coarse<kFilter>;
            D3G_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(CoarseShared))));
            kernel<<<unsigned(std::min(nsets, kNumSMs)), kCoarseThreads, sizeof(CoarseShared), s>>>(T, A, K, Rd, vx.p);
            D3G_CUDA(cudaGetLastError());
            R.stats.launches_async += 1;
        }
        for (int lev = 0; lev < nlev; ++lev) {
            if (m_of[lev] == 0 && lev < nlev - 1 && !opt.validate) continue;
            char level_name[32];
            std::snprintf(level_name, sizeof level_name, "d3g.level %d", lev);
            NvtxRange nvtx_level(level_name);
            cudaEvent_t ev0 = nullptr, ev1 = nullptr;
            if (trace) {
                cudaEventCreate(&ev0);
                cudaEventCreate(&ev1);
                cudaEventRecord(ev0, s);
            }
            const int G = group_lanes(groups_of[size_t(lev)]);
            A.items = items.p + first_of[lev];
            A.n_items = dctl.p + lev;
            A.next = head_of(list);
            // What narrower groups leave goes to wider ones at once; what those leave
            // (points in each other's way) waits for the next level's pass.
            A.left = left_of(G < 32 ? list : list + 1);
            A.n_left = n_left_of(G < 32 ? list : list + 1);
            if (m_of[lev] > 0) {
                // (The first level grows from one tet: there the guides are nearer.  A
                // caller's walk limit holds for an insertion's whole walk.)
                if ((lev > 0 || use_coarse) && opt.walk_limit <= 0)
                    k_locate<<<grid_for(m_of[lev], 128), 128, 0, s>>>(T, A, vx.p);
                launch(G, int(std::min<int64_t>(groups_of[size_t(lev)], 1 << 24)), main_mode);
                left_pass(kNumSMs * (kGroupThreads / 32));
                if (may_defer && lev < nlev - 1) D3G_TRY(look_behind(lev));   // (the last level is drained)
            }
            D3G_CUDA(cudaGetLastError());
            if (trace) {
                cudaEventRecord(ev1, s);
                cudaEventSynchronize(ev1);
                float ms = 0.f;
                cudaEventElapsedTime(&ms, ev0, ev1);
                int c[4] = {0, 0, 0, 0}, nd = 0;
                unsigned long long as[6], ht[2];
                cudaMemcpy(c, cnt.p + 4 * std::max(list - 1, 0), sizeof c, cudaMemcpyDeviceToHost);
                cudaMemcpy(&nd, A.n_defer, sizeof nd, cudaMemcpyDeviceToHost);
                cudaMemcpy(as, astats.p, sizeof as, cudaMemcpyDeviceToHost);
                cudaMemcpy(ht, totals.p, sizeof ht, cudaMemcpyDeviceToHost);
                fprintf(stderr, "d3g level %d sets %d points %d groups %d of %d lanes: left to wider groups %d, "
                        "deferred so far %d, %.3f ms | inserted %llu attempts %llu lock-conflicts %llu walk-restarts %llu "
                        "bad-seeds %llu too-big %llu left %llu undecided %llu\n",
                        lev, sets_of[size_t(lev)], m_of[lev], int(std::min<int64_t>(groups_of[size_t(lev)], kMaxGroups)),
                        G, c[1], nd, ms, ht[0], ht[1], as[0], as[1], as[2], as[3], as[4], as[5]);
                cudaEventDestroy(ev0);
                cudaEventDestroy(ev1);
            }
            if (lev == nlev - 1) {
                // The points still left, with fewer and fewer groups in the way of one another.
                for (int k = 0; k < kLastPasses; ++k)
                    left_pass(std::max(kNumSMs * (kGroupThreads / 32) >> (3 * k), 16), k == kLastPasses - 1);
            }
            if (opt.validate || lev == nlev - 1) {
                D3G_TRY(drain());
                if (opt.validate) D3G_TRY(validate_tables("after", lev));
                if (opt.timing) cudaEventRecord(kev[0], s);
            }
        }
        return D3G_OK;
    };
    if (use_async) {
        D3G_TRY(run_async());
    } else {
        D3G_TRY(run_lockstep());
    }
    {
        unsigned long long hs2[2] = {0, 0}, ht[6], hst[2] = {0, 0}, hp[4] = {0, 0, 0, 0}, ha[6] = {};
        D3G_CUDA(cudaMemcpyAsync(hp, pstats.p, sizeof hp, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaMemcpyAsync(ha, astats.p, sizeof ha, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaMemcpyAsync(hs2, sums.p, sizeof hs2, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaMemcpyAsync(hst, steps.p, sizeof hst, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaMemcpyAsync(ht, totals.p, sizeof ht, cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaStreamSynchronize(s));
        R.stats.region_tets = int64_t(hs2[0]);
        R.stats.boundary_facets = int64_t(hs2[1]);
        R.stats.rounds = int(ht[2]);
        R.stats.attempts = int64_t(ht[1]);
        R.stats.walk_steps = int64_t(hst[0]);
        R.stats.bfs_steps = int64_t(hst[1]);
        R.stats.conflict_tests = int64_t(hp[0]);
        R.stats.uncertain_tests = int64_t(hp[1]);
        R.stats.tie_breaks = int64_t(hp[2]);
        R.stats.max_region_tets = int64_t(hp[3]);
        R.stats.deferred_points = int64_t(ha[5]);
        if (use_async) R.stats.async_inserted = int64_t(ht[0]) - to_rounds;
    }
    // Release round scratch before the output stage.
    wcav.release();
    wfac.release();
    wsv.release();
    wsn.release();
    alock.release();
    claim.release();
    fnew.release();

    cudaEventRecord(ph[2], s);
    nvtx_phase.reset();
    nvtx_phase.emplace("d3g.output");
    // ---- output: canonical cells ----
    int ntet = 0;
    D3G_CUDA(cudaMemcpyAsync(&ntet, tet_count.p, sizeof ntet, cudaMemcpyDeviceToHost, s));
    D3G_CUDA(cudaStreamSynchronize(s));
    const int kbits = bits_for(uint64_t(max_n) + 1);
    // Every cell's flag and place among the flagged (for the radix sorts).
    DevBuf<int32_t> flag, pos;
    auto flag_cells = [&](bool with_inf, int64_t* n) -> int {
        D3G_TRY(flag.alloc(size_t(ntet), s));
        D3G_TRY(pos.alloc(size_t(ntet), s));
        k_cell_flags<<<grid_for(ntet, 256), 256, 0, s>>>(rec.p, ntet, with_inf, flag.p);
        D3G_TRY(exclusive_scan(flag.p, pos.p, ntet, s));
        int last_pos = 0, last_flag = 0;
        D3G_CUDA(cudaMemcpyAsync(&last_pos, pos.p + ntet - 1, sizeof(int), cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaMemcpyAsync(&last_flag, flag.p + ntet - 1, sizeof(int), cudaMemcpyDeviceToHost, s));
        D3G_CUDA(cudaStreamSynchronize(s));
        *n = int64_t(last_pos) + last_flag;
        return D3G_OK;
    };
    auto radix_cells = [&](bool with_inf, DevBuf<int4>& out, int64_t* n) -> int {
        DevBuf<int4> raw;
        DevBuf<unsigned long long> khi, klo;
        DevBuf<int32_t> idx, cset;
        D3G_TRY(flag_cells(with_inf, n));
        D3G_TRY(raw.alloc(size_t(*n), s));
        D3G_TRY(khi.alloc(size_t(*n), s));
        D3G_TRY(klo.alloc(size_t(*n), s));
        D3G_TRY(idx.alloc(size_t(*n), s));
        if (!single) D3G_TRY(cset.alloc(size_t(*n), s));
        k_cells_out<<<grid_for(ntet, 256), 256, 0, s>>>(rec.p, flag.p, pos.p, ntet, vert_point.p, vset.p, kbits, raw.p,
                                                        khi.p, klo.p, idx.p, single ? nullptr : cset.p);
        D3G_TRY(sort_cells(raw, khi, klo, idx, single ? nullptr : cset.p, nsets, *n, kbits, out, s));
        return D3G_OK;
    };
    {
        // Buckets by first vertex; the radix sort of every cell only if a bucket is
        // too large for one block.
        DevBuf<int4> raw;
        DevBuf<int> bucket, bstart, bcount, ctl, mid;
        D3G_TRY(raw.alloc(size_t(ntet), s));
        D3G_TRY(bucket.alloc(size_t(ntet), s));
        D3G_TRY(bstart.alloc(size_t(N) + 1, s));
        D3G_TRY(bcount.alloc(size_t(N) + 1, s));
        D3G_TRY(ctl.alloc(3, s));
        D3G_TRY(mid.alloc(size_t(ntet / (kBucketThread + 1)) + 1, s));
        D3G_TRY(R.cells.alloc(size_t(ntet), s));
        D3G_CUDA(cudaMemsetAsync(bcount.p, 0, sizeof(int) * (size_t(N) + 1), s));
        D3G_CUDA(cudaMemsetAsync(ctl.p, 0, 3 * sizeof(int), s));
        k_cells_emit<<<unsigned((ntet + kEmitTets - 1) / kEmitTets), kEmitThreads, 0, s>>>(
            rec.p, ntet, vert_point.p, vset.p, d_off.p, !single, raw.p, bucket.p, bcount.p, ctl.p);
        D3G_TRY(exclusive_scan(bcount.p, bstart.p, int64_t(N) + 1, s));
        k_bucket_place<<<grid_for(ntet, 256), 256, 0, s>>>(raw.p, bucket.p, ctl.p, bstart.p, bcount.p, R.cells.p);
        k_bucket_sort<<<unsigned((N + 127) / 128), 128, 0, s>>>(R.cells.p, bstart.p, N, mid.p, ctl.p + 2, ctl.p + 1);
        int hctl[3] = {0, 0, 0};
        D3G_CUDA(cudaMemcpyAsync(hctl, ctl.p, sizeof hctl, cudaMemcpyDeviceToHost, s));
        if (!single) {
            DevBuf<int64_t> coff;
            D3G_TRY(coff.alloc(size_t(nsets) + 1, s));
            k_cell_off<<<grid_for(nsets + 1, 128), 128, 0, s>>>(bstart.p, d_off.p, nsets, coff.p);
            D3G_CUDA(cudaMemcpyAsync(R.cell_off.data(), coff.p, sizeof(int64_t) * (size_t(nsets) + 1),
                                     cudaMemcpyDeviceToHost, s));
        }
        D3G_CUDA(cudaStreamSynchronize(s));
        R.n_cells = hctl[0];
        if (single) R.cell_off[1] = R.n_cells;
        if (hctl[1]) D3G_TRY(radix_cells(false, R.cells, &R.n_cells));
        else if (hctl[2] > 0)
            k_bucket_sort_block<<<unsigned(hctl[2]), 512, 0, s>>>(R.cells.p, bstart.p, mid.p);
    }
    if (single && opt.want_all_cells) D3G_TRY(radix_cells(true, R.all, &R.n_all));
    if (single && opt.want_incident) {
        const int64_t m = 4 * R.n_cells;
        DevBuf<int32_t> pt, cell, pt2, cnt;
        D3G_TRY(R.inc_off.alloc(size_t(N) + 1, s));
        D3G_TRY(R.inc.alloc(size_t(m > 0 ? m : 1), s));
        D3G_TRY(cnt.alloc(size_t(N) + 1, s));
        D3G_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(int32_t) * (size_t(N) + 1), s));
        if (m > 0) {
            D3G_TRY(pt.alloc(size_t(m), s));
            D3G_TRY(cell.alloc(size_t(m), s));
            D3G_TRY(pt2.alloc(size_t(m), s));
            k_incident_pairs<<<grid_for(R.n_cells, 256), 256, 0, s>>>(R.cells.p, R.n_cells, pt.p, cell.p,
                                                                     cnt.p);
            D3G_TRY(sort_pairs(pt.p, pt2.p, cell.p, R.inc.p, m, 0, bits_for(uint64_t(N)), s));
        }
        DevBuf<int64_t> cnt64;
        D3G_TRY(cnt64.alloc(size_t(N) + 1, s));
        k_widen<<<grid_for(n + 1, 256), 256, 0, s>>>(cnt.p, n + 1, cnt64.p);
        D3G_TRY(exclusive_scan(cnt64.p, R.inc_off.p, n + 1, s));
        R.n_inc = m;
    }
    D3G_CUDA(cudaGetLastError());
    cudaEventRecord(ph[3], s);
    D3G_CUDA(cudaMemcpyAsync(hst, status.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    D3G_CUDA(cudaStreamSynchronize(s));
    {
        float a = 0.f, b = 0.f, c = 0.f;
        cudaEventElapsedTime(&a, ph[0], ph[1]);
        cudaEventElapsedTime(&b, ph[1], ph[2]);
        cudaEventElapsedTime(&c, ph[2], ph[3]);
        R.stats.ms_order = a;
        R.stats.ms_rounds = b;
        R.stats.ms_output = c;
    }
    return status_from_bits(hst[0]);
}

}  // namespace d3g

using namespace d3g;

namespace d3g {
namespace {

// The settings d3g_autotune_device chose, per device (d3g_options_default
// hands them out).
constexpr int kMaxTunedDevices = 64;
std::mutex g_tuning_mu;
d3g_tuning g_tuning[kMaxTunedDevices];
bool g_tuned[kMaxTunedDevices] = {};

bool current_tuning(d3g_tuning* out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxTunedDevices) {
        cudaGetLastError();
        return false;
    }
    std::lock_guard<std::mutex> lock(g_tuning_mu);
    if (!g_tuned[dev]) return false;
    *out = g_tuning[dev];
    return true;
}

}  // namespace
}  // namespace d3g

extern "C" {

void d3g_options_default(d3g_options* o) {
    if (!o) return;
    o->want_all_cells = 1;
    o->want_incident = 1;
    o->chunk = 0;
    o->max_rounds = 0;
    o->timing = 0;
    o->alpha_small = 24;
    o->lanes = 0;
    o->schedule = 0;
    o->split = 0;
    o->tet_capacity = 0;
    o->walk_limit = 0;
    o->cavity_capacity = 0;
    o->level_growth = 0;
    // D3G_VALIDATE=1 in the environment turns the device self-check on for every
    // build that takes the defaults (as the reference's DEL3D_VALIDATE builds do).
    const char* val = getenv("D3G_VALIDATE");
    o->validate = (val && val[0] && val[0] != '0') ? 1 : 0;
    d3g_tuning t;
    if (current_tuning(&t)) {
        o->schedule = t.schedule;
        o->chunk = t.chunk;
        o->alpha_small = t.alpha_small;
        o->lanes = t.lanes;
    }
}

int d3g_get_tuning(d3g_tuning* out) {
    if (!out) return D3G_ERR_INVALID_ARGUMENT;
    if (!current_tuning(out)) {
        d3g_options o;
        d3g_options_default(&o);
        *out = d3g_tuning{o.schedule, o.chunk, o.alpha_small, o.lanes, 0.0, 0};
    }
    return D3G_OK;
}

int d3g_reset_tuning(void) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxTunedDevices) {
        cudaGetLastError();
        return D3G_ERR_NO_DEVICE;
    }
    std::lock_guard<std::mutex> lock(g_tuning_mu);
    g_tuned[dev] = false;
    return D3G_OK;
}

int d3g_autotune_device(const double* d_xyz, const int64_t* set_offsets, int32_t n_sets, void* stream,
                        d3g_tuning* best) {
    if (n_sets < 1 || !set_offsets || set_offsets[0] != 0 || set_offsets[n_sets] < 0 ||
        (set_offsets[n_sets] > 0 && !d_xyz))
        return D3G_ERR_INVALID_ARGUMENT;
    D3G_TRY(ensure_device());
    int dev = 0;
    D3G_CUDA(cudaGetDevice(&dev));
    if (dev >= kMaxTunedDevices) return D3G_ERR_NO_DEVICE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // Candidates: the schedule, the worker density (one worker per `alpha`
    // earlier points, denser below one wave: `alpha_small`) and, for the
    // lockstep rounds, the lanes per worker.  Every setting gives the same
    // cells; only the time differs.
    struct Cand { int schedule, alpha, alpha_small, lanes; };
    std::vector<Cand> cands;
    for (int a : {24, 48, 96})
        for (int as : {12, 24}) cands.push_back({0, a, as, 0});
    for (int a : {24, 48})
        for (int l : {32, 16}) cands.push_back({1, a, 24, l});
    cudaEvent_t e0, e1;
    D3G_CUDA(cudaEventCreate(&e0));
    D3G_CUDA(cudaEventCreate(&e1));
    d3g_tuning win{0, 0, 24, 0, 1e30, 0};
    int st = D3G_OK;
    for (const Cand& c : cands) {
        d3g_options o;
        d3g_options_default(&o);
        o.want_all_cells = 0;
        o.want_incident = 0;
        o.schedule = c.schedule;
        o.chunk = -c.alpha;
        o.alpha_small = c.alpha_small;
        o.lanes = c.lanes;
        float best_ms = 1e30f;
        for (int rep = 0; rep < 2 && st == D3G_OK; ++rep) {   // first run warms the pool
            DeviceResult R;
            cudaEventRecord(e0, s == nullptr ? cudaStreamLegacy : s);
            st = build_on_stream(d_xyz, set_offsets, n_sets, o, s, R);
            cudaEventRecord(e1, s == nullptr ? cudaStreamLegacy : s);
            R.reset();
            if (st != D3G_OK) break;
            if (cudaEventSynchronize(e1) != cudaSuccess) {
                st = D3G_ERR_CUDA;
                break;
            }
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (rep > 0) best_ms = ms;
        }
        if (st != D3G_OK) break;
        win.candidates += 1;
        if (best_ms < win.ms) win = d3g_tuning{c.schedule, -c.alpha, c.alpha_small, c.lanes, best_ms, win.candidates};
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st != D3G_OK) return st;
    {
        std::lock_guard<std::mutex> lock(g_tuning_mu);
        g_tuning[dev] = win;
        g_tuned[dev] = true;
    }
    if (best) *best = win;
    return D3G_OK;
}

void d3g_result_free(d3g_result* r) {
    if (!r) return;
    host_result_free(r->cells);
    host_result_free(r->all_cells);
    host_result_free(r->incident_offsets);
    host_result_free(r->incident);
    *r = d3g_result{};
}

int d3g_build(const double* xyz, int64_t n, const d3g_options* opts, d3g_result* out) {
    if (!out || n < 0 || (n > 0 && !xyz)) return D3G_ERR_INVALID_ARGUMENT;
    *out = d3g_result{};
    d3g_options o;
    d3g_options_default(&o);
    if (opts) o = *opts;
    out->n_points = n;
    if (n == 0) {
        out->incident_offsets = static_cast<int64_t*>(calloc(1, sizeof(int64_t)));
        return D3G_OK;
    }
    D3G_TRY(ensure_device());
    cudaStream_t s = nullptr;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int st;
    DeviceResult R;
    {
        DevBuf<double> dx;
        D3G_TRY(dx.alloc(size_t(3 * n), s));
        D3G_CUDA(cudaMemcpyAsync(dx.p, xyz, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, s));
        cudaEventRecord(e0, s);
        st = build_on_stream(dx.p, n, o, s, R);
        cudaEventRecord(e1, s);
    }
    if (st == D3G_OK) {
        out->n_vertices = R.n_vertices;
        out->n_cells = R.n_cells;
        out->n_all = R.n_all;
        out->stats = R.stats;
        out->cells = static_cast<int32_t*>(host_result_alloc(sizeof(int32_t) * 4 * size_t(R.n_cells > 0 ? R.n_cells : 1)));
        if (R.n_cells > 0)
            cudaMemcpyAsync(out->cells, R.cells.p, sizeof(int4) * R.n_cells, cudaMemcpyDeviceToHost, s);
        if (o.want_all_cells) {
            out->all_cells = static_cast<int32_t*>(host_result_alloc(sizeof(int32_t) * 4 * size_t(R.n_all > 0 ? R.n_all : 1)));
            if (R.n_all > 0)
                cudaMemcpyAsync(out->all_cells, R.all.p, sizeof(int4) * R.n_all, cudaMemcpyDeviceToHost, s);
        }
        if (o.want_incident) {
            out->incident_offsets = static_cast<int64_t*>(host_result_alloc(sizeof(int64_t) * (size_t(n) + 1)));
            out->incident = static_cast<int32_t*>(host_result_alloc(sizeof(int32_t) * size_t(R.n_inc > 0 ? R.n_inc : 1)));
            cudaMemcpyAsync(out->incident_offsets, R.inc_off.p, sizeof(int64_t) * (n + 1),
                            cudaMemcpyDeviceToHost, s);
            if (R.n_inc > 0)
                cudaMemcpyAsync(out->incident, R.inc.p, sizeof(int32_t) * R.n_inc, cudaMemcpyDeviceToHost, s);
        }
        const cudaError_t e = cudaStreamSynchronize(s);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        out->device_ms = ms;
        if (e != cudaSuccess) {
            set_error(std::string("d3g_build: ") + cudaGetErrorString(e));
            st = D3G_ERR_CUDA;
        }
    }
    R.reset();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st != D3G_OK) d3g_result_free(out);
    return st;
}

int d3g_build_device(const double* d_xyz, int64_t n, const d3g_options* opts, int32_t* d_cells,
                     int64_t cap_cells, int64_t* n_cells_out, int64_t* n_vertices_out, void* stream,
                     d3g_build_stats* stats) {
    if (n < 0 || (n > 0 && !d_xyz) || cap_cells < 0) return D3G_ERR_INVALID_ARGUMENT;
    d3g_options o;
    d3g_options_default(&o);
    if (opts) o = *opts;
    o.want_all_cells = 0;
    o.want_incident = 0;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    DeviceResult R;
    const int st = build_on_stream(d_xyz, n, o, s, R);
    if (st != D3G_OK) return st;
    if (n_cells_out) *n_cells_out = R.n_cells;
    if (n_vertices_out) *n_vertices_out = R.n_vertices;
    if (stats) *stats = R.stats;
    if (R.n_cells > cap_cells) {
        set_error("d3g_build_device: output capacity too small");
        return D3G_ERR_INVALID_ARGUMENT;
    }
    if (R.n_cells > 0) {
        if (!d_cells) return D3G_ERR_INVALID_ARGUMENT;
        D3G_CUDA(cudaMemcpyAsync(d_cells, R.cells.p, sizeof(int4) * R.n_cells, cudaMemcpyDeviceToDevice, s));
    }
    R.reset();
    D3G_CUDA(cudaStreamSynchronize(s));
    return D3G_OK;
}

}  // extern "C"

extern "C" {

void d3g_batch_result_free(d3g_batch_result* r) {
    if (!r) return;
    host_result_free(r->cell_offsets);
    host_result_free(r->cells);
    host_result_free(r->n_vertices);
    *r = d3g_batch_result{};
}

int d3g_build_batch(const double* xyz, const int64_t* set_offsets, int32_t n_sets, const d3g_options* opts,
                    d3g_batch_result* out) {
    if (!out || n_sets < 1 || !set_offsets) return D3G_ERR_INVALID_ARGUMENT;
    *out = d3g_batch_result{};
    const int64_t n = set_offsets[n_sets];
    if (set_offsets[0] != 0 || n < 0 || (n > 0 && !xyz)) return D3G_ERR_INVALID_ARGUMENT;
    d3g_options o;
    d3g_options_default(&o);
    if (opts) o = *opts;
    D3G_TRY(ensure_device());
    cudaStream_t s = nullptr;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int st;
    DeviceResult R;
    {
        DevBuf<double> dx;
        D3G_TRY(dx.alloc(size_t(3 * (n > 0 ? n : 1)), s));
        if (n > 0) D3G_CUDA(cudaMemcpyAsync(dx.p, xyz, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, s));
        cudaEventRecord(e0, s);
        st = build_on_stream(dx.p, set_offsets, n_sets, o, s, R);
        cudaEventRecord(e1, s);
    }
    if (st == D3G_OK) {
        out->n_sets = n_sets;
        out->stats = R.stats;
        out->cell_offsets = static_cast<int64_t*>(host_result_alloc(sizeof(int64_t) * (size_t(n_sets) + 1)));
        out->n_vertices = static_cast<int64_t*>(host_result_alloc(sizeof(int64_t) * size_t(n_sets)));
        out->cells = static_cast<int32_t*>(host_result_alloc(sizeof(int32_t) * 4 * size_t(R.n_cells > 0 ? R.n_cells : 1)));
        for (int i = 0; i <= n_sets; ++i) out->cell_offsets[i] = R.cell_off[size_t(i)];
        for (int i = 0; i < n_sets; ++i) out->n_vertices[i] = R.set_nv[size_t(i)];
        if (R.n_cells > 0)
            cudaMemcpyAsync(out->cells, R.cells.p, sizeof(int4) * R.n_cells, cudaMemcpyDeviceToHost, s);
        const cudaError_t e = cudaStreamSynchronize(s);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        out->device_ms = ms;
        if (e != cudaSuccess) {
            set_error(std::string("d3g_build_batch: ") + cudaGetErrorString(e));
            st = D3G_ERR_CUDA;
        }
    }
    R.reset();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st != D3G_OK) d3g_batch_result_free(out);
    return st;
}

int d3g_build_batch_device(const double* d_xyz, const int64_t* set_offsets, int32_t n_sets,
                           const d3g_options* opts, int32_t* d_cells, int64_t cap_cells,
                           int64_t* cell_offsets, int64_t* n_vertices, void* stream, d3g_build_stats* stats) {
    if (n_sets < 1 || !set_offsets || cap_cells < 0) return D3G_ERR_INVALID_ARGUMENT;
    if (set_offsets[0] != 0 || set_offsets[n_sets] < 0 || (set_offsets[n_sets] > 0 && !d_xyz))
        return D3G_ERR_INVALID_ARGUMENT;
    d3g_options o;
    d3g_options_default(&o);
    if (opts) o = *opts;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    DeviceResult R;
    const int st = build_on_stream(d_xyz, set_offsets, n_sets, o, s, R);
    if (st != D3G_OK) return st;
    if (cell_offsets)
        for (int i = 0; i <= n_sets; ++i) cell_offsets[i] = R.cell_off[size_t(i)];
    if (n_vertices)
        for (int i = 0; i < n_sets; ++i) n_vertices[i] = R.set_nv[size_t(i)];
    if (stats) *stats = R.stats;
    if (R.n_cells > cap_cells) {
        set_error("d3g_build_batch_device: output capacity too small");
        return D3G_ERR_INVALID_ARGUMENT;
    }
    if (R.n_cells > 0) {
        if (!d_cells) return D3G_ERR_INVALID_ARGUMENT;
        D3G_CUDA(cudaMemcpyAsync(d_cells, R.cells.p, sizeof(int4) * R.n_cells, cudaMemcpyDeviceToDevice, s));
    }
    R.reset();
    D3G_CUDA(cudaStreamSynchronize(s));
    return D3G_OK;
}

}  // extern "C"
