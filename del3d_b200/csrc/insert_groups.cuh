// The asynchronous insertion kernel (included by build.cu, inside its
// anonymous namespace).
//
// A group of G lanes inserts one point at a time; 32 / G groups share a warp
// and go through the phases of an insertion - fetch, walk, grow, re-star,
// publish - together: every loop runs until all groups of the warp are done, so
// their memory accesses are issued together and no phase is executed twice.
// A conflict region has about 21 tets and 28 boundary facets and offers about
// 64 facets to test, most of them in steps of fewer than 32: with G = 32 half
// of the lanes idle, with G = 8 nearly none do.
//
// Locking is the one described at "asynchronous insertion" in build.cu.  Tet
// slots that hold no tet yet are locked (-1) from the start, so a slot handed
// out needs no lock of its own: it is released when its tet is written.
//
// Everything an insertion needs between reading the mesh and writing it - the
// facets still to test, the region's tets, the boundary facets with their
// vertices - stays in shared memory, so each tet and each lock word goes over
// L2 once per insertion, but for a record read along with its lock attempt and
// again under the lock.

constexpr int kGroupThreads = 128;
/// Blocks per SM the insertion kernel is compiled for: 20 warps at 96 registers
/// (94 used with 8 or 16 lanes, 96 with 32; no spills) and 38 KB of scratch a block.  With 6 (80 registers, 80
/// bytes of spills, 228 KB of the SM's 256 taken by scratch, so spills miss L1)
/// 4096 mixed sets took 440 ms against 409, with 4 457 against 429.
constexpr int kGroupBlocks = 5;
constexpr int kExactBlocks = 2;       // the same with kExact (255 registers)
constexpr int kGroupStash = 6;        // points a group keeps to try again later
constexpr int kGroupTries = 24;       // attempts before a point is left
constexpr int kWaitPolls = 150;       // polls of a lock before its holder's point is given way to
/// The same with kExact: an insertion with a dozen steps in the exact stage holds its locks
/// for some 300 us, ten times as long as others.
constexpr int kExactTries = 100, kExactPolls = 2000;
/// Region tets and boundary facets of the widest groups' last pass (139 KB of scratch;
/// 4096 mixed sets, whose largest region is 2592 tets, with 2048 386 ms, since the
/// region beyond it needed the rounds and their tables; with this 377, with 6144 the same).
constexpr int kBigCapacity = 4096;
constexpr int kPoolSlots = 16;        // tet slots a group takes from the table at a time

/// kCap: region tets, and boundary facets, a group has room for.
template <int G, int kCapacity>
struct alignas(16) GroupScratch {
    static constexpr int kCap = kCapacity;
    static constexpr int kFront = 3 * kCap + 4;     // facets met: three per region tet, four at the seed
    static constexpr int kTable = 2 * kCap;         // edges: at most 3/2 per facet
    int now[G];           // growth: the region tets each lane found in this step
    int4 fac[kCap];       // boundary facets: a, b, c and the outside facet (tet * 4 + facet), its sign
                          // bit set if another facet's entry holds the outside tet's lock
    int reg[kCap];        // region tets
    union {
        int front[kFront];                          // growth: facets across which the region may go on
        struct {
            unsigned table[kTable];                 // re-star: hash table of the boundary's edges
            uint16_t link[3 * kCap];                // partner of each facet's three edges
        } m;
    };
    int stash[kGroupStash], stash_tries[kGroupStash];
    // The group's state between points (here, not in registers: the growth loop needs those).
    int nstash, open;                               // points to try again; more points may be had
    int item, attempt, vlo, vhi;                    // the point in hand, its failed attempts, its set's vertices
    unsigned won, tries, nC, nF;
    int4 pool;                                      // tet slots in hand: [x, x + y), then [z, z + w)
};

/// What a launch works on and where it leaves what it could not do.
struct GroupArgs {
    int* lock;
    const int* items;        // points to insert (-1: nothing to do)
    const int* guide;        // per vertex: a vertex near it that should be in already
    const int* n_items;      // how many
    int first, most;         // of them, the launch takes those from `first` on, at most `most`
    int* hint;               // per vertex: a tet near it (k_locate), -1: none
    int* next;               // queue head
    int* left;               // points to try again by wider groups or with kNear (regions too big, too many
                             // conflicts, undecided tests), ...
    int* n_left;
    int* defer;              // ... points with a test that kNear cannot decide either (for kExact), ...
    int* n_defer;
    int* big;                // ... and points whose region has no room with the widest groups
    int* n_big;
    int4* pool;              // per group: tet slots it holds (GroupScratch::pool)
    const int4* skips;       // per set: its first tet's vertices
    const uint8_t* set_exact;    // per set: EX_*
    const double* inv_grid;      // per set: see in_sphere_near
    const int32_t* voff;     // per set: its vertices
    unsigned long long* stats;   // as AsyncCtx::stats
    int cavity;              // region tets at most (and twice as many boundary facets), if fewer than kCap
    int ngroups;
};

__device__ __forceinline__ int cas_lock(int* p, int value) {
    int old;
    asm volatile("atom.acquire.gpu.global.cas.b32 %0, [%1], 0, %2;" : "=r"(old) : "l"(p), "r"(value) : "memory");
    return old;
}
__device__ __forceinline__ void set_lock(int* p, int value) {
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(value) : "memory");
}
/// A tet's whole record in one access, past L1.
__device__ __forceinline__ void ld_rec(const Tables& T, int t, int4& tv, int4& tn) {
    asm volatile("ld.relaxed.gpu.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(tv.x), "=r"(tv.y), "=r"(tv.z), "=r"(tv.w), "=r"(tn.x), "=r"(tn.y), "=r"(tn.z), "=r"(tn.w)
                 : "l"(&T.tv(t))
                 : "memory");
}
__device__ __forceinline__ void st_rec(const Tables& T, int t, const int4& tv, const int4& tn) {
    asm volatile("st.relaxed.gpu.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(&T.tv(t)), "r"(tv.x),
                 "r"(tv.y), "r"(tv.z), "r"(tv.w), "r"(tn.x), "r"(tn.y), "r"(tn.z), "r"(tn.w)
                 : "memory");
}

/// Five blocks with their static shared memory (counters, queue) and the 1 KB that the
/// system takes of each leave L1 60 KB.
static_assert(kGroupBlocks * (sizeof(GroupScratch<8, 64>) * 16 + 15 * kCounterThreads + 64 + 1024) <= 196 * 1024,
              "k_insert_groups' shared memory");

/// The most groups a launch has.
constexpr int kMaxGroups = kNumSMs * kGroupBlocks * (kGroupThreads / 8);

/// Lanes a group gets at a level with work for `groups` of them.  Wide groups
/// finish one insertion sooner (28 K cycles with 32 lanes, 41 K with 16, 65 K with
/// 8 on a quiet GPU), narrow ones insert more per instruction; a level with work
/// for more groups than the GPU holds at 32 or 16 lanes (2960, 5920) twice over is
/// worth the narrower ones.  10^6 uniform points: 21.6 ms by this rule, 22.9 with the
/// lines at 6000 and 3000, 22.3 with 32 lanes throughout; 10^7: 106, 109 and 131 ms;
/// 4096 mixed sets: 405, 407 and 546 ms.
inline int group_lanes(int64_t groups) { return groups >= 12000 ? 8 : (groups >= 6000 ? 16 : 32); }

/// A live tet incident to vertex `guide` of the set with vertices from `vlo` -
/// or, while that vertex is not in, to the nearest before it that is, or to the
/// set's first tet's `first`.
__device__ __forceinline__ int tet_near(const Tables& T, int guide, int vlo, int first) {
    int t = guide >= 0 ? __ldcg(T.vert_tet + guide) : -1;
    for (int u = guide - 1, k = 0; t < 0 && u >= vlo && k < 64; --u, ++k) t = __ldcg(T.vert_tet + u);
    if (t < 0) t = __ldcg(T.vert_tet + first);
    return max(t, 0);
}

/// The mesh in device memory, as k_insert_groups sees it.
struct GlobalMesh {
    const Tables& T;
    const GroupArgs& A;
    const double* __restrict__ vx;
    static constexpr int kPool = kPoolSlots;
    static constexpr bool kLocal = false;
    __device__ __forceinline__ Pt point(int v) const { return vpt(vx, v); }
    __device__ __forceinline__ Pt again(int v) const { return ld_vertex(vx, v); }   // not kept in registers
    __device__ __forceinline__ double inv(int v) const { return A.inv_grid[T.vset[v]]; }
    __device__ __forceinline__ int4 tv4(int t) const { return ld4(&T.tv(t)); }
    __device__ __forceinline__ int4 tn4(int t) const { return ld4(&T.tn(t)); }
    __device__ __forceinline__ void rec(int t, int4& tv, int4& tn) const { ld_rec(T, t, tv, tn); }
    __device__ __forceinline__ void store(int t, const int4& tv, const int4& tn) const { st_rec(T, t, tv, tn); }
    __device__ __forceinline__ void link(int enc, int to) const { T.link(enc) = to; }
    __device__ __forceinline__ void kill(int t) const { T.kill(t); }
    __device__ __forceinline__ void vert(int v, int t) const { T.vert_tet[v] = t; }
    __device__ __forceinline__ int cas(int t, int value) const { return cas_lock(A.lock + t, value); }
    __device__ __forceinline__ void set(int t, int value) const { set_lock(A.lock + t, value); }
    __device__ __forceinline__ int take(int n) const { return atomicAdd(T.tet_count, n); }
    __device__ __forceinline__ int cap() const { return T.cap; }
    __device__ __forceinline__ int walk_limit() const { return T.walk_limit; }
    __device__ __forceinline__ int start(int v, int vlo) const {
        return tet_near(T, A.guide[v], vlo, A.skips[T.vset[v]].x);
    }
    __device__ __forceinline__ void fence() const { __threadfence(); }
};

/// How a kernel treats a test its filter cannot decide: it gives the point up, settles
/// the test for near points on a grid (in_sphere_near), or settles every test (the
/// exact stage, out of line).
enum : int { kFilter = 0, kNear = 1, kExact = 2 };

/// orient_facet_filter's sign from the exact stage; 0 as well where the stage's limbs
/// do not reach (the walk then does not cross the facet).
__device__ __noinline__ int orient_facet_exact(const double* __restrict__ vx, int4 t, int i, int v) {
    const int x = i == 0 ? t.z : (i == 2 ? t.y : t.x);
    const int y = i == 0 ? t.y : (i == 1 ? t.z : (i == 2 ? t.x : t.y));
    const int z = i == 3 ? t.z : t.w;
    return orient3d(vpt(vx, x), vpt(vx, y), vpt(vx, z), vpt(vx, v), nullptr);
}

/// Locates a level's points, one thread each, in the mesh as it is before the
/// level: the walk of an insertion, which has a group's lanes wait for one chain
/// of reads, then starts a step or two from its end.  Reads may use L1, since
/// nothing writes the mesh meanwhile.  A facet the filter cannot decide is not
/// crossed and a long walk ends where it is: the tet is only where the insertion
/// starts.
__global__ void __launch_bounds__(128) k_locate(Tables T, GroupArgs A, const double* __restrict__ vx) {
    const GlobalMesh m{T, A, vx};
    const int n = *A.n_items;
    for (int k = int(blockIdx.x) * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int v = A.items[k];
        if (v < 0) continue;
        const int set = T.vset[v];
        const bool ex = A.set_exact[set] & EX_ORIENT;
        const Pt p = vpt(vx, v);
        int t = tet_near(T, A.guide[v], A.voff[set], A.skips[set].x);
        int4 tv = T.tv(t);
        const int ip = inf_pos(tv);
        if (ip >= 0) {
            t = at(T.tn(t), ip) >> 2;
            tv = T.tv(t);
        }
        int prev = -1;
        uint32_t h = uint32_t(v) * 2654435761u + 12345u;
        for (int step = 0; step < 128; ++step) {
            const int4 tn = T.tn(t);
            h = h * 1664525u + 1013904223u;
            int next = -1;
#pragma unroll 1
            for (int k2 = 0; k2 < 4 && next < 0; ++k2) {
                const int i = int((h >> 30) + unsigned(k2)) & 3;
                const int nb = at(tn, i) >> 2;
                if (nb == prev) continue;
                if (orient_facet_filter(m, tv, i, p, ex) < 0) next = nb;
            }
            if (next < 0) break;
            prev = t;
            t = next;
            tv = T.tv(t);
            if (inf_pos(tv) >= 0) break;
        }
        A.hint[v] = t;
    }
}

/// One attempt of each of the warp's groups to insert its point v (`live`: it has
/// one), the walk starting at tet t: walk, grow, re-star, publish.  Returns AI_*
/// (-1 for a group without a point); `t` becomes the seed, -1 after a walk that hit
/// its limit.  M is where the mesh lies: in device memory (GlobalMesh) or in a
/// block's shared memory (SharedMesh).
template <int G, int kMode, class M, class Scratch>
__device__ __forceinline__ int insert_step(const M& m, Scratch& S, const Lanes<G>& L, int group, bool live, int v, int ex,
                                           int& t, int cavity, uint32_t* status, unsigned long long* stats,
                                           const SharedCounters& ctr, unsigned& tests, uint32_t* lacking = nullptr) {
    constexpr int kPool = M::kPool;
    const unsigned lt = (1u << L.lane) - 1u;
    const int region = (group + 1) << 1, ring = region | 1;
    const Pt p = m.point(v);
    cavity = min(cavity, Scratch::kCap);
    const int fac_cap = min(2 * cavity, Scratch::kCap);

    // Slots for its new tets, asked for here so that the answer is there by the re-star.
    const bool ask = live && S.pool.w == 0 && S.pool.y < kPool;
    int block = 0;
    if (L.sub == 0 && ask) block = m.take(kPool);

    // ---- walk (see walk_async; lanes 0-3 test the facets, lanes 4-7 fetch the
    //      neighbours' records) ----
    // A facet the filter cannot decide is not crossed (kExact: the exact stage
    // decides it): the seed is tested in any case, and if it fails the test the
    // point is deferred.
    int outcome = live ? AI_DONE : -1;
    bool fuzzy = false;
    {
        int4 tv, tn;
        m.rec(t, tv, tn);
        if (live && tv.x == tv.y) {                   // the hint's tet has gone since
            t = m.start(v, S.vlo);
            m.rec(t, tv, tn);
        }
        t = __shfl_sync(kFull, t, L.gbase);
        const int ip = inf_pos(tv);
        if (live && ip >= 0) {
            t = at(tn, ip) >> 2;
            m.rec(t, tv, tn);
        }
        int prev = -1, step = 0;
        // Another way and more steps at each attempt, so that a point whose way is very long
        // (along the hull of points nearly in a line, say) does not go it time and again.
        const int attempt = S.attempt;
        uint32_t h = (uint32_t(v) + uint32_t(attempt) * 0x9E3779B9u) * 2654435761u + 12345u;
        const int limit = min(min(kAsyncWalkLimit, 1024 << min(attempt, 4)), m.walk_limit());
        bool walking = live;
        while (__any_sync(kFull, walking)) {
            int4 pv = make_int4(0, 0, 0, 0), pn = pv;
            if (!M::kLocal && walking && L.sub >= 4 && L.sub < 8) m.rec(at(tn, L.sub & 3) >> 2, pv, pn);
            h = h * 1664525u + 1013904223u;
            const int s0 = int(h >> 30);
            bool neg = false;
            if (walking && L.sub < 4 && (at(tn, L.sub) >> 2) != prev && min(min(tv.x, tv.y), min(tv.z, tv.w)) >= 0) {
                int o = orient_facet_filter(m, tv, L.sub, p, ex & EX_ORIENT);
                if constexpr (kMode == kExact)
                    if (o == 2) o = orient_facet_exact(m.vx, tv, L.sub, v);
                fuzzy = fuzzy || o == 2;
                neg = o < 0;
            }
            const unsigned cross = L.own(__ballot_sync(kFull, neg)) & 0xFu;
            const unsigned rot = ((cross >> s0) | (cross << (4 - s0))) & 0xFu;
            const int i = (s0 + __ffs(int(rot)) - 1) & 3;
            int4 nv, nn;
            if (M::kLocal) {                              // the chosen neighbour is as near as a shuffle
                m.rec(cross ? at(tn, i) >> 2 : t, nv, nn);
            } else {
                const int src = L.gbase + 4 + i;
                nv = make_int4(__shfl_sync(kFull, pv.x, src), __shfl_sync(kFull, pv.y, src),
                               __shfl_sync(kFull, pv.z, src), __shfl_sync(kFull, pv.w, src));
                nn = make_int4(__shfl_sync(kFull, pn.x, src), __shfl_sync(kFull, pn.y, src),
                               __shfl_sync(kFull, pn.z, src), __shfl_sync(kFull, pn.w, src));
            }
            if (!walking) continue;
            if (cross == 0) {
                walking = false;
            } else {
                const int next = at(tn, i) >> 2;
                prev = t;
                t = next;
                tv = nv;
                tn = nn;
                if (inf_pos(nv) >= 0) {
                    walking = false;
                } else if (++step >= limit) {
                    outcome = AI_RETRY;
                    walking = false;
                    if (attempt & 1) t = -1;        // from the guide again, else on from here
                    if (L.sub == 0) atomicAdd(stats + 1, 1ull);
                }
            }
        }
    }

    // ---- grow: the seed is the first facet to test; a region tet adds the
    //      three facets other than the one it was reached through ----
    int nreg = 0, nfac = 0, head = 0, nfront = 1;
    bool growing = live && outcome == AI_DONE;
    if (L.sub == 0) S.front[0] = t * 4;
    __syncwarp();
    fuzzy = L.own(__ballot_sync(kFull, fuzzy)) != 0;
    while (__any_sync(kFull, growing)) {
        const bool valid = growing && head + L.sub < nfront;
        int enc = 0, kind = 0;      // 1: boundary facet, 2: new region tet, 3: decided below
        bool got = false, abort = false, undecided = false, bad_seed = false;
        int4 tv = make_int4(0, 0, 0, 0), tn = tv;
        if (valid) {
            enc = S.front[head + L.sub];
            const int nb = enc >> 2;
            // In device memory the record is read along with the lock attempt, so that its
            // vertices are known one trip to L2 earlier; the copy read under the lock decides.
            int4 guess = tv, ignore;
            if (!M::kLocal) m.rec(nb, guess, ignore);
            int seen = m.cas(nb, ring);
            if (G == 32) {
                // Of two insertions in each other's way one must go on: a group waits for
                // one with a higher number, which gives way itself when it meets this one's
                // locks (so no two wait for each other), and gives way to one with a lower
                // number.  Not for narrower groups, where the other may be in the same warp.
                for (int k = 0; k < (kMode == kExact ? kExactPolls : kWaitPolls) && seen > ring; ++k) {
                    __nanosleep(200);
                    seen = m.cas(nb, ring);
                }
            }
            got = seen == 0;
            if (seen == ring) kind = 3;               // locked by this group: in this step, or before
            else if (!got && seen != region) abort = true;   // another group holds it
            if (got || kind == 3) m.rec(nb, tv, tn);
            if (M::kLocal) guess = tv;
            if (got) {
                int r = 0;
                for (;;) {
                    r = in_conflict_fast<kMode != kFilter>(m, nb, guess, p, v, ex);
                    if (guess.x == tv.x && guess.y == tv.y && guess.z == tv.z && guess.w == tv.w) break;
                    guess = tv;
                }
                if (nreg == 0) {
                    // The seed may come from a half-written record: only a live
                    // tet of the point's own set will do.
                    const int u = tv.x != kInf ? tv.x : tv.y;
                    bad_seed = tv.x == tv.y || u < S.vlo || u >= S.vhi;
                    if (bad_seed) r = 0;
                }
                if constexpr (kMode == kExact) {
                    // Where the exact stage's limbs do not reach either, the point waits: with
                    // others in, the test may no longer come up.
                    if (r & CT_UNDECIDED) {
                        *lacking = 0;
                        r = conflict_test_exact(tv, p.x, p.y, p.z, v, m.vx, (ex & EX_BOTH) == EX_BOTH, lacking);
                        if (*static_cast<volatile uint32_t*>(lacking)) r = CT_UNCERTAIN | CT_UNDECIDED;
                    }
                }
                ++tests;
                if (r & (CT_UNCERTAIN | CT_TIE)) ctr.count(r);
                undecided = (r & CT_UNDECIDED) != 0;
                kind = (r & CT_IN) ? 2 : 1;
                if (kind == 2) m.set(nb, region);
                else if (nreg == 0) bad_seed = true;
            }
        }
        __syncwarp();
        const unsigned mc = __ballot_sync(kFull, kind == 2) & L.gm;
        if (__any_sync(kFull, kind == 3)) {
            // A tet met twice in this step is in the region if the lane that took its
            // lock found it so; one locked in an earlier step and not since made part
            // of the region is outside.
            S.now[L.sub] = kind == 2 ? enc >> 2 : -1;
            __syncwarp();
            if (kind == 3) {
                bool in = false;
#pragma unroll
                for (int k = 0; k < G; k += 4) {
                    const int4 w = *reinterpret_cast<const int4*>(S.now + k);
                    const int nb = enc >> 2;
                    in = in || w.x == nb || w.y == nb || w.z == nb || w.w == nb;
                }
                kind = in ? 0 : 1;
            }
        }
        const unsigned trouble = L.own(__ballot_sync(kFull, abort || undecided || bad_seed));
        const unsigned mf = __ballot_sync(kFull, kind == 1) & L.gm;
        const int nc = __popc(mc), nf = __popc(mf);
        const bool full = nreg + nc > cavity || nfac + nf > fac_cap;
        const bool stop = growing && (trouble || full);
        if (__any_sync(kFull, stop)) {
            const unsigned und = L.own(__ballot_sync(kFull, undecided));
            const unsigned ab = L.own(__ballot_sync(kFull, abort));
            if (stop) {
                // Give everything back: this step's locks, the region, the ring.
                if (got) m.set(enc >> 2, 0);
                for (int k = L.sub; k < nfac; k += G) {
                    const int w = S.fac[k].w;
                    if (w >= 0) m.set(w >> 2, 0);
                }
                for (int k = L.sub; k < nreg; k += G) m.set(S.reg[k], 0);
                const bool bad = trouble && !und && !ab;   // the seed
                if (L.sub == 0) atomicAdd(stats + (ab ? 0 : (und ? 5 : (bad ? 2 : 3))), 1ull);
                outcome = und || (bad && fuzzy) ? AI_DEFER : (ab || bad ? AI_RETRY : AI_LEAVE);
                growing = false;
            }
        }
        if (growing) {
            const int j = enc & 3;
            if (kind == 2) {
                const int k = __popc(mc & lt);
                S.reg[nreg + k] = enc >> 2;
                if (nreg == 0) {                      // the seed
                    S.front[1] = tn.x;
                    S.front[2] = tn.y;
                    S.front[3] = tn.z;
                    S.front[4] = tn.w;
                } else {
                    int* f = S.front + nfront + 3 * k;
                    f[0] = j == 0 ? tn.y : tn.x;
                    f[1] = j <= 1 ? tn.z : tn.y;
                    f[2] = j <= 2 ? tn.w : tn.z;
                }
            } else if (kind == 1) {
                // The facet's vertices, in the order that makes (a, b, c, v) positive:
                // the outside tet's other three in order, the first two swapped when
                // its own vertex there sits at an odd place.
                const int x = j == 0 ? tv.y : tv.x, y = j <= 1 ? tv.z : tv.y, z = j <= 2 ? tv.w : tv.z;
                S.fac[nfac + __popc(mf & lt)] =
                    make_int4((j & 1) ? y : x, (j & 1) ? x : y, z, got ? enc : enc | int(0x80000000));
            }
            const bool first = nreg == 0;
            head = min(head + G, nfront);
            nreg += nc;
            nfac += nf;
            nfront += first ? 4 : 3 * nc;
            growing = head < nfront;
        }
        __syncwarp();
    }

    // ---- re-star: new tet (a, b, c, v) on every boundary facet ----
    const bool win = live && outcome == AI_DONE;
    bool write = win;
    const int C = win ? nreg : 0, F = win ? nfac : 0;
    const int extra = max(F - C, 0);
    if (L.sub == 0 && ask) {
        if (block + kPool > m.cap()) report(status, ST_TET_CAPACITY);
        else S.pool.z = block, S.pool.w = kPool;
    }
    __syncwarp();
    // Slots: what the group holds, and for a very large star a block more.
    const int4 pool = S.pool;
    const int need = extra - pool.y - pool.w;
    int fresh = 0;
    if (need > 0) {
        if (L.sub == 0) {
            fresh = m.take(need);
            if (fresh + need > m.cap()) {
                if (!M::kLocal) report(status, ST_TET_CAPACITY);
                fresh = -1;
            }
        }
    }
    fresh = __shfl_sync(kFull, fresh, L.gbase);
    if (fresh < 0) {
        write = false;
        if (M::kLocal) outcome = AI_LEAVE;   // the table in device memory may have room
    }
    auto slot_of = [&](int k) {
        if (k < C) return S.reg[k];
        const int e = k - C;
        return e < pool.y ? pool.x + e : (e - pool.y < pool.w ? pool.z + (e - pool.y) : fresh + (e - pool.y - pool.w));
    };
    // Each edge of the boundary lies on exactly two facets.  The first to come
    // enters it in the hash table, the second finds it there: their new tets
    // are neighbours across the edge and v.
    if (win) {
        for (int k = L.sub; k < Scratch::kTable / 4; k += G)
            reinterpret_cast<int4*>(S.m.table)[k] = make_int4(0, 0, 0, 0);
        for (int k = L.sub; k < 3 * F; k += G) S.m.link[k] = 0xFFFFu;
    }
    __syncwarp();
    for (int k = L.sub; k < F; k += G) {
        const int4 f = S.fac[k];
        unsigned lo[3], hi[3], h[3], old[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {                 // the three edges' first probes together
            const int x = q == 0 ? f.y : f.x, y = q == 2 ? f.y : f.z;
            lo[q] = unsigned(min(x, y));
            hi[q] = unsigned(max(x, y));
            h[q] = (lo[q] * 0x9E3779B1u ^ hi[q] * 0x85EBCA77u) >> 16;
            old[q] = atomicCAS(&S.m.table[h[q] % Scratch::kTable], 0u, unsigned(3 * k + q) + 1);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const unsigned me = unsigned(3 * k + q);
            for (int probe = 0; old[q] != 0 && probe < Scratch::kTable; ++probe) {
                const int o = int(old[q]) - 1, ko = o / 3, mo = o - 3 * ko;
                const int4 g = S.fac[ko];
                const int xo = mo == 0 ? g.y : g.x, yo = mo == 2 ? g.y : g.z;
                if (unsigned(min(xo, yo)) == lo[q] && unsigned(max(xo, yo)) == hi[q]) {
                    S.m.link[me] = uint16_t(o);
                    S.m.link[o] = uint16_t(me);
                    break;
                }
                old[q] = atomicCAS(&S.m.table[++h[q] % Scratch::kTable], 0u, me + 1);
            }
        }
    }
    __syncwarp();
    if (write) {
        bool bad = false;
        for (int k = L.sub; k < F; k += G) {
            const int4 f = S.fac[k];
            const int enc = f.w & 0x7FFFFFFF, id = slot_of(k);
            int nn[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const int o = S.m.link[3 * k + q];
                if (o == 0xFFFF || S.m.link[o] != 3 * k + q) {
                    bad = true;
                    nn[q] = 0;
                    continue;
                }
                const int k2 = o / 3;
                nn[q] = slot_of(k2) * 4 + (o - 3 * k2);
            }
            m.store(id, make_int4(f.x, f.y, f.z, v), make_int4(nn[0], nn[1], nn[2], enc));
            m.link(enc, id * 4 + 3);
            if (f.x != kInf) m.vert(f.x, id);
            if (f.y != kInf) m.vert(f.y, id);
            if (f.z != kInf) m.vert(f.z, id);
            if (k == 0) m.vert(v, id);
        }
        for (int k = F + L.sub; k < C; k += G) m.kill(S.reg[k]);
        if (bad) report(status, ST_INTERNAL);
    }
    // ---- publish, then give the locks back ----
    // A lane gives back locks of tets that other lanes wrote, so its fence has to
    // stand behind the barrier: the barrier orders their writes before the fence,
    // and the fence with the plain store to the lock word behind it is the release
    // that the next owner's acquire meets.
    __syncwarp();
    m.fence();
    if (win) {
        for (int k = L.sub; k < F; k += G) {
            const int w = S.fac[k].w;
            if (w >= 0) m.set((w >> 2), 0);
        }
        const int n = write ? max(C, F) : C;
        for (int k = L.sub; k < n; k += G) m.set(slot_of(k), 0);
        if (write) {
            if (L.sub == 0) {
                const int a = min(extra, pool.y), b = min(extra - a, pool.w);
                const int2 rest = make_int2(pool.z + b, pool.w - b);
                S.pool = a < pool.y ? make_int4(pool.x + a, pool.y - a, rest.x, rest.y)
                                    : make_int4(rest.x, rest.y, 0, 0);
                ++S.won;
                S.nC += unsigned(C);
                S.nF += unsigned(F);
                ctr.region(C);
            }
        }
    }
    return outcome;
}

template <int G, int kMode, int kCapacity, int kThreads>
__global__ void __launch_bounds__(kThreads, kThreads != kGroupThreads ? 1 : (kMode == kExact ? kExactBlocks : kGroupBlocks))
    k_insert_groups(Tables T, GroupArgs A, Round R, const double* __restrict__ vx) {
    typedef GroupScratch<G, kCapacity> Scratch;
    const GlobalMesh m{T, A, vx};
    constexpr int kPerBlock = kThreads / G;
    extern __shared__ __align__(16) unsigned char group_smem[];
    Scratch* scratch = reinterpret_cast<Scratch*>(group_smem);
    D3G_SHARED_COUNTERS(ctr);
    const Lanes<G> L;
    Scratch& S = scratch[threadIdx.x / G];
    const int group = int(blockIdx.x) * kPerBlock + int(threadIdx.x) / G;
    __shared__ uint32_t lacking[kMode == kExact ? kThreads : 1];   // status words of the lanes' exact tests
    __shared__ int nitems;
    __shared__ long long stride;
    if (threadIdx.x == 0) {
        nitems = min(max(*A.n_items - A.first, 0), A.most);
        // Points go out in a scattered order (a stride near the golden ratio of their
        // number and coprime with it), so that those in flight lie far apart along the
        // curve.
        long long st = max(1LL, (long long)(double(nitems) * 0.6180339887));
        for (;; ++st) {
            long long a = st, b = nitems;
            while (b > 0) {
                const long long r = a % b;
                a = b;
                b = r;
            }
            if (a <= 1) break;
        }
        stride = st;
    }
    if (L.sub == 0) {
        S.nstash = 0;
        S.open = group < A.ngroups;
        S.won = S.tries = S.nC = S.nF = 0;
        S.pool = group < A.ngroups ? A.pool[group] : make_int4(0, 0, 0, 0);
    }
    unsigned tests = 0;
    __syncthreads();
    for (;;) {
        // ---- fetch: a new point, or one to try again ----
        int t = -1;
        if (L.sub == 0) {
            int item = -1;
            S.attempt = 0;
            while (item < 0 && S.nstash < kGroupStash && S.open) {
                const int q = atomicAdd(A.next, 1);
                if (q < nitems) item = A.items[A.first + int((q * stride) % nitems)];
                else S.open = 0;
            }
            if (item < 0 && S.nstash > 0) {
                item = S.stash[0];
                S.attempt = S.stash_tries[0];
                for (int k = 1; k < S.nstash; ++k) {
                    S.stash[k - 1] = S.stash[k];
                    S.stash_tries[k - 1] = S.stash_tries[k];
                }
                --S.nstash;
            }
            if (__ldcg(R.status) != 0) item = -1;
            S.item = item;
            if (item >= 0) {
                const int v = item, set = T.vset[v];
                t = __ldcg(A.hint + v);
                S.vlo = A.voff[set];
                S.vhi = A.voff[set + 1];
                if (t < 0) t = m.start(v, S.vlo);
                ++S.tries;
            }
        }
        __syncwarp();
        const bool live = S.item >= 0;
        if (!__any_sync(kFull, live)) break;
        const int v = live ? S.item : 0;
        const int ex = A.set_exact[T.vset[v]];
        t = max(__shfl_sync(kFull, t, L.gbase), 0);

        const int outcome = insert_step<G, kMode>(m, S, L, group, live, v, ex, t, A.cavity, R.status, A.stats, ctr, tests,
                                                  lacking + (kMode == kExact ? threadIdx.x : 0));
        const bool win = live && outcome == AI_DONE;
        // ---- what was not inserted: again later, or left ----
        bool idle = true;
        unsigned wait = 0;
        if (L.sub == 0 && live && !win) {
            const int attempt = S.attempt + 1;
            if (outcome == AI_RETRY && attempt < (kMode == kExact ? kExactTries : kGroupTries)) {
                S.stash[S.nstash] = v;
                S.stash_tries[S.nstash++] = attempt;
                if (t >= 0) A.hint[v] = t;
                idle = !S.open;
                wait = min(attempt, 3);
            } else {
                const bool def = outcome == AI_DEFER && kMode != kFilter, big = outcome == AI_LEAVE && G == 32;
                int* const list = def ? A.defer : (big ? A.big : A.left);
                list[atomicAdd(def ? A.n_defer : (big ? A.n_big : A.n_left), 1)] = v;
                atomicAdd(A.stats + 4, 1ull);
            }
        } else if (win) {
            idle = false;
        }
        // A warp that got nowhere and has no other points waits before it tries again,
        // longer each time and each warp another while, so that the groups in each
        // other's way drift apart.
        if (__all_sync(kFull, idle)) {
            wait = __reduce_max_sync(kFull, wait);
            __nanosleep(500u + (((unsigned(v) ^ unsigned(clock())) * 2654435761u) >> (21 - wait)));
        }
        __syncwarp();
    }
    if (L.sub == 0 && group < A.ngroups) {
        A.pool[group] = S.pool;
        atomicAdd(R.totals, (unsigned long long)S.won);
        atomicAdd(R.totals + 1, (unsigned long long)S.tries);
        atomicAdd(R.sums, (unsigned long long)S.nC);
        atomicAdd(R.sums + 1, (unsigned long long)S.nF);
    }
    ctr.tests[threadIdx.x] = tests;
    flush_counters(ctr, R);
}

// ---- the first levels of a set in one block's shared memory --------------------
//
// A set's first few hundred points keep few groups busy, and each of their
// insertions is a chain of some 30 trips to L2 of 400-800 cycles: half of the time
// of a 10^6-point build went into its first 2000 points.  k_coarse builds them
// where a trip takes 30-50 cycles: a block holds the coordinates, the tets (16-bit
// indices) and their locks of up to kCoarseCap vertices in shared memory, 16
// groups of 32 lanes insert into it (insert_step as everywhere), and the block
// then writes the finished mesh to the tables, where the later levels go on.

constexpr int kCoarseAlpha = 16;   // (12 and 24 were within 3 %)
constexpr int kCoarseThreads = 512;
constexpr int kCoarseVerts = kCoarseCap + 2;                 // and two of the first tet's from outside
constexpr int kCoarseTets = 8 * kCoarseVerts + 32;
typedef GroupScratch<32, 96> CoarseScratch;

struct CoarseShared {
    double xyz[3 * kCoarseVerts];
    unsigned long long tv[kCoarseTets], tn[kCoarseTets];     // four 16-bit indices each
    int lock[kCoarseTets];
    uint16_t vert_tet[kCoarseVerts], guide[kCoarseVerts];    // 0xFFFF: none
    CoarseScratch scratch[kCoarseThreads / 32];
    unsigned long long flags[kCoarseThreads];
    unsigned tests[kCoarseThreads];
    uint16_t max_region[kCoarseThreads];
    int count, next, set, base, extra[2], first[4];
    int stride;
};

static_assert(sizeof(CoarseShared) <= 227 * 1024, "k_coarse's scratch");

__device__ __forceinline__ unsigned long long pack16(const int4& q) {   // -1 becomes 0xFFFF
    return (unsigned long long)(unsigned(q.x) & 0xFFFFu) | (unsigned long long)(unsigned(q.y) & 0xFFFFu) << 16 |
           (unsigned long long)(unsigned(q.z) & 0xFFFFu) << 32 | (unsigned long long)(unsigned(q.w) & 0xFFFFu) << 48;
}
__device__ __forceinline__ int4 unpack16(unsigned long long u) {
    return make_int4(int(u & 0xFFFFu), int(u >> 16 & 0xFFFFu), int(u >> 32 & 0xFFFFu), int(u >> 48));
}
/// Vertices: 0xFFFF is the infinite one.
__device__ __forceinline__ int4 unpack_vertices(unsigned long long u) {
    int4 q = unpack16(u);
    q.x = q.x == 0xFFFF ? kInf : q.x;
    q.y = q.y == 0xFFFF ? kInf : q.y;
    q.z = q.z == 0xFFFF ? kInf : q.z;
    q.w = q.w == 0xFFFF ? kInf : q.w;
    return q;
}

/// The mesh in a block's shared memory: vertices and tets by their place there.
struct SharedMesh {
    CoarseShared& C;
    double grid;          // see in_sphere_near
    static constexpr int kPool = 0;
    static constexpr bool kLocal = true;
    __device__ __forceinline__ Pt point(int v) const { return Pt{C.xyz[3 * v], C.xyz[3 * v + 1], C.xyz[3 * v + 2]}; }
    __device__ __forceinline__ Pt again(int v) const {
        const volatile double* q = C.xyz + 3 * v;
        return Pt{q[0], q[1], q[2]};
    }
    __device__ __forceinline__ double inv(int) const { return grid; }
    __device__ __forceinline__ int4 tv4(int t) const {
        return unpack_vertices(*static_cast<volatile unsigned long long*>(C.tv + t));
    }
    __device__ __forceinline__ int4 tn4(int t) const {
        return unpack16(*static_cast<volatile unsigned long long*>(C.tn + t));
    }
    __device__ __forceinline__ void rec(int t, int4& tv, int4& tn) const {
        tv = tv4(t);
        tn = tn4(t);
    }
    __device__ __forceinline__ void store(int t, const int4& tv, const int4& tn) const {
        *static_cast<volatile unsigned long long*>(C.tv + t) = pack16(tv);
        *static_cast<volatile unsigned long long*>(C.tn + t) = pack16(tn);
    }
    __device__ __forceinline__ void link(int enc, int to) const {
        reinterpret_cast<volatile uint16_t*>(C.tn)[enc] = uint16_t(to);
    }
    __device__ __forceinline__ void kill(int t) const {
        const int4 q = tv4(t);
        const int x = max(q.x, q.y);
        *static_cast<volatile unsigned long long*>(C.tv + t) = pack16(make_int4(x, x, x, x));
    }
    __device__ __forceinline__ void vert(int v, int t) const {
        static_cast<volatile uint16_t*>(C.vert_tet)[v] = uint16_t(t);
    }
    __device__ __forceinline__ int cas(int t, int value) const {
        const int old = atomicCAS(C.lock + t, 0, value);
        __threadfence_block();
        return old;
    }
    __device__ __forceinline__ void set(int t, int value) const { *static_cast<volatile int*>(C.lock + t) = value; }
    __device__ __forceinline__ int take(int n) const { return atomicAdd(&C.count, n); }
    __device__ __forceinline__ int cap() const { return kCoarseTets; }
    __device__ __forceinline__ int walk_limit() const { return kAsyncWalkLimit; }
    __device__ __forceinline__ int start(int, int) const {
        return static_cast<volatile uint16_t*>(C.vert_tet)[C.first[0]];
    }
    /// A tet of the nearest vertex among those in already next to v along the curve:
    /// 16 of its own level, 16 about its guide.  All 32 lanes.
    __device__ __forceinline__ int near_start(int v, int n, int lane) const {
        const int g = C.guide[v];
        const int u = lane < 16 ? v - 8 + lane : g - 24 + lane;
        int t = 0xFFFF;
        float d = 3e38f;
        if (u >= 0 && u < n && (lane < 16 || g != 0xFFFF)) {
            t = static_cast<volatile uint16_t*>(C.vert_tet)[u];
            const Pt a = point(v), b = point(u);
            const float x = float(b.x - a.x), y = float(b.y - a.y), z = float(b.z - a.z);
            if (t != 0xFFFF) d = fminf(x * x + y * y + z * z, 3e38f);   // (a NaN gives 3e38)
        }
        // Distances are not negative: their bits order as they do.
        const unsigned best = __reduce_min_sync(kFull, (__float_as_uint(d) & ~31u) | unsigned(lane));
        t = __shfl_sync(kFull, t, int(best & 31u));
        return t != 0xFFFF ? t : start(0, 0);
    }
    __device__ __forceinline__ void fence() const { __threadfence_block(); }
};

/// What k_coarse reads besides GroupArgs: where each set's levels start, how many
/// of them are its, and the queue of sets.
struct CoarseArgs {
    const int* starts;
    int stride;
    const int* levels;
    int nsets;
    int* next;
};

template <int kMode>
__global__ void __launch_bounds__(kCoarseThreads, 1)
    k_coarse(Tables T, GroupArgs A, CoarseArgs K, Round R, const double* __restrict__ vx) {
    extern __shared__ __align__(16) unsigned char coarse_smem[];
    CoarseShared& C = *reinterpret_cast<CoarseShared*>(coarse_smem);
    const Lanes<32> L;
    const int group = int(threadIdx.x >> 5);
    CoarseScratch& S = C.scratch[group];
    const SharedCounters ctr{C.tests, C.flags, C.max_region};
    ctr.clear();
    unsigned tests = 0;
    if (L.sub == 0) S.won = S.tries = S.nC = S.nF = 0;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            int set;
            do set = atomicAdd(K.next, 1);
            while (set < K.nsets && K.levels[set] == 0);
            C.set = __ldcg(R.status) != 0 ? K.nsets : set;
        }
        __syncthreads();
        const int set = C.set;
        if (set >= K.nsets) break;
        const int4 sk = A.skips[set];
        const int* ls = K.starts + int64_t(set) * K.stride;
        const int nlev = K.levels[set];
        const int v0 = ls[0], n0 = ls[nlev] - v0;
        const SharedMesh m{C, kMode != kFilter ? A.inv_grid[set] : 0.0};
        // ---- vertices, the first tet and its four caps, from the tables ----
        if (threadIdx.x == 0) {
            C.count = 5;
            C.extra[0] = C.extra[1] = -1;
            int ne = 0;
            const int f[4] = {sk.x, sk.y, sk.z, sk.w};
            for (int k = 0; k < 4; ++k) {
                C.first[k] = f[k] - v0;
                if (f[k] - v0 >= n0 && k >= 2) {
                    C.extra[ne] = f[k];
                    C.first[k] = n0 + ne++;
                }
            }
        }
        __syncthreads();
        auto local_of = [&](int v) {
            return v == kInf ? kInf : (v == sk.x ? C.first[0] : (v == sk.y ? C.first[1] : (v == sk.z ? C.first[2] : C.first[3])));
        };
        auto global_of = [&](int v) { return v == kInf ? kInf : (v < n0 ? v0 + v : C.extra[v - n0]); };
        for (int v = int(threadIdx.x); v < n0 + 2; v += kCoarseThreads) {
            const int g = v < n0 ? v0 + v : C.extra[v - n0];
            if (g < 0) continue;
            const Pt p = vpt(vx, g);
            C.xyz[3 * v] = p.x;
            C.xyz[3 * v + 1] = p.y;
            C.xyz[3 * v + 2] = p.z;
            C.vert_tet[v] = 0xFFFFu;
            const int gd = v < n0 ? A.guide[g] - v0 : -1;
            C.guide[v] = gd >= 0 && gd < n0 ? uint16_t(gd) : uint16_t(0xFFFFu);
        }
        for (int t = int(threadIdx.x); t < kCoarseTets; t += kCoarseThreads) {
            C.tv[t] = C.tn[t] = 0;
            C.lock[t] = -1;
        }
        __syncthreads();
        if (threadIdx.x < 5) {
            const int t = int(threadIdx.x), gt = 5 * set + t;
            const int4 tv = T.tv(gt), tn = T.tn(gt);
            C.tv[t] = pack16(make_int4(local_of(tv.x), local_of(tv.y), local_of(tv.z), local_of(tv.w)));
            C.tn[t] = pack16(make_int4(tn.x - 20 * set, tn.y - 20 * set, tn.z - 20 * set, tn.w - 20 * set));
            C.lock[t] = 0;
            if (t < 4) C.vert_tet[C.first[t]] = 0;
        }
        const int ex = A.set_exact[set];
        // ---- level by level ----
        for (int lev = 0; lev < nlev; ++lev) {
            const int lb = ls[lev] - v0, cnt = ls[lev + 1] - ls[lev];
            __syncthreads();
            if (threadIdx.x == 0) {
                C.next = 0;
                int st = max(1, int(float(cnt) * 0.618034f));
                for (;; ++st) {
                    int a = st, b = cnt;
                    while (b > 0) {
                        const int r = a % b;
                        a = b;
                        b = r;
                    }
                    if (a <= 1) break;
                }
                C.stride = st;
            }
            // About one group per kCoarseAlpha points in the mesh.
            if (L.sub == 0) {
                S.nstash = 0;
                S.open = cnt > 0 && group * kCoarseAlpha <= lb;
                S.pool = make_int4(0, 0, 0, 0);
                S.vlo = 0;
                S.vhi = n0 + 2;
            }
            __syncthreads();
            for (;;) {
                if (L.sub == 0) {
                    int item = -1;
                    S.attempt = 0;
                    while (item < 0 && S.nstash < kGroupStash && S.open) {
                        const int q = atomicAdd(&C.next, 1);
                        if (q < cnt) {
                            item = lb + (q * C.stride) % cnt;
                            if (item == C.first[0] || item == C.first[1] || item == C.first[2] || item == C.first[3])
                                item = -1;
                        } else {
                            S.open = 0;
                        }
                    }
                    if (item < 0 && S.nstash > 0) {
                        item = S.stash[0];
                        S.attempt = S.stash_tries[0];
                        for (int k = 1; k < S.nstash; ++k) {
                            S.stash[k - 1] = S.stash[k];
                            S.stash_tries[k - 1] = S.stash_tries[k];
                        }
                        --S.nstash;
                    }
                    S.item = item;
                    if (item >= 0) ++S.tries;
                }
                __syncwarp();
                const int v = S.item;
                if (v < 0) break;
                int t = m.near_start(v, n0, L.lane);
                const int outcome = insert_step<32, kMode>(m, S, L, group, true, v, ex, t, 96, R.status, A.stats, ctr, tests);
                bool again = false;
                if (outcome != AI_DONE) {
                    again = outcome == AI_RETRY && S.attempt + 1 < kGroupTries;
                    __syncwarp();
                    if (L.sub == 0) {
                        if (again) {
                            S.stash[S.nstash] = v;
                            S.stash_tries[S.nstash++] = S.attempt + 1;
                        } else {
                            A.left[atomicAdd(A.n_left, 1)] = global_of(v);
                            atomicAdd(A.stats + 4, 1ull);
                        }
                    }
                    __syncwarp();
                    if (again && !S.open) __nanosleep(200u + ((unsigned(clock()) * 2654435761u) >> 20));
                }
            }
        }
        __syncthreads();
        // ---- the mesh goes to the tables ----
        const int total = min(C.count, kCoarseTets);   // (more were asked for if it was full)
        if (threadIdx.x == 0) {
            C.base = total > 5 ? atomicAdd(T.tet_count, total - 5) : 0;
            if (C.base + total - 5 > T.cap) {
                report(R.status, ST_TET_CAPACITY);
                C.base = -1;
            }
        }
        __syncthreads();
        if (C.base >= 0) {
            const int base = C.base;
            auto tet_of = [&](int t) { return t < 5 ? 5 * set + t : base + t - 5; };
            auto enc_of = [&](int e) { return tet_of(e >> 2) * 4 + (e & 3); };
            for (int t = int(threadIdx.x); t < total; t += kCoarseThreads) {
                const int4 tv = unpack_vertices(C.tv[t]), tn = unpack16(C.tn[t]);
                const int g = tet_of(t);
                T.tv(g) = make_int4(global_of(tv.x), global_of(tv.y), global_of(tv.z), global_of(tv.w));
                T.tn(g) = make_int4(enc_of(tn.x), enc_of(tn.y), enc_of(tn.z), enc_of(tn.w));
                T.lock[g] = 0;
            }
            for (int v = int(threadIdx.x); v < n0 + 2; v += kCoarseThreads) {
                const int g = v < n0 ? v0 + v : C.extra[v - n0];
                if (g >= 0 && C.vert_tet[v] != 0xFFFFu) T.vert_tet[g] = tet_of(C.vert_tet[v]);
            }
        }
    }
    if (L.sub == 0) {
        atomicAdd(R.totals, (unsigned long long)S.won);
        atomicAdd(R.totals + 1, (unsigned long long)S.tries);
        atomicAdd(R.sums, (unsigned long long)S.nC);
        atomicAdd(R.sums + 1, (unsigned long long)S.nF);
    }
    ctr.tests[threadIdx.x] = tests;
    flush_counters(ctr, R);
}
