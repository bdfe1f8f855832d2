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
// L2 once.

constexpr int kGroupThreads = 128;
/// Blocks per SM the insertion kernel is compiled for: 20 warps at 96 registers
/// (92 used, no spills) and 38 KB of scratch a block.  With 6 (80 registers, 80
/// bytes of spills, 228 KB of the SM's 256 taken by scratch, so spills miss L1)
/// 4096 mixed sets took 440 ms against 409, with 4 457 against 429.
constexpr int kGroupBlocks = 5;
constexpr int kGroupStash = 6;        // points a group keeps to try again later
constexpr int kGroupTries = 24;       // attempts before a point is left
constexpr int kWaitPolls = 150;       // polls of a lock before its holder's point is given way to
constexpr int kPoolSlots = 16;        // tet slots a group takes from the table at a time

template <int G>
struct alignas(16) GroupScratch {
    static constexpr int kCap = 8 * G;              // region tets; boundary facets
    static constexpr int kFront = 3 * kCap + 4;     // facets met: three per region tet, four at the seed
    static constexpr int kTable = 16 * G;           // edges: at most 3/2 per facet
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
    int* hint;               // per vertex: a tet near it (k_locate), -1: none
    int* next;               // queue head
    int* left;               // points to try again by wider groups or with kNear (regions too big, too many
                             // conflicts, undecided tests) ...
    int* n_left;
    int* defer;              // ... and points for the full variant (a test the filters cannot decide)
    int* n_defer;
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

/// Locates a level's points, one thread each, in the mesh as it is before the
/// level: the walk of an insertion, which has a group's lanes wait for one chain
/// of reads, then starts a step or two from its end.  Reads may use L1, since
/// nothing writes the mesh meanwhile.  A facet the filter cannot decide is not
/// crossed and a long walk ends where it is: the tet is only where the insertion
/// starts.
__global__ void __launch_bounds__(128) k_locate(Tables T, GroupArgs A, const double* __restrict__ vx) {
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
            const Pt a = vpt(vx, tv.x), b = vpt(vx, tv.y), c = vpt(vx, tv.z), d = vpt(vx, tv.w);
            h = h * 1664525u + 1013904223u;
            int next = -1;
#pragma unroll 1
            for (int m = 0; m < 4 && next < 0; ++m) {
                const int i = int((h >> 30) + unsigned(m)) & 3;
                const int nb = at(tn, i) >> 2;
                if (nb == prev) continue;
                const int o = orient_replaced_filter(a, b, c, d, i, p, ex);
                if (o < 0) next = nb;
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

template <int G, bool kNear>
__global__ void __launch_bounds__(kGroupThreads, kGroupBlocks)
    k_insert_groups(Tables T, GroupArgs A, Round R, const double* __restrict__ vx) {
    typedef GroupScratch<G> Scratch;
    constexpr int kPerBlock = kGroupThreads / G;
    __shared__ Scratch scratch[kPerBlock];
    D3G_SHARED_COUNTERS(ctr);
    const Lanes<G> L;
    Scratch& S = scratch[threadIdx.x / G];
    const int group = int(blockIdx.x) * kPerBlock + int(threadIdx.x) / G;
    const unsigned lt = (1u << L.lane) - 1u;
    const int region = (group + 1) << 1, ring = region | 1;
    __shared__ int nitems;
    __shared__ long long stride;
    if (threadIdx.x == 0) {
        nitems = *A.n_items;
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
                if (q < nitems) item = A.items[int((q * stride) % nitems)];
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
                if (t < 0) t = tet_near(T, A.guide[v], S.vlo, A.skips[set].x);
                ++S.tries;
            }
        }
        __syncwarp();
        const bool live = S.item >= 0;
        if (!__any_sync(kFull, live)) break;
        const int v = live ? S.item : 0;
        const Pt p = vpt(vx, v);
        const int ex = A.set_exact[T.vset[v]];
        t = max(__shfl_sync(kFull, t, L.gbase), 0);

        // Slots for its new tets, asked for here so that the answer is there by the re-star.
        const bool ask = live && S.pool.w == 0 && S.pool.y < kPoolSlots;
        int block = 0;
        if (L.sub == 0 && ask) block = atomicAdd(T.tet_count, kPoolSlots);

        // ---- walk (see walk_async; lanes 0-3 test the facets, lanes 4-7 fetch the
        //      neighbours' records) ----
        // A facet the filter cannot decide is not crossed: the seed is tested in any
        // case, and if it fails the test the point is left to the full variant.
        int outcome = live ? AI_DONE : -1;
        bool fuzzy = false;
        {
            int4 tv, tn;
            ld_rec(T, t, tv, tn);
            if (live && tv.x == tv.y) {                   // the hint's tet has gone since
                t = tet_near(T, A.guide[v], S.vlo, A.skips[T.vset[v]].x);
                ld_rec(T, t, tv, tn);
            }
            t = __shfl_sync(kFull, t, L.gbase);
            const int ip = inf_pos(tv);
            if (live && ip >= 0) {
                t = at(tn, ip) >> 2;
                ld_rec(T, t, tv, tn);
            }
            int prev = -1, step = 0;
            uint32_t h = uint32_t(v) * 2654435761u + 12345u;
            const int limit = min(kAsyncWalkLimit, T.walk_limit);
            bool walking = live;
            while (__any_sync(kFull, walking)) {
                int4 pv = make_int4(0, 0, 0, 0), pn = pv;
                if (walking && L.sub >= 4 && L.sub < 8) ld_rec(T, at(tn, L.sub & 3) >> 2, pv, pn);
                h = h * 1664525u + 1013904223u;
                const int s0 = int(h >> 30);
                bool neg = false, undecided = false;
                if (walking && L.sub < 4 && (at(tn, L.sub) >> 2) != prev && tv.x != kInf && tv.y != kInf &&
                    tv.z != kInf && tv.w != kInf) {
                    const int o = orient_replaced_filter(vpt(vx, tv.x), vpt(vx, tv.y), vpt(vx, tv.z), vpt(vx, tv.w),
                                                         L.sub, p, ex & EX_ORIENT);
                    undecided = o == 2;
                    neg = o < 0;
                }
                const unsigned und = L.own(__ballot_sync(kFull, undecided));
                const unsigned m = L.own(__ballot_sync(kFull, neg)) & 0xFu;
                const unsigned rot = ((m >> s0) | (m << (4 - s0))) & 0xFu;
                const int i = (s0 + __ffs(int(rot)) - 1) & 3;
                const int src = L.gbase + 4 + i;
                const int4 nv = make_int4(__shfl_sync(kFull, pv.x, src), __shfl_sync(kFull, pv.y, src),
                                          __shfl_sync(kFull, pv.z, src), __shfl_sync(kFull, pv.w, src));
                const int4 nn = make_int4(__shfl_sync(kFull, pn.x, src), __shfl_sync(kFull, pn.y, src),
                                          __shfl_sync(kFull, pn.z, src), __shfl_sync(kFull, pn.w, src));
                if (!walking) continue;
                fuzzy = fuzzy || und;
                if (m == 0) {
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
                        t = -1;
                        if (L.sub == 0) atomicAdd(A.stats + 1, 1ull);
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
        while (__any_sync(kFull, growing)) {
            const bool valid = growing && head + L.sub < nfront;
            int enc = 0, kind = 0;      // 1: boundary facet, 2: new region tet, 3: decided below
            bool got = false, abort = false, undecided = false, bad_seed = false;
            int4 tv = make_int4(0, 0, 0, 0), tn = tv;
            if (valid) {
                enc = S.front[head + L.sub];
                const int nb = enc >> 2;
                // The record is read along with the lock attempt, so that its vertices are
                // known one trip to L2 earlier; the copy read under the lock decides.
                int4 guess, ignore;
                ld_rec(T, nb, guess, ignore);
                int seen = cas_lock(A.lock + nb, ring);
                if (G == 32) {
                    // Of two insertions in each other's way one must go on: a group waits for
                    // one with a higher number, which gives way itself when it meets this one's
                    // locks (so no two wait for each other), and gives way to one with a lower
                    // number.  Not for narrower groups, where the other may be in the same warp.
                    for (int k = 0; k < kWaitPolls && seen > ring; ++k) {
                        __nanosleep(200);
                        seen = cas_lock(A.lock + nb, ring);
                    }
                }
                got = seen == 0;
                if (seen == ring) kind = 3;               // locked by this group: in this step, or before
                else if (!got && seen != region) abort = true;   // another group holds it
                if (got || kind == 3) ld_rec(T, nb, tv, tn);
                if (got) {
                    int r = 0;
                    for (;;) {
                        r = in_conflict_fast<kNear>(T, nb, guess, p, v, vx, ex, A.inv_grid);
                        if (guess.x == tv.x && guess.y == tv.y && guess.z == tv.z && guess.w == tv.w) break;
                        guess = tv;
                    }
                    if (nreg == 0) {
                        // The seed may come from a half-written record: only a live
                        // tet of the point's own set will do (see insert_full).
                        const int u = tv.x != kInf ? tv.x : tv.y;
                        bad_seed = tv.x == tv.y || u < S.vlo || u >= S.vhi;
                        if (bad_seed) r = 0;
                    }
                    ++tests;
                    if (r & (CT_UNCERTAIN | CT_TIE)) ctr.count(r);
                    undecided = (r & CT_UNDECIDED) != 0;
                    kind = (r & CT_IN) ? 2 : 1;
                    if (kind == 2) set_lock(A.lock + nb, region);
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
            const unsigned ab = L.own(__ballot_sync(kFull, abort));
            const unsigned und = L.own(__ballot_sync(kFull, undecided));
            const unsigned bad = L.own(__ballot_sync(kFull, bad_seed && !undecided));
            const unsigned mf = __ballot_sync(kFull, kind == 1) & L.gm;
            const int nc = __popc(mc), nf = __popc(mf);
            const bool full = nreg + nc > Scratch::kCap || nfac + nf > Scratch::kCap ||
                              nreg + nc > A.cavity || nfac + nf > 2 * A.cavity;
            if (growing && (ab || und || bad || full)) {
                // Give everything back: this step's locks, the region, the ring.
                if (got) set_lock(A.lock + (enc >> 2), 0);
                for (int k = L.sub; k < nfac; k += G) {
                    const int w = S.fac[k].w;
                    if (w >= 0) set_lock(A.lock + (w >> 2), 0);
                }
                for (int k = L.sub; k < nreg; k += G) set_lock(A.lock + S.reg[k], 0);
                if (L.sub == 0) atomicAdd(A.stats + (ab ? 0 : (und ? 6 : (bad ? 2 : 3))), 1ull);
                outcome = und || (bad && fuzzy) ? AI_DEFER : (ab || bad ? AI_RETRY : AI_LEAVE);
                growing = false;
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
            if (block + kPoolSlots > T.cap) report(R.status, ST_TET_CAPACITY);
            else S.pool.z = block, S.pool.w = kPoolSlots;
        }
        __syncwarp();
        // Slots: what the group holds, and for a very large star a block more.
        const int4 pool = S.pool;
        const int need = extra - pool.y - pool.w;
        int fresh = 0;
        if (need > 0) {
            if (L.sub == 0) {
                fresh = atomicAdd(T.tet_count, need);
                if (fresh + need > T.cap) {
                    report(R.status, ST_TET_CAPACITY);
                    fresh = -1;
                }
            }
        }
        fresh = __shfl_sync(kFull, fresh, L.gbase);
        if (fresh < 0) write = false;
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
            for (int m = 0; m < 3; ++m) {                 // the three edges' first probes together
                const int x = m == 0 ? f.y : f.x, y = m == 2 ? f.y : f.z;
                lo[m] = unsigned(min(x, y));
                hi[m] = unsigned(max(x, y));
                h[m] = (lo[m] * 0x9E3779B1u ^ hi[m] * 0x85EBCA77u) >> 16;
                old[m] = atomicCAS(&S.m.table[h[m] % Scratch::kTable], 0u, unsigned(3 * k + m) + 1);
            }
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const unsigned me = unsigned(3 * k + m);
                for (int probe = 0; old[m] != 0 && probe < Scratch::kTable; ++probe) {
                    const int o = int(old[m]) - 1, ko = o / 3, mo = o - 3 * ko;
                    const int4 g = S.fac[ko];
                    const int xo = mo == 0 ? g.y : g.x, yo = mo == 2 ? g.y : g.z;
                    if (unsigned(min(xo, yo)) == lo[m] && unsigned(max(xo, yo)) == hi[m]) {
                        S.m.link[me] = uint16_t(o);
                        S.m.link[o] = uint16_t(me);
                        break;
                    }
                    old[m] = atomicCAS(&S.m.table[++h[m] % Scratch::kTable], 0u, me + 1);
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
                for (int m = 0; m < 3; ++m) {
                    const int o = S.m.link[3 * k + m];
                    if (o == 0xFFFF || S.m.link[o] != 3 * k + m) {
                        bad = true;
                        nn[m] = 0;
                        continue;
                    }
                    const int k2 = o / 3;
                    nn[m] = slot_of(k2) * 4 + (o - 3 * k2);
                }
                st_rec(T, id, make_int4(f.x, f.y, f.z, v), make_int4(nn[0], nn[1], nn[2], enc));
                T.link(enc) = id * 4 + 3;
                if (f.x != kInf) T.vert_tet[f.x] = id;
                if (f.y != kInf) T.vert_tet[f.y] = id;
                if (f.z != kInf) T.vert_tet[f.z] = id;
                if (k == 0) T.vert_tet[v] = id;
            }
            for (int k = F + L.sub; k < C; k += G) T.kill(S.reg[k]);
            if (bad) report(R.status, ST_INTERNAL);
        }
        // ---- publish, then give the locks back ----
        __threadfence();
        __syncwarp();
        if (win) {
            for (int k = L.sub; k < F; k += G) {
                const int w = S.fac[k].w;
                if (w >= 0) set_lock(A.lock + (w >> 2), 0);
            }
            const int n = write ? max(C, F) : C;
            for (int k = L.sub; k < n; k += G) set_lock(A.lock + slot_of(k), 0);
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
        // ---- what was not inserted: again later, or left ----
        bool idle = true;
        unsigned wait = 0;
        if (L.sub == 0 && live && !win) {
            const int attempt = S.attempt + 1;
            if (outcome == AI_RETRY && attempt < kGroupTries) {
                S.stash[S.nstash] = v;
                S.stash_tries[S.nstash++] = attempt;
                if (t >= 0) A.hint[v] = t;
                idle = !S.open;
                wait = min(attempt, 3);
            } else {
                // Too big for the widest group, or undecided even so: the full variant.
                const bool def = (outcome == AI_DEFER && kNear) || (outcome == AI_LEAVE && G == 32);
                (def ? A.defer : A.left)[atomicAdd(def ? A.n_defer : A.n_left, 1)] = v;
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
