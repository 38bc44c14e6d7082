// Warp triangle queue: the closest-hit walk with its triangle tests shared
// by the whole warp.
//
// In the per-lane walk (traverse.cuh, walk_step) every lane tests its own hit
// leaves' triangles one at a time right after the node that found them, so a
// warp spends as many iterations as its busiest lane has triangles while the
// other lanes idle (measured at the bench's wave sizes: 23 % of lanes active
// in the triangle loop on the material chart, 14 % on the terrain). Here a
// lane appends each triangle group (first triangle, 24 pending bits) to a
// per-warp FIFO in shared memory and keeps walking; once the FIFO holds a
// warp's worth of triangles (or no lane has nodes left), a round hands one
// (ray, triangle) pair to every lane: a warp scan of the entries' bit counts
// maps lane j to its entry and bit, the owner's ray comes over shuffles and
// shared memory, and each owner's candidates reduce to the lexicographic
// minimum of (t, instance, primitive) through a shared-memory atomic minimum
// (any-hit queries: an OR of occluders). A lane whose walk has ended waits for its queued
// triangles before it takes a new ray.
//
// Results are bitwise those of the per-lane walk: the watertight test of a
// (ray, triangle) pair is the same arithmetic wherever it runs, and both
// commit the lexicographic minimum of (t, instance, primitive) over the
// candidates with t within the ray's bound (the walk's node culling keeps a
// slack above the current hit, so a later commit never drops a winner; a ray
// walking here culls with a bound at least as large as the per-lane walk's,
// which only adds candidates that lose). Only scenes whose triangles are all
// opaque use it: fractional opacity draws its Bernoulli decisions in visit
// order.
#pragma once
#include "shadow.cuh"
#include "traverse.cuh"

namespace cn {

constexpr uint32_t TQ_CAP = 64;  // FIFO entries per warp (a power of two, at least 2 x 32)
constexpr uint32_t TQ_FULL = 0xffffffffu;
// A closest-hit round also runs, partly filled, once this many lanes have
// ended their walks and only wait for queued triangles, so they take new rays
// sooner (chart intersect -4 %; 4 and 16 measured slower; the shadow walk
// measured no gain from it).
constexpr uint32_t TQ_WAITING = 8;

// One warp's queue in shared memory (1,920 bytes: a full SM of traversal
// blocks keeps 60 KB, and the L1 cache, which holds the walks' stacks and the
// nodes and triangles they revisit, most of its capacity). What a lane's ray
// needs only in the triangle rounds lives here instead of in registers: ten
// registers a lane, without which the node test spilled.
struct TriQueueSmem {
    uint2 entry[TQ_CAP];     // (first triangle, owner lane << 24 | untested triangle bits)
    // Per owner lane, a round's running minimum of the candidates' t key and
    // the winning lane; ~0 between rounds. `key2` serves exact ties.
    uint32_t key[32], key2[32], winner[32];
    // Per lane: the watertight test's shear constants (sx, sy, sz) and its
    // axes kx | ky << 2 | kz << 4.
    float4 shear[32];
    // Per lane: the closest hit so far (instance, primitive, b1, b2), or a
    // shadow query's target (leaf, instance, primitive, unused).
    uint4 best[32];
};
static_assert(sizeof(TriQueueSmem) == 1920, "1,920 bytes a warp");

// What a walking lane keeps of its ray: the node test's inputs.
struct WalkRay {
    float3 org, idir;
    uint32_t oct_inv;
};

// Split a lane's ray between its registers and the warp's shared memory.
__device__ __forceinline__ WalkRay tq_ray(TriQueueSmem& sm, const Ray& r) {
    sm.shear[threadIdx.x & 31u] =
        make_float4(r.sx, r.sy, r.sz, __uint_as_float(uint32_t(r.kx) | (uint32_t(r.ky) << 2) | (uint32_t(r.kz) << 4)));
    return {r.org, r.idir, r.oct_inv};
}

// The warp's queue positions; every lane holds the same values. Entries
// head .. tail-1 are pending; `tris` counts their untested bits.
struct TriQueue {
    uint32_t head, tail, tris;
};

// Position of the (k+1)-th lowest set bit of m (m has more than k set bits):
// the largest x with popc(m below x) <= k, by binary search.
__device__ __forceinline__ uint32_t nth_set_bit(uint32_t m, uint32_t k) {
    uint32_t p = 0;
#pragma unroll
    for (uint32_t w = 16; w > 0; w >>= 1)
        if (uint32_t(__popc(m & ((1u << (p + w)) - 1u))) <= k) p += w;
    return p;
}

// Append each lane's triangle group (low 24 bits of grp.y; none when zero).
// All 32 lanes call it together; the caller keeps at most TQ_CAP - 32
// entries pending before the call.
__device__ __forceinline__ void tq_append(TriQueueSmem& sm, TriQueue& q, uint2 grp, uint32_t& last_seq) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t bits = grp.y & 0x00ffffffu;
    const uint32_t ball = __ballot_sync(TQ_FULL, bits != 0u);
    if (bits) {
        const uint32_t seq = q.tail + __popc(ball & ((1u << lane) - 1u));
        sm.entry[seq & (TQ_CAP - 1u)] = make_uint2(grp.x, (lane << 24) | bits);
        last_seq = seq + 1u;
    }
    q.tail += __popc(ball);
    q.tris += __reduce_add_sync(TQ_FULL, __popc(bits));
    __syncwarp();
}

// A round's work for one lane: triangle `tri` of the ray owned by lane
// `owner`, when `act`.
struct TqWork {
    uint32_t tri, owner;
    bool act;
};

// Take the next min(32, pending) triangles of the FIFO, one per lane: a warp
// scan of the entries' bit counts maps lane j to its entry and bit; the entry
// crossing the last slot keeps the bits this round does not reach. Advances
// the queue; all 32 lanes call it together with q.tris > 0.
__device__ __forceinline__ TqWork tq_take(TriQueueSmem& sm, TriQueue& q) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t idx = q.head + lane;
    const bool has = idx < q.tail;
    const uint2 e = has ? sm.entry[idx & (TQ_CAP - 1u)] : make_uint2(0u, 0u);
    const uint32_t bits = e.y & 0x00ffffffu;
    const uint32_t cnt = __popc(bits);
    uint32_t incl = cnt;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(TQ_FULL, incl, o);
        if (lane >= o) incl += v;
    }
    const uint32_t excl = incl - cnt;
    const uint32_t n = min(__shfl_sync(TQ_FULL, incl, 31), 32u);
    // The entry serving slot `lane`: the last one whose prefix is <= lane.
    uint32_t k = 0;
#pragma unroll
    for (uint32_t st = 16; st > 0; st >>= 1)
        if (__shfl_sync(TQ_FULL, excl, k + st) <= lane) k += st;
    const uint32_t kbits = __shfl_sync(TQ_FULL, bits, k);
    const uint32_t kbase = __shfl_sync(TQ_FULL, e.x, k);
    const uint32_t kexcl = __shfl_sync(TQ_FULL, excl, k);
    TqWork wk;
    wk.owner = __shfl_sync(TQ_FULL, e.y >> 24, k);
    wk.act = lane < n;
    wk.tri = wk.act ? kbase + nth_set_bit(kbits, lane - kexcl) : 0u;
    if (has && excl < n && incl > n) {
        const uint32_t cut = nth_set_bit(bits, n - excl - 1u);
        sm.entry[idx & (TQ_CAP - 1u)].y = (e.y & 0xff000000u) | (bits & ~((2u << cut) - 1u));
    }
    q.head += __popc(__ballot_sync(TQ_FULL, has && incl <= n));
    q.tris -= n;
    return wk;
}

// The owner's ray as the watertight test reads it: its origin over shuffles,
// the rest from shared memory.
__device__ __forceinline__ Ray owner_ray(const TriQueueSmem& sm, const WalkRay& ray, uint32_t owner) {
    Ray ro;
    ro.org = f3(__shfl_sync(TQ_FULL, ray.org.x, owner), __shfl_sync(TQ_FULL, ray.org.y, owner),
                __shfl_sync(TQ_FULL, ray.org.z, owner));
    const float4 sh = sm.shear[owner];
    ro.sx = sh.x;
    ro.sy = sh.y;
    ro.sz = sh.z;
    const uint32_t kp = __float_as_uint(sh.w);
    ro.kx = int(kp & 3u);
    ro.ky = int((kp >> 2) & 3u);
    ro.kz = int((kp >> 4) & 3u);
    return ro;
}

// One closest-hit round: each lane's triangle tested against its owner's
// ray; every owner commits the best of its candidates. All 32 lanes call it
// together with q.tris > 0.
template <bool COUNT = false>
__device__ __forceinline__ void tq_round(const DeviceScene& s, TriQueueSmem& sm, TriQueue& q, const WalkRay& ray,
                                         float& tmax, uint32_t ray_mask, uint32_t* tests) {
    const uint32_t lane = threadIdx.x & 31u;
    const TqWork wk = tq_take(sm, q);
    const uint32_t owner = wk.owner;
    const Ray ro = owner_ray(sm, ray, owner);
    const float tmo = __shfl_sync(TQ_FULL, tmax, owner);
    bool cand = false;
    float t = 0.0f, b1 = 0.0f, b2 = 0.0f;
    uint32_t inst = 0u, prim = 0u;
    if (wk.act && wk.tri < s.tri_count) {
        const float4* tp = s.tris + 3u * wk.tri;
        const float4 a = __ldg(tp), b = __ldg(tp + 1), cc = __ldg(tp + 2);
        if (COUNT) ++*tests;
        if ((__float_as_uint(cc.w) & ray_mask) && tri_hit(ro, a, b, cc, tmo, t, b1, b2)) {
            cand = true;
            inst = __float_as_uint(a.w);
            prim = __float_as_uint(b.w);
        }
    }
    if (!__any_sync(TQ_FULL, cand)) {
        __syncwarp();
        return;
    }
    // Per owner, the lexicographic minimum of (t, instance, primitive); both
    // zeros of t order as one, as they compare equal in the per-lane walk.
    // The nearest t is a shared-memory minimum per owner (the slots start at
    // ~0 and are reset by their owners after the round; grouping the lanes by
    // owner with a warp match instead measured 30 % slower), and a lane alone
    // at it wins. Only when two lanes of one owner meet at the same t do the
    // identities decide.
    const uint32_t tkey = cand ? (t == 0.0f ? 0u : __float_as_uint(t)) : 0xffffffffu;
    if (cand) atomicMin(&sm.key[owner], tkey);
    __syncwarp();
    const bool c2 = cand && sm.key[owner] == tkey;
    if (c2) atomicMin(&sm.winner[owner], lane);
    __syncwarp();
    bool win = c2 && sm.winner[owner] == lane;
    if (__any_sync(TQ_FULL, c2 && !win)) {
        if (c2) sm.winner[owner] = sm.key2[owner] = 0xffffffffu;
        __syncwarp();
        if (c2) atomicMin(&sm.key2[owner], inst);
        __syncwarp();
        const bool c3 = c2 && sm.key2[owner] == inst;
        if (c3) atomicMin(&sm.winner[owner], prim);
        __syncwarp();
        win = c3 && sm.winner[owner] == prim;
        __syncwarp();
        if (win) sm.winner[owner] = lane;
    }
    // The winner commits to its owner's slot unless the hit there has the
    // same t and the smaller identity; the owner takes the new bound.
    if (win) {
        bool better = t < tmo;
        if (!better) {
            const uint4 cur = sm.best[owner];
            better = inst < cur.x || (inst == cur.x && prim < cur.y);
        }
        if (better) sm.best[owner] = make_uint4(inst, prim, __float_as_uint(b1), __float_as_uint(b2));
    }
    __syncwarp();
    const uint32_t from = sm.winner[lane];
    const bool mine = from != 0xffffffffu;
    const float wt = __shfl_sync(TQ_FULL, t, mine ? from : lane);
    if (mine) {
        if (wt < tmax) tmax = wt;
        sm.key[lane] = 0xffffffffu;
        sm.winner[lane] = 0xffffffffu;
    }
    __syncwarp();
}

// The queued closest-hit walk of a persistent warp. `src` supplies and
// retires the rays (all members are called by the whole warp unless noted):
//   uint32_t next(bool live, bool& drained)  an item for each idle lane (~0u: none)
//   void ray(uint32_t item, float3& org, float3& dir)      (per lane)
//   void emit(uint32_t item, uint4 hit, float t)          (per lane)
//   void step(bool finished, uint32_t item, uint32_t instance, float t)  before every refill
//   uint32_t want_idle(bool drained)  idle lanes before the warp refills
// Each step a walking lane expands one node and queues the triangles of the
// leaves it hits; rounds run while the FIFO holds a warp's worth of
// triangles, while TQ_WAITING lanes wait on it, or until it is empty once no
// lane has nodes left. A lane whose walk has ended completes when its last
// queued entry has been tested; the finished lanes are retired together
// before the warp refills, so the stores and the sort's key counts run once
// per refill and not at every step that ends a ray.
// Sets `overflow` when a walk hit its iteration or stack bound.
template <bool COUNT, class Src, int S = TRAVERSAL_STACK>
__device__ __forceinline__ void queued_closest(const DeviceScene& s, TriQueueSmem& sm, Src& src, uint32_t ray_mask,
                                               bool& overflow, uint32_t* visits, uint32_t* tests) {
    const uint32_t lane = threadIdx.x & 31u;
    TriQueue q{0u, 0u, 0u};
    uint2 stack[S];
    Walk w;
    WalkRay ray{f3(0.0f), f3(0.0f), 0u};
    float tmax = 1e30f;
    uint32_t item = 0u, last_seq = 0u;
    bool live = false, walking = false, drained = false, finished = false;
    sm.key[lane] = 0xffffffffu;
    sm.winner[lane] = 0xffffffffu;
    __syncwarp();
    for (;;) {
        uint32_t inst = 0u;
        if (finished) {
            const uint4 hit = sm.best[lane];
            inst = hit.x;
            src.emit(item, hit, tmax);
        }
        src.step(finished, item, inst, tmax);
        finished = false;
        if (!drained) {
            const uint32_t i = src.next(live, drained);
            if (i != ~0u) {
                float3 o, d;
                src.ray(i, o, d);
                const Ray r = make_ray(o, d);
                ray = tq_ray(sm, r);
                sm.best[lane] = make_uint4(LIGHT_NONE, 0u, 0u, 0u);
                tmax = 1e30f;
                walk_begin(w, r);
                item = i;
                last_seq = 0u;
                live = true;
                walking = s.node_count != 0;
            }
        }
        if (!__any_sync(TQ_FULL, live)) {
            if (drained) break;
            continue;
        }
        const uint32_t want_idle = src.want_idle(drained);
        for (;;) {
            uint2 grp = make_uint2(0u, 0u);
            if (live && walking) {
                if (++w.iter > walk_bound(s) || !expand_node<COUNT, S>(s, ray, tmax, w, stack, visits)) {
                    overflow = true;
                    walking = false;
                } else {
                    grp = w.t;
                    if (!(w.g.y & 0xff000000u)) {
                        if (w.sp == 0) walking = false;
                        else w.g = stack[--w.sp];
                    }
                }
            }
            tq_append(sm, q, grp, last_seq);
            const bool any_walking = __any_sync(TQ_FULL, live && walking);
            const bool many_waiting = uint32_t(__popc(__ballot_sync(TQ_FULL, live && !walking))) >= TQ_WAITING;
            while (q.tris >= 32u || (q.tris > 0u && (!any_walking || many_waiting)))
                tq_round<COUNT>(s, sm, q, ray, tmax, ray_mask, tests);
            if (live && !walking && q.head >= last_seq) {
                finished = true;
                live = false;
            }
            if (uint32_t(__popc(__ballot_sync(TQ_FULL, !live))) >= want_idle) break;
        }
    }
}

// ---- shadow queries (trace_shadow.slang:29-72) ------------------------------------

// A shadow query as its source sets it up: its bound (the target triangle's
// distance, or tmax without one), the target's leaf (~0 when the target was
// not hit or there is none) and (instance, primitive) identity. The walk
// keeps the bound in a register and the target in shared memory.
struct AnyQuery {
    float tm;
    uint32_t leaf, light, lprim;
};

// One any-hit round: each lane's triangle tested against its owner's query;
// an opaque hit nearer than the owner's target (equal distance: the smaller
// (instance, primitive) key) occludes it, as in shadow_step. All 32 lanes
// call it together with q.tris > 0.
template <bool COUNT = false>
__device__ __forceinline__ void tq_round_any(const DeviceScene& s, TriQueueSmem& sm, TriQueue& q, const WalkRay& ray,
                                             float tm, bool& occluded, uint32_t* tests) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t dead = __ballot_sync(TQ_FULL, occluded);
    const TqWork wk = tq_take(sm, q);
    const uint32_t owner = wk.owner;
    const Ray ro = owner_ray(sm, ray, owner);
    const float tmo = __shfl_sync(TQ_FULL, tm, owner);
    bool occl = false;
    if (wk.act && !((dead >> owner) & 1u) && wk.tri < s.tri_count) {
        const uint4 target = sm.best[owner];  // leaf, instance, primitive
        if (wk.tri != target.x) {
            const float4* tp = s.tris + 3u * wk.tri;
            const float4 v0 = __ldg(tp), v1 = __ldg(tp + 1), v2 = __ldg(tp + 2);
            if (COUNT) ++*tests;
            float t, b1, b2;
            if (tri_hit(ro, v0, v1, v2, tmo, t, b1, b2)) {
                const uint32_t inst = __float_as_uint(v0.w), prim = __float_as_uint(v1.w);
                occl = !(target.x != 0xffffffffu && t == tmo &&
                         !(inst < target.y || (inst == target.y && prim < target.z)));
            }
        }
    }
    if ((__reduce_or_sync(TQ_FULL, occl ? (1u << owner) : 0u) >> lane) & 1u) occluded = true;
    __syncwarp();
}

// The queued shadow walk of a persistent warp over scenes whose triangles
// are all opaque. `src` supplies and retires the queries (the whole warp
// calls each member unless noted):
//   uint32_t next(bool live, bool& drained)  an item for each idle lane (~0u: none)
//   bool begin(uint32_t item, Ray& ray, AnyQuery& a)   (per lane) false: the
//       query has no target leaf to bound it; then `closest(item)` answers it
//       with the per-lane closest-hit walk (only where FALLBACK is set)
//   template <int S> void closest(uint32_t item, uint2* stack)  (per lane; the
//       stack holds S entries)
//   void emit(uint32_t item, bool visible)              (per lane; a query
//       whose walk hit a bound counts as occluded)
//   uint32_t want_idle(bool drained)
// An occluded query stops walking at once; its entries still queued are
// skipped, and it completes when they have left the queue. Finished queries
// are retired together before the warp refills.
template <bool COUNT, class Src, int S = TRAVERSAL_STACK>
__device__ __forceinline__ void queued_any(const DeviceScene& s, TriQueueSmem& sm, Src& src, bool& overflow,
                                           uint32_t* visits, uint32_t* tests) {
    const uint32_t lane = threadIdx.x & 31u;
    TriQueue q{0u, 0u, 0u};
    uint2 stack[S];
    Walk w;
    WalkRay ray{f3(0.0f), f3(0.0f), 0u};
    float tm = 0.0f;
    uint32_t item = 0u, last_seq = 0u;
    bool live = false, walking = false, drained = false, occluded = false, finished = false;
    for (;;) {
        if (finished) src.emit(item, !occluded);
        finished = false;
        if (!drained) {
            const uint32_t i = src.next(live, drained);
            if (i != ~0u) {
                item = i;
                last_seq = 0u;
                live = true;
                occluded = false;
                Ray r;
                AnyQuery a;
                walking = src.begin(i, r, a) && s.node_count != 0;
                if constexpr (Src::FALLBACK) {
                    if (!walking && s.node_count != 0) {
                        src.template closest<S>(i, stack);  // no target leaf: the per-lane closest-hit query
                        live = false;
                    }
                }
                ray = tq_ray(sm, r);
                tm = a.tm;
                sm.best[lane] = make_uint4(a.leaf, a.light, a.lprim, 0u);
                walk_begin(w, r);
            }
        }
        if (!__any_sync(TQ_FULL, live)) {
            if (drained) break;
            continue;
        }
        const uint32_t want_idle = src.want_idle(drained);
        for (;;) {
            uint2 grp = make_uint2(0u, 0u);
            if (live && walking && !occluded) {
                if (++w.iter > walk_bound(s) || !expand_node<COUNT, S>(s, ray, tm, w, stack, visits)) {
                    overflow = true;
                    occluded = true;  // dropped, as the per-lane walk drops it
                    walking = false;
                } else {
                    grp = w.t;
                    if (!(w.g.y & 0xff000000u)) {
                        if (w.sp == 0) walking = false;
                        else w.g = stack[--w.sp];
                    }
                }
            }
            tq_append(sm, q, grp, last_seq);
            const bool any_walking = __any_sync(TQ_FULL, live && walking && !occluded);
            while (q.tris >= 32u || (q.tris > 0u && !any_walking))
                tq_round_any<COUNT>(s, sm, q, ray, tm, occluded, tests);
            if (live && (!walking || occluded) && q.head >= last_seq) {
                finished = true;
                live = false;
            }
            if (uint32_t(__popc(__ballot_sync(TQ_FULL, !live))) >= want_idle) break;
        }
    }
}

}  // namespace cn
