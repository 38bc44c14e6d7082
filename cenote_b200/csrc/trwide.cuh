// Eight lanes to a ray: the walks of a queue too short to fill the device.
//
// The bounces that end a wave hold few rays, and their walk takes as long as
// its longest ray: about a microsecond a node when one lane tests a node's
// eight children and its triangles in turn. Here a group of eight lanes walks
// one ray, a lane to each child slot and to each candidate triangle, so a node
// costs its latency and a few dozen instructions. Per ray that is more work
// for the device, which has nothing else to do then; the kernels choose by
// the queue's length (CN_WIDE_RAYS). Walks of a one-sample 640x360 chart
// frame: intersect 0.52 -> 0.45 ms, shadow 0.37 -> 0.31 ms; of a two-sample
// 853x479 terrain frame 1.79 -> 1.57 and 1.24 -> 1.00 ms.
//
// Hits are bitwise those of the other walks: the planes, slacks and triangle
// test are the same arithmetic, and the committed hit is the lexicographic
// minimum of (t, instance, primitive) over the candidates. Only scenes whose
// triangles are all opaque use it.
#pragma once
#include "trqueue.cuh"

namespace cn {

// One group's stack entries; the four groups' stacks of a warp take the place
// of its triangle queue.
constexpr uint32_t WIDE_STACK = TRAVERSAL_STACK;
static_assert(4u * WIDE_STACK * sizeof(uint2) <= sizeof(TriQueueSmem), "the stacks fit the triangle queue's memory");

// What a group's lanes keep of its ray (the same in all eight, but for the
// lane's own plane offsets into a node).
struct WideRay {
    Ray r;
    uint32_t near_at[3], far_at[3];  // byte offsets of this lane's near and far planes per axis
};

__device__ __forceinline__ WideRay wide_ray(const Ray& r, uint32_t slot) {
    WideRay w;
    w.r = r;
    const bool neg[3] = {r.idir.x < 0.0f, r.idir.y < 0.0f, r.idir.z < 0.0f};
#pragma unroll
    for (uint32_t a = 0; a < 3u; ++a) {
        w.near_at[a] = (neg[a] ? 56u : 32u) + 8u * a + slot;
        w.far_at[a] = (neg[a] ? 32u : 56u) + 8u * a + slot;
    }
    return w;
}

__device__ __forceinline__ float biased_load(const uint8_t* p) { return PLANE_BIAS + float(__ldg(p)); }

// Test the eight children of node `ni`, one per lane of the group: the hit
// mask as intersect_node gives it, in every lane of the group. All 32 lanes
// call it together.
__device__ __forceinline__ uint32_t wide_node(const DeviceScene& s, uint32_t ni, const WideRay& w, float tmax,
                                              uint32_t slot, uint32_t& base_child, uint32_t& base_tri,
                                              uint32_t& imask) {
    const uint8_t* node = reinterpret_cast<const uint8_t*>(s.nodes + ni);
    const uint4 n0 = __ldg(reinterpret_cast<const uint4*>(node));
    const uint2 n1 = __ldg(reinterpret_cast<const uint2*>(node + 16));
    uint32_t meta = __ldg(node + 24 + slot);
    const float nx = biased_load(node + w.near_at[0]), fx = biased_load(node + w.far_at[0]);
    const float ny = biased_load(node + w.near_at[1]), fy = biased_load(node + w.far_at[1]);
    const float nz = biased_load(node + w.near_at[2]), fz = biased_load(node + w.far_at[2]);
    const Ray& r = w.r;
    const float sx = __uint_as_float((n0.w & 0xffu) << 23), sy = __uint_as_float(((n0.w >> 8) & 0xffu) << 23),
                sz = __uint_as_float(((n0.w >> 16) & 0xffu) << 23);
    imask = n0.w >> 24;
    base_child = n1.x;
    base_tri = n1.y;
    const PlanePair px = node_axis(sx * r.idir.x, (__uint_as_float(n0.x) - r.org.x) * r.idir.x);
    const PlanePair py = node_axis(sy * r.idir.y, (__uint_as_float(n0.y) - r.org.y) * r.idir.y);
    const PlanePair pz = node_axis(sz * r.idir.z, (__uint_as_float(n0.z) - r.org.z) * r.idir.z);
    float tnx, tny, tnz, tfx, tfy, tfz;
    plane_t(nx, fx, px, tnx, tfx);
    plane_t(ny, fy, py, tny, tfy);
    plane_t(nz, fz, pz, tnz, tfz);
    const float t0 = fmaxf(max3f(tnx, tny, tnz), 0.0f);
    const float t1 = fminf(min3f(tfx, tfy, tfz), tmax * 1.000021f);
    if ((meta & 0x18u) == 0x18u) meta ^= r.oct_inv;  // an inner child: its slot XOR the octant
    uint32_t mask = t0 <= t1 ? (meta >> 5) << (meta & 0x1fu) : 0u;
    mask |= __shfl_xor_sync(TQ_FULL, mask, 4);
    mask |= __shfl_xor_sync(TQ_FULL, mask, 2);
    mask |= __shfl_xor_sync(TQ_FULL, mask, 1);
    return mask;
}

// A group's walk: the node group being expanded, the triangles of the last
// node's hit leaves, the stack height.
struct WideWalk {
    uint2 g, t;
    uint32_t sp, iter;
    bool on;
};

__device__ __forceinline__ void wide_begin(WideWalk& w, const Ray& r, bool on) {
    w.g = make_uint2(0u, (1u << (24u + r.oct_inv)) | 1u);
    w.t = make_uint2(0u, 0u);
    w.sp = 0u;
    w.iter = 0u;
    w.on = on;
}

// Expand one node in every walking group (false in a group whose bounds ran
// out). All 32 lanes call it together.
template <bool COUNT>
__device__ __forceinline__ bool wide_expand(const DeviceScene& s, const WideRay& r, float tmax, WideWalk& w,
                                            uint2* stack, uint32_t slot, uint32_t* visits) {
    bool ok = true;
    uint32_t ni = 0u;
    if (w.on) {
        const uint32_t pos = 31u - __clz(w.g.y & 0xff000000u);
        w.g.y &= ~(1u << pos);
        ni = w.g.x + __popc(w.g.y & 0xffu & ((1u << ((pos - 24u) ^ r.r.oct_inv)) - 1u));
        ok = ++w.iter <= walk_bound(s);
        if (w.g.y & 0xff000000u) {
            if (w.sp >= WIDE_STACK) ok = false;
            else if (slot == 0u) stack[w.sp] = w.g;
            ++w.sp;
        }
        if (COUNT && slot == 0u) ++*visits;
    }
    uint32_t bc, bt, im;
    const uint32_t hits = wide_node(s, ni, r, tmax, slot, bc, bt, im);  // an idle group looks at node 0
    w.g = make_uint2(bc, (hits & 0xff000000u) | im);
    w.t = make_uint2(bt, w.on ? hits & 0x00ffffffu : 0u);
    __syncwarp();
    return ok;
}

// After the node's triangles: the next group off the stack, or the end.
__device__ __forceinline__ void wide_next(WideWalk& w, const uint2* stack) {
    if (w.on && !(w.g.y & 0xff000000u)) {
        if (w.sp == 0u) w.on = false;
        else w.g = stack[--w.sp];
    }
    __syncwarp();
}

// m without its k lowest set bits.
__device__ __forceinline__ uint32_t drop_low(uint32_t m, uint32_t k) {
    for (; k > 0u && m != 0u; --k) m &= m - 1u;
    return m;
}

// The k-th (from 0) pending triangle of the group.
__device__ __forceinline__ uint32_t wide_tri(const WideWalk& w, uint32_t k) {
    return w.t.x + __ffs(drop_low(w.t.y, k)) - 1u;
}

// Closest hits of items `begin .. end - 1` (at most four groups' worth at a
// time): `src` as queued_closest takes it, without its queue.
template <bool COUNT, class Src>
__device__ __forceinline__ void wide_closest(const DeviceScene& s, TriQueueSmem& sm, Src& src, uint32_t begin,
                                             uint32_t end, uint32_t ray_mask, bool& overflow, uint32_t* visits,
                                             uint32_t* tests) {
    const uint32_t lane = threadIdx.x & 31u, slot = lane & 7u, group = lane >> 3;
    uint2* stack = reinterpret_cast<uint2*>(&sm) + group * WIDE_STACK;
    for (uint32_t base = begin; base < end; base += 4u) {
        const uint32_t item = base + group;
        const bool mine = item < end;
        float3 o = f3(0.0f), d = f3(1.0f);
        if (mine) src.ray(item, o, d);
        const WideRay ray = wide_ray(make_ray(o, d), slot);
        WideWalk w;
        wide_begin(w, ray.r, mine && s.node_count != 0u);
        float tmax = 1e30f;
        uint4 best = make_uint4(LIGHT_NONE, 0u, 0u, 0u);
        while (__any_sync(TQ_FULL, w.on)) {
            if (!wide_expand<COUNT>(s, ray, tmax, w, stack, slot, visits)) {
                overflow = true;
                w.on = false;
                w.t.y = 0u;
            }
            while (__any_sync(TQ_FULL, w.t.y != 0u)) {
                float t = 0.0f, b1 = 0.0f, b2 = 0.0f;
                uint32_t inst = 0u, prim = 0u, key = 0xffffffffu;
                if (slot < uint32_t(__popc(w.t.y))) {
                    const uint32_t tri = wide_tri(w, slot);
                    const float4* tp = s.tris + 3u * min(tri, s.tri_count - 1u);
                    const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                    if (COUNT) ++*tests;
                    if ((__float_as_uint(c.w) & ray_mask) && tri_hit(ray.r, a, b, c, tmax, t, b1, b2)) {
                        inst = __float_as_uint(a.w);
                        prim = __float_as_uint(b.w);
                        key = t == 0.0f ? 0u : __float_as_uint(t);
                    }
                }
                w.t.y = drop_low(w.t.y, 8u);
                if (!__any_sync(TQ_FULL, key != 0xffffffffu)) continue;
                // The group's lexicographic minimum of (t, instance, primitive).
#pragma unroll
                for (uint32_t x = 4u; x > 0u; x >>= 1) {
                    const uint32_t k2 = __shfl_xor_sync(TQ_FULL, key, x), i2 = __shfl_xor_sync(TQ_FULL, inst, x),
                                   p2 = __shfl_xor_sync(TQ_FULL, prim, x);
                    const float t2 = __shfl_xor_sync(TQ_FULL, t, x), u2 = __shfl_xor_sync(TQ_FULL, b1, x),
                                v2 = __shfl_xor_sync(TQ_FULL, b2, x);
                    if (k2 < key || (k2 == key && (i2 < inst || (i2 == inst && p2 < prim)))) {
                        key = k2;
                        inst = i2;
                        prim = p2;
                        t = t2;
                        b1 = u2;
                        b2 = v2;
                    }
                }
                if (key != 0xffffffffu &&
                    (t < tmax || (t == tmax && (inst < best.x || (inst == best.x && prim < best.y))))) {
                    tmax = t;
                    best = make_uint4(inst, prim, __float_as_uint(b1), __float_as_uint(b2));
                }
            }
            wide_next(w, stack);
        }
        if (mine && slot == 0u) src.emit(item, best, tmax);
        src.step(mine && slot == 0u, item, best.x, tmax);
    }
}

// Shadow queries of items `begin .. end - 1`, as queued_any answers them.
template <bool COUNT, class Src>
__device__ __forceinline__ void wide_any(const DeviceScene& s, TriQueueSmem& sm, Src& src, uint32_t begin,
                                         uint32_t end, bool& overflow, uint32_t* visits, uint32_t* tests) {
    const uint32_t lane = threadIdx.x & 31u, slot = lane & 7u, group = lane >> 3;
    uint2* stack = reinterpret_cast<uint2*>(&sm) + group * WIDE_STACK;
    for (uint32_t base = begin; base < end; base += 4u) {
        const uint32_t item = base + group;
        const bool mine = item < end;
        Ray r = make_ray(f3(0.0f), f3(1.0f));
        AnyQuery q{0.0f, 0xffffffffu, LIGHT_NONE, 0u};
        if (mine) src.begin(item, r, q);
        const WideRay ray = wide_ray(r, slot);
        WideWalk w;
        wide_begin(w, ray.r, mine && s.node_count != 0u);
        bool occluded = false;
        while (__any_sync(TQ_FULL, w.on)) {
            if (!wide_expand<COUNT>(s, ray, q.tm, w, stack, slot, visits)) {
                overflow = true;
                occluded = true;  // dropped, as the other walks drop it
                w.on = false;
                w.t.y = 0u;
            }
            while (__any_sync(TQ_FULL, w.t.y != 0u)) {
                bool hit = false;
                if (slot < uint32_t(__popc(w.t.y))) {
                    const uint32_t tri = min(wide_tri(w, slot), s.tri_count - 1u);
                    if (tri != q.leaf) {
                        const float4* tp = s.tris + 3u * tri;
                        const float4 v0 = __ldg(tp), v1 = __ldg(tp + 1), v2 = __ldg(tp + 2);
                        if (COUNT) ++*tests;
                        float t, b1, b2;
                        if (tri_hit(ray.r, v0, v1, v2, q.tm, t, b1, b2)) {
                            const uint32_t inst = __float_as_uint(v0.w), prim = __float_as_uint(v1.w);
                            hit = !(q.leaf != 0xffffffffu && t == q.tm &&
                                    !(inst < q.light || (inst == q.light && prim < q.lprim)));
                        }
                    }
                }
                w.t.y = drop_low(w.t.y, 8u);
                if ((__ballot_sync(TQ_FULL, hit) >> (8u * group)) & 0xffu) {
                    occluded = true;
                    w.on = false;
                    w.t.y = 0u;
                }
            }
            wide_next(w, stack);
        }
        if (mine && slot == 0u) src.emit(item, !occluded);
    }
}

}  // namespace cn
