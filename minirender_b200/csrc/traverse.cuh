// traverse.cuh — FP32 ray queries over the BVH: slab test, watertight triangle test, nearest and
// any-hit traversal.
//
// Semantics follow the reference exactly (src/render/intersection.cpp, src/render/bvh.cpp:206-300):
// closed intervals, ties to the lower primitive id, single-sided culling by geometric winding,
// any-hit exit on the first accepted triangle, pruning of popped subtrees whose entry distance
// exceeds the current nearest hit. Differences are numeric only:
//  - slab distances are widened by 2^-20 relative instead of one double ulp, so the box test
//    stays conservative in FP32 (FP32 rounding of (b - o) * inv is at most a few ulps);
//  - the triangle test is the same permute/shear/difference-of-products algorithm in FP32 with
//    the error bound of the reference evaluated with FP32's unit roundoff.
#pragma once

#include "device_scene.cuh"

namespace mr {

// A wide node pushes <= 3 entries and sits at most 63 levels deep (built trees stop at 48,
// bvh.cpp:16; imported trees are refused beyond 64 levels), so at most 3 * 63 entries are
// stacked before any push: the check `sp > kStackSize - 3` never fires on an accepted tree.
constexpr int      kStackSize  = 195;
constexpr uint32_t kMaxVisits  = 1u << 16;  // node visits and leaves per ray before the query gives up

// The part of a ray that the triangle test uses: origin, permutation and shear.
struct TriangleRay {
    f3    o;
    int   kx, ky, kz;
    float sx, sy, sz;
};

struct RayQuery {
    f3    o, d;
    float inv_lo[3];  // 1/d scaled down by 2^-20: near slab distances round toward the origin
    float inv_hi[3];  // 1/d scaled up by 2^-20: far slab distances round away
    bool  neg[3];     // direction sign per axis (the near slab is the max bound)
    int   kx, ky, kz;
    float sx, sy, sz;

    __device__ __forceinline__ TriangleRay triangle_ray() const { return {o, kx, ky, kz, sx, sy, sz}; }
    __device__ __forceinline__ void init(f3 origin, f3 direction) {
        o = origin;
        d = direction;
        const float lo = 0.99999904632568359375f;  // 1 - 2^-20
        const float hi = 1.00000095367431640625f;  // 1 + 2^-20
        for (int a = 0; a < 3; ++a) {
            const float c = comp(d, a);
            const float inv = 1.0f / c;  // +-inf for +-0: the slab then imposes no bound
            inv_lo[a] = inv * lo;
            inv_hi[a] = inv * hi;
            neg[a]    = signbit(c);
        }
        // Permutation and shear (src/render/intersection.cpp:62-74).
        const f3 ad = fabs3(d);
        kz          = ad.x > ad.y ? 0 : 1;
        if (ad.z > comp(ad, kz)) {
            kz = 2;
        }
        kx = kz == 2 ? 0 : kz + 1;
        ky = kx == 2 ? 0 : kx + 1;
        if (comp(d, kz) < 0) {
            const int t = kx;
            kx          = ky;
            ky          = t;
        }
        const float dz = comp(d, kz);
        sx             = comp(d, kx) / dz;
        sy             = comp(d, ky) / dz;
        sz             = 1.0f / dz;
    }
};

// Entry distance of one child box, or NaN when the slab intervals do not overlap within
// [tmin, tmax] (NaN compares false against every interval end, +inf would not for tmax = inf). `xy` = (lo.x, hi.x, lo.y, hi.y); (zlo, zhi) the z extent.
__device__ __forceinline__ float slab_enter(const RayQuery& q, float4 xy, float zlo, float zhi,
                                            float tmin, float tmax) {
    const float nx = ((q.neg[0] ? xy.y : xy.x) - q.o.x) * q.inv_lo[0];
    const float fx = ((q.neg[0] ? xy.x : xy.y) - q.o.x) * q.inv_hi[0];
    const float ny = ((q.neg[1] ? xy.w : xy.z) - q.o.y) * q.inv_lo[1];
    const float fy = ((q.neg[1] ? xy.z : xy.w) - q.o.y) * q.inv_hi[1];
    const float nz = ((q.neg[2] ? zhi : zlo) - q.o.z) * q.inv_lo[2];
    const float fz = ((q.neg[2] ? zlo : zhi) - q.o.z) * q.inv_hi[2];
    // fmaxf/fminf ignore the NaN of 0 * inf (origin on the slab plane of a zero component).
    const float enter = fmaxf(fmaxf(tmin, nx), fmaxf(ny, nz));
    const float leave = fminf(fminf(tmax, fx), fminf(fy, fz));
    return enter <= leave ? enter : __int_as_float(0x7fffffff);
}

// A 32-byte load (one sector of a wide node): half the load instructions, and half the L1
// wavefronts of divergent lanes, that two 16-byte loads would take.
__device__ __forceinline__ void load_sector(const float4* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// Slab planes of a wide node's four children, two children per packed FP32 operation: the
// distances ((p - o) * inv) of four planes, each operation rounded as its scalar form is.
__device__ __forceinline__ float4 plane_distances(float4 p, float neg_o, float inv) {
    const float2 o2 = make_float2(neg_o, neg_o), i2 = make_float2(inv, inv);
    const float2 a  = __fmul2_rn(__fadd2_rn(make_float2(p.x, p.y), o2), i2);
    const float2 b  = __fmul2_rn(__fadd2_rn(make_float2(p.z, p.w), o2), i2);
    return make_float4(a.x, a.y, b.x, b.y);
}

// Entry distance of a child box from the distances of its near and far planes, or +inf when the
// ray misses it. A hit's entry is at most `tmax` (leave <= tmax), and +inf is also what an
// unbounded entry means, so interior traversal treats +inf as "no child" without a second
// comparison against the interval. fmaxf/fminf ignore the NaN of 0 * inf (origin on the slab plane
// of a zero direction component).
__device__ __forceinline__ float box_entry(float nx, float ny, float nz, float fx, float fy, float fz,
                                           float tmin, float tmax) {
    const float enter = fmaxf(fmaxf(tmin, nx), fmaxf(ny, nz));
    const float leave = fminf(fminf(tmax, fx), fminf(fy, fz));
    return enter <= leave ? enter : __int_as_float(0x7f800000);
}

// Offsets (in float4) of the sectors a ray reads of a wide node (layout in device_scene.cuh).
struct SectorOffsets {
    int near_xy, near_z;
    __device__ __forceinline__ void init(const bool* neg) {
        near_xy = (neg[0] ? 2 : 0) + (neg[1] ? 4 : 0);
        near_z  = neg[2] ? 10 : 8;
    }
    __device__ __forceinline__ int far_xy() const { return 6 - near_xy; }
    __device__ __forceinline__ int far_z() const { return 18 - near_z; }
};

__device__ __forceinline__ void order2(float& ta, int& ra, float& tb, int& rb) {
    if (tb < ta) {
        const float t = ta;
        ta            = tb;
        tb            = t;
        const int r   = ra;
        ra            = rb;
        rb            = r;
    }
}

// A wide node against a ray: the children's refs and their entries, +inf where the ray misses the
// child within [tmin, tmax] or there is none.
struct NodeVisit {
    int   r0, r1, r2, r3;
    float t0, t1, t2, t3;
    __device__ __forceinline__ void visit(const float4* n, SectorOffsets at, f3 neg_near, f3 neg_far,
                                          const float* inv_lo, const float* inv_hi, float tmin, float tmax) {
        float4 nx, ny, nz, fx, fy, rf;
        load_sector(n + at.near_xy, nx, ny);
        load_sector(n + at.near_z, nz, rf);
        load_sector(n + at.far_xy(), fx, fy);
        float4 fz = __ldg(n + at.far_z());
        nx = plane_distances(nx, neg_near.x, inv_lo[0]);
        ny = plane_distances(ny, neg_near.y, inv_lo[1]);
        nz = plane_distances(nz, neg_near.z, inv_lo[2]);
        fx = plane_distances(fx, neg_far.x, inv_hi[0]);
        fy = plane_distances(fy, neg_far.y, inv_hi[1]);
        fz = plane_distances(fz, neg_far.z, inv_hi[2]);
        r0 = __float_as_int(rf.x), r1 = __float_as_int(rf.y), r2 = __float_as_int(rf.z), r3 = __float_as_int(rf.w);
        t0 = box_entry(nx.x, ny.x, nz.x, fx.x, fy.x, fz.x, tmin, tmax);
        t1 = box_entry(nx.y, ny.y, nz.y, fx.y, fy.y, fz.y, tmin, tmax);
        t2 = box_entry(nx.z, ny.z, nz.z, fx.z, fy.z, fz.z, tmin, tmax);
        t3 = box_entry(nx.w, ny.w, nz.w, fx.w, fy.w, fz.w, tmin, tmax);
    }
    __device__ __forceinline__ uint32_t children() const { return 2 + (r2 != 0 ? 1 : 0) + (r3 != 0 ? 1 : 0); }
    // Nearest child first.
    __device__ __forceinline__ void sort() {
        order2(t0, r0, t1, r1);
        order2(t2, r2, t3, r3);
        order2(t0, r0, t2, r2);
        order2(t1, r1, t3, r3);
        order2(t1, r1, t2, r2);
    }
};

__device__ __forceinline__ float permuted(f3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

// Sheared vertices (x, y; z before the scale) and the three unnormalised edge functions of the
// watertight triangle test.
__device__ __forceinline__ void triangle_edges(const TriangleRay& q, f3 v0, f3 v1, f3 v2, float* x, float* y,
                                               float* z, float& a, float& b, float& c) {
    const f3 t0 = v0 - q.o, t1 = v1 - q.o, t2 = v2 - q.o;
    z[0] = permuted(t0, q.kz), z[1] = permuted(t1, q.kz), z[2] = permuted(t2, q.kz);
    x[0] = fmaf(-q.sx, z[0], permuted(t0, q.kx));
    y[0] = fmaf(-q.sy, z[0], permuted(t0, q.ky));
    x[1] = fmaf(-q.sx, z[1], permuted(t1, q.kx));
    y[1] = fmaf(-q.sy, z[1], permuted(t1, q.ky));
    x[2] = fmaf(-q.sx, z[2], permuted(t2, q.kx));
    y[2] = fmaf(-q.sy, z[2], permuted(t2, q.ky));
    a = difference_of_products(x[1], y[2], y[1], x[2]);
    b = difference_of_products(x[2], y[0], y[2], x[0]);
    c = difference_of_products(x[0], y[1], y[0], x[1]);
}

// Watertight triangle test (src/render/intersection.cpp:108-152) in FP32. On acceptance returns
// the distance and the three unnormalised edge functions plus their sum (the determinant).
__device__ __forceinline__ bool triangle_test(const TriangleRay& q, f3 v0, f3 v1, f3 v2, float tmin,
                                              float tmax, float& t, float& ea, float& eb,
                                              float& ec, float& det) {
    float px[3], py[3], pz[3], a, b, c;
    triangle_edges(q, v0, v1, v2, px, py, pz, a, b, c);
    if ((a < 0 || b < 0 || c < 0) && (a > 0 || b > 0 || c > 0)) {
        return false;
    }
    const float determinant = a + b + c;
    if (determinant == 0) {
        return false;
    }
    const float pz0 = pz[0] * q.sz, pz1 = pz[1] * q.sz, pz2 = pz[2] * q.sz;
    const float distance = __fdiv_rn(a * pz0 + b * pz1 + c * pz2, determinant);
    if (!(distance >= tmin && distance <= tmax)) {
        return false;
    }
    // Error bound of PBRT 4 section 6.5.3 with FP32's unit roundoff u = 2^-24.
    constexpr float g2 = 2.0f * 5.9604644775390625e-08f / (1.0f - 2.0f * 5.9604644775390625e-08f);
    constexpr float g3 = 3.0f * 5.9604644775390625e-08f / (1.0f - 3.0f * 5.9604644775390625e-08f);
    constexpr float g5 = 5.0f * 5.9604644775390625e-08f / (1.0f - 5.0f * 5.9604644775390625e-08f);
    const float x = fmaxf(fmaxf(fabsf(px[0]), fabsf(px[1])), fabsf(px[2]));
    const float y = fmaxf(fmaxf(fabsf(py[0]), fabsf(py[1])), fabsf(py[2]));
    const float z = fmaxf(fmaxf(fabsf(pz0), fabsf(pz1)), fabsf(pz2));
    const float error_x    = g5 * (x + z);
    const float error_y    = g5 * (y + z);
    const float error_edge = 2.0f * (g2 * x * y + error_y * x + error_x * y);
    const float edge       = fmaxf(fmaxf(fabsf(a), fabsf(b)), fabsf(c));
    const float error = 3.0f * (g3 * edge * z + error_edge * z + g3 * z * edge);
    // distance <= error / |determinant|, with the division only where the products are within
    // 2^-20 of each other (or not finite, or where the product or the distance is near or below the
    // normal range, so that the quotient may be subnormal and round up by more): elsewhere their
    // rounding cannot change the answer.
    const float scaled = distance * fabsf(determinant);
    if (!(scaled > error * 1.00000095367431640625f && scaled < __int_as_float(0x7f800000) && scaled > 1e-30f &&
          distance >= kFltMin)) {
        if (distance <= error / fabsf(determinant)) {
            return false;
        }
    }
    t   = distance;
    ea  = a;
    eb  = b;
    ec  = c;
    det = determinant;
    return true;
}

// Hit of a two-level traversal: its distance, edge functions and instance.
struct TraceResult {
    float    t;
    uint32_t slot;  // the flat primitive id, kNone: miss
    uint32_t prim;
    float    a, b, c, det;
    uint32_t flags;  // the hit instance's flags
};

// Nearest hit of a flattened traversal. The edge functions are not carried through the traversal:
// hit_edges evaluates them again for the triangle that won, with the arithmetic that accepted it.
struct NearestHit {
    float    t;
    uint32_t slot;  // triangle slot in leaf order, kNone: miss
};

struct TraceCounters {
    uint32_t bounds;
    uint32_t triangles;
};

// No further node: larger than any node index, so one unsigned comparison tells an interior node
// from a leaf reference (negative) and from the end.
constexpr int kNoNode = 0x7fffffff;
constexpr int kDeepNode = 0x7ffffffe;  // stream.cuh: the next nodes are in the stack's local part
constexpr int kPopNode  = 0x7ffffffd;  // stream.cuh: the next node is on the stack

// Nearest hit (ANY_HIT = false) or occlusion (ANY_HIT = true) in [tmin, tmax] over the flattened
// tree. Lanes of a warp traverse interior nodes together and postpone the first leaf they reach
// until every active lane holds one (or has finished), then test leaves together: interior and
// leaf work are not interleaved across lanes.
//
// What bounds it is the load-store pipe (one wavefront per divergent lane and load) and issue
// slots, so a node visit is four 32-byte loads and packed arithmetic, and the state kept across
// the loops is what the loops use: the hit is a distance and a slot, `direction()` fetches the
// ray's direction again for the rare single-sided triangle.
template <bool ANY_HIT, typename Direction>
__device__ __forceinline__ NearestHit trace(const DeviceScene& s, const RayQuery& q, float tmin, float tmax,
                                            Direction direction, TraceCounters& counters, unsigned& error) {
    NearestHit result{tmax, kNone};
    if (!s.has_nodes) {
        return result;
    }
    if (!(finite3(q.o) && finite3(q.d))) {
        error |= kErrorRay;
        return result;
    }
    counters.bounds++;
    const float root_enter =
        slab_enter(q, make_float4(s.root_lo[0], s.root_hi[0], s.root_lo[1], s.root_hi[1]),
                   s.root_lo[2], s.root_hi[2], tmin, tmax);
    if (!(root_enter <= tmax)) {
        return result;
    }
    int2        stack[kStackSize];
    int         sp    = 0;
    int         node  = s.root;  // next node: interior (>= 0) or leaf (< 0)
    bool        alive = true;
    int         leaf  = 0;       // a postponed leaf
    bool        held  = false;
    const float inf   = __int_as_float(0x7f800000);
    const f3    neg_o = -q.o;
    SectorOffsets at;
    at.init(q.neg);
    // Every pass of every loop below visits a node or tests a leaf, and both count against
    // kMaxVisits, so traversal ends on any tree; the streamed walk counts the same. The count is looked
    // at where a subtree is popped, which a descent comes to after at most 64 visits, and at the end
    // (looking at every visit: 64x64x4 frame 252 -> 254 us).
    uint32_t visits = 0;
    // Next stacked subtree that can still contain a nearer hit, or kNoNode.
    const auto pop = [&]() {
        while (sp > 0) {
            const int2 e = stack[--sp];
            if (__int_as_float(e.y) <= result.t) {
                node  = e.x;
                alive = visits <= kMaxVisits;
                return;
            }
        }
        alive = false;
    };
    while (alive || held) {
        if (alive && node < 0 && !held) {  // a leaf to test next (also a root that is a leaf)
            leaf = node;
            held = true;
            pop();
        }
        // Interior phase.
        while (alive && node >= 0) {
            ++visits;
            NodeVisit v;
            v.visit(s.nodes + kWideNode * static_cast<size_t>(node), at, neg_o, neg_o, q.inv_lo, q.inv_hi, tmin,
                    result.t);
            counters.bounds += v.children();
            v.sort();
            if (v.t0 != inf) {
                if (sp > kStackSize - 3) {
                    error |= kErrorStack;
                    return result;
                }
                if (v.t3 != inf) {
                    stack[sp++] = make_int2(v.r3, __float_as_int(v.t3));
                }
                if (v.t2 != inf) {
                    stack[sp++] = make_int2(v.r2, __float_as_int(v.t2));
                }
                if (v.t1 != inf) {
                    stack[sp++] = make_int2(v.r1, __float_as_int(v.t1));
                }
                node = v.r0;
            } else {
                pop();
            }
            if (alive && node < 0 && !held) {  // postpone the first leaf and keep descending
                leaf = node;
                held = true;
                pop();
            }
            if (!__any_sync(__activemask(), !held)) {
                break;  // every lane here holds a leaf
            }
        }
        // Leaf phase: the postponed leaf, then any leaf the lane now points at.
        while (held) {
            ++visits;
            for (uint32_t slot = static_cast<uint32_t>(~leaf);; ++slot) {
                const float4* tp = s.tris + 3 * static_cast<size_t>(slot);
                const float4  a4 = __ldg(tp + 0);
                const float4  b4 = __ldg(tp + 1);
                const float4  c4 = __ldg(tp + 2);
                const unsigned flags = __float_as_uint(b4.w);
                counters.triangles++;
                float t, ea, eb, ec, det;
                if (triangle_test(q.triangle_ray(), xyz(a4), xyz(b4), xyz(c4), tmin, result.t, t, ea, eb, ec,
                                  det)) {
                    bool visible = true;
                    if (flags & kTriSingleSided) {
                        const f3 outward = cross(xyz(b4) - xyz(a4), xyz(c4) - xyz(a4));
                        const float side = dot(direction(), outward);
                        visible = (flags & kTriMirrored) ? side > 0 : side < 0;
                    }
                    // t <= result.t here: nearer, or a tie, which goes to the lower primitive id.
                    if (visible &&
                        (t < result.t || result.slot == kNone ||
                         __float_as_uint(a4.w) <
                             __float_as_uint(__ldg(s.tris + 3 * static_cast<size_t>(result.slot)).w))) {
                        result.t    = t;
                        result.slot = slot;
                        if (ANY_HIT) {
                            error |= visits > kMaxVisits ? kErrorVisits : 0u;
                            return result;
                        }
                    }
                }
                if (flags & kTriLeafEnd) {
                    break;
                }
            }
            held = false;
            if (alive && node < 0) {
                leaf = node;
                held = true;
                pop();
            }
        }
    }
    error |= visits > kMaxVisits ? kErrorVisits : 0u;
    return result;
}

// Edge functions and determinant of the triangle in `slot` for a ray that hit it: the values
// triangle_test accepted.
__device__ __forceinline__ void hit_edges(const DeviceScene& s, const TriangleRay& q, uint32_t slot, float& ea,
                                          float& eb, float& ec, float& det, unsigned& flags, uint32_t& prim) {
    const float4* tp = s.tris + 3 * static_cast<size_t>(slot);
    const float4  a4 = __ldg(tp + 0), b4 = __ldg(tp + 1), c4 = __ldg(tp + 2);
    float         z[3], x[3], y[3];
    triangle_edges(q, xyz(a4), xyz(b4), xyz(c4), x, y, z, ea, eb, ec);
    det   = ea + eb + ec;
    flags = __float_as_uint(b4.w);
    prim  = __float_as_uint(a4.w);
}

// ---- two-level scenes ----

// The world ray mapped into an instance's object space (same parameter t: the direction is not
// renormalised), for slab tests against the instance's mesh boxes grown by `margin` on every
// side. The growth is folded into the origin per axis: o_near/o_far are the origins the near and
// far planes are measured from. It covers the rounding of this mapping and of the flattening's
// FP32 world vertices (whose world-space triangles are the ones tested), so a box that a
// world-space triangle of the instance hits is never culled.
struct ObjectRay {
    float o_near[3], o_far[3];
    float inv_lo[3], inv_hi[3];
    bool  neg[3];
    __device__ __forceinline__ f3 near_origin() const { return {o_near[0], o_near[1], o_near[2]}; }
    __device__ __forceinline__ f3 far_origin() const { return {o_far[0], o_far[1], o_far[2]}; }
};

constexpr float kInstanceMarginScale = 1.9073486328125e-06f;  // 2^-19 = 32 FP32 unit roundoffs

__device__ __forceinline__ void object_ray(const DeviceInstance2& inst, const RayQuery& qw,
                                           float t_exit, ObjectRay& r) {
    const float* m = inst.to_object;
    const f3 o = {fmaf(m[0], qw.o.x, fmaf(m[1], qw.o.y, fmaf(m[2], qw.o.z, m[3]))),
                  fmaf(m[4], qw.o.x, fmaf(m[5], qw.o.y, fmaf(m[6], qw.o.z, m[7]))),
                  fmaf(m[8], qw.o.x, fmaf(m[9], qw.o.y, fmaf(m[10], qw.o.z, m[11])))};
    const f3 d = {fmaf(m[0], qw.d.x, fmaf(m[1], qw.d.y, m[2] * qw.d.z)),
                  fmaf(m[4], qw.d.x, fmaf(m[5], qw.d.y, m[6] * qw.d.z)),
                  fmaf(m[8], qw.d.x, fmaf(m[9], qw.d.y, m[10] * qw.d.z))};
    const float reach  = max3(fabs3(qw.o)) + t_exit * max3(fabs3(qw.d));
    const float margin = inst.margin_static +
                         kInstanceMarginScale * (fmaf(inst.a_norm, reach, inst.b_norm));
    const float lo = 0.99999904632568359375f, hi = 1.00000095367431640625f;  // 1 -+ 2^-20
    for (int a = 0; a < 3; ++a) {
        const float c   = comp(d, a);
        const float inv = 1.0f / c;
        r.inv_lo[a]     = inv * lo;
        r.inv_hi[a]     = inv * hi;
        r.neg[a]        = signbit(c);
        const float oa  = comp(o, a);
        r.o_near[a]     = r.neg[a] ? oa - margin : oa + margin;
        r.o_far[a]      = r.neg[a] ? oa + margin : oa - margin;
    }
}

// Entry and exit of a world box, or false when the ray misses it within [tmin, tmax].
__device__ __forceinline__ bool world_box(const RayQuery& q, const float* lo, const float* hi,
                                          float tmin, float tmax, float& enter, float& leave) {
    const float nx = ((q.neg[0] ? hi[0] : lo[0]) - q.o.x) * q.inv_lo[0];
    const float fx = ((q.neg[0] ? lo[0] : hi[0]) - q.o.x) * q.inv_hi[0];
    const float ny = ((q.neg[1] ? hi[1] : lo[1]) - q.o.y) * q.inv_lo[1];
    const float fy = ((q.neg[1] ? lo[1] : hi[1]) - q.o.y) * q.inv_hi[1];
    const float nz = ((q.neg[2] ? hi[2] : lo[2]) - q.o.z) * q.inv_lo[2];
    const float fz = ((q.neg[2] ? lo[2] : hi[2]) - q.o.z) * q.inv_hi[2];
    enter = fmaxf(fmaxf(tmin, nx), fmaxf(ny, nz));
    leave = fminf(fminf(tmax, fx), fminf(fy, fz));
    return enter <= leave;
}

// A wide node's or a lone leaf's stack discipline: a stack of (ref, entry) pairs shared by the
// two levels; entries beyond the current nearest hit are skipped when popped.
constexpr int kStackSize2 = 3 * 64 * 2 + 3;

// Nearest hit / occlusion in a two-level scene. The instance-level tree is traversed with the
// world ray; an instance whose world box the ray enters has its mesh tree traversed with the
// ray mapped into object space, and every candidate triangle is transformed to world space with
// the flattening's arithmetic (transform_point) and tested with the world ray: the same vertices,
// ray and test as the flattened scene, so the same hits (ties still go to the lower flat
// primitive id).
template <bool ANY_HIT>
__device__ __forceinline__ TraceResult trace2(const DeviceScene& s, const RayQuery& q, float tmin,
                                           float tmax, TraceCounters& counters, unsigned& error) {
    TraceResult result;
    result.t     = tmax;
    result.slot  = kNone;
    result.prim  = kNone;
    result.flags = 0;
    if (!s.has_nodes) {
        return result;
    }
    if (!(finite3(q.o) && finite3(q.d))) {
        error |= kErrorRay;
        return result;
    }
    counters.bounds++;
    float enter, leave;
    if (!world_box(q, s.root_lo, s.root_hi, tmin, tmax, enter, leave)) {
        return result;
    }
    int2     stack[kStackSize2];
    int      sp     = 0;
    uint32_t visits = 0;
    const float inf = __int_as_float(0x7f800000);
    SectorOffsets at_w;
    at_w.init(q.neg);
    stack[sp++] = make_int2(s.root, __float_as_int(enter));
    while (sp > 0) {
        const int2 top = stack[--sp];
        if (__int_as_float(top.y) > result.t) {
            continue;
        }
        if (++visits > kMaxVisits) {
            error |= kErrorVisits;
            return result;
        }
        const int node = top.x;
        if (node >= 0) {  // instance-level interior node
            NodeVisit v;
            v.visit(s.nodes + kWideNode * static_cast<size_t>(node), at_w, -q.o, -q.o, q.inv_lo, q.inv_hi, tmin, result.t);
            counters.bounds += v.children();
            v.sort();
            if (sp > kStackSize2 - 4) {
                error |= kErrorStack;
                return result;
            }
            const int   r[4] = {v.r0, v.r1, v.r2, v.r3};
            const float t[4] = {v.t0, v.t1, v.t2, v.t3};
            for (int k = 3; k >= 0; --k) {
                if (t[k] != inf) {
                    stack[sp++] = make_int2(r[k], __float_as_int(t[k]));
                }
            }
            continue;
        }
        // Instance-level leaf: its instances in order.
        for (uint32_t item = static_cast<uint32_t>(~node);; ++item) {
            const uint32_t         word = __ldg(s.tlas_items + item);
            const DeviceInstance2& inst = s.instances[word & 0x7fffffffu];
            counters.bounds++;
            float ienter, ileave;
            if (world_box(q, inst.lo, inst.hi, tmin, result.t, ienter, ileave)) {
                ObjectRay ro;
                object_ray(inst, q, ileave, ro);
                SectorOffsets at_o;
                at_o.init(ro.neg);
                const int base = sp;
                stack[sp++] = make_int2(inst.blas_root, __float_as_int(ienter));
                while (sp > base) {
                    const int2 e = stack[--sp];
                    if (__int_as_float(e.y) > result.t) {
                        continue;
                    }
                    if (++visits > kMaxVisits) {
                        error |= kErrorVisits;
                        return result;
                    }
                    if (e.x >= 0) {  // mesh-level interior node
                        NodeVisit v;
                        v.visit(s.blas_nodes + kWideNode * static_cast<size_t>(e.x), at_o, -ro.near_origin(), -ro.far_origin(), ro.inv_lo, ro.inv_hi, tmin, result.t);
                        counters.bounds += v.children();
                        v.sort();
                        if (sp > kStackSize2 - 4) {
                            error |= kErrorStack;
                            return result;
                        }
                        const int   r[4] = {v.r0, v.r1, v.r2, v.r3};
                        const float t[4] = {v.t0, v.t1, v.t2, v.t3};
                        for (int k = 3; k >= 0; --k) {
                            if (t[k] != inf) {
                                stack[sp++] = make_int2(r[k], __float_as_int(t[k]));
                            }
                        }
                        continue;
                    }
                    // Mesh-level leaf: its triangles, transformed to world space.
                    for (uint32_t slot = static_cast<uint32_t>(~e.x);; ++slot) {
                        const float4* tp = s.blas_tris + 3 * static_cast<size_t>(slot);
                        const float4  a4 = __ldg(tp + 0);
                        const float4  b4 = __ldg(tp + 1);
                        const float4  c4 = __ldg(tp + 2);
                        const f3 v0 = transform_point(inst.to_world, a4.x, a4.y, a4.z);
                        const f3 v1 = transform_point(inst.to_world, b4.x, b4.y, b4.z);
                        const f3 v2 = transform_point(inst.to_world, c4.x, c4.y, c4.z);
                        counters.triangles++;
                        float tt, ea, eb, ec, det;
                        if (triangle_test(q.triangle_ray(), v0, v1, v2, tmin, result.t, tt, ea, eb, ec, det)) {
                            bool visible = true;
                            if (inst.flags & kTriSingleSided) {
                                const float side = dot(q.d, cross(v1 - v0, v2 - v0));
                                visible = (inst.flags & kTriMirrored) ? side > 0 : side < 0;
                            }
                            const uint32_t prim = inst.first_prim + __float_as_uint(a4.w);
                            if (visible && (tt < result.t || (tt == result.t && prim < result.prim) ||
                                            result.slot == kNone)) {
                                result.t     = tt;
                                result.slot  = prim;
                                result.prim  = prim;
                                result.a     = ea;
                                result.b     = eb;
                                result.c     = ec;
                                result.det   = det;
                                result.flags = inst.flags;
                                if (ANY_HIT) {
                                    return result;
                                }
                            }
                        }
                        if (__float_as_uint(b4.w) & kTriLeafEnd) {
                            break;
                        }
                    }
                }
            }
            if (word & 0x80000000u) {
                break;
            }
        }
    }
    return result;
}

}  // namespace mr
