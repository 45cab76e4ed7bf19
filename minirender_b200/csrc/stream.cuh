// stream.cuh — warps that stream rays through the flattened traversal.
//
// A warp keeps up to 32 rays in flight and every step of its loop is one of three, chosen by votes
// of all 32 lanes, so the warp is converged at each choice:
//   refill  when kRefill lanes have finished (or all have): their results are handed on and the
//           lanes take the next rays of the warp's chunk of the queue;
//   visit   lanes at an interior node test its four children;
//   leaf    lanes holding a leaf test one of its triangles.
// Visit or leaf goes to the larger group. A lane postpones the leaf it reaches and keeps descending
// until it meets a second one, so most lanes can do either. (Persistent warps that fetch rays by a vote
// and a postponed leaf per lane: Aila and Laine, "Understanding the Efficiency of Ray Traversal on
// GPUs", HPG 2009.)
//
// Against one fetch of 32 rays that a warp traces to the end of the slowest, a step runs 18 lanes of
// 32 where it ran 11 (half of the lane slots had waited for the slowest ray of their fetch, and
// visits and leaves had excluded one another's lanes). What bounds it now is the load-store pipe:
// one wavefront per divergent lane and load (76% busy), then issue slots (69%). Hence a node visit
// of four 32-byte loads instead of eight of 16 bytes, a traversal stack in shared memory, where
// lanes at different depths do not conflict, and a hit kept as distance and slot alone. Traversal
// launches of one frame on a B200, before and after: 261k-triangle room, 556^2 x 49, depth 11: 38.7
// and 30.9 ms; 1M-triangle field, 1920 x 1080 x 16, depth 12: 62.6 and 53.2 ms; the same in fog,
// 961 x 541 x 8, depth 16, with its medium launches: 16.1 and 14.2 ms.
#pragma once

#include "traverse.cuh"

namespace mr {

// Lanes that have to be idle before a refill. Each one waits for the queue, the ray and the bin
// counters, so few, large refills win, until too few lanes are left to run (room, traversal launches
// with 20, 22, 24 and 26: 30.9, 30.9, 31.2 and 31.7 ms; 8: 8% more than 24).
constexpr int kRefill = 22;
// Largest chunk of the queue that a warp claims at once: its rays are neighbours in the sorted queue
// and so in the tree.
constexpr uint32_t kStreamChunk = 256;
constexpr int      kStreamBlock = 128;  // threads per block of a kernel that streams
// Stack entries per lane in shared memory. 16 entries of 8 resident blocks take 128 KB of the SM's
// 256 KB; 24 leave the nodes too little L1 (room 4% slower).
constexpr uint32_t kStackShared = 16;
constexpr size_t   kStreamSharedBytes = kStackShared * kStreamBlock * sizeof(int2);

// A lane's traversal stack: column threadIdx.x of a (entries x block) array in shared memory, whose
// first entry is the end mark. `top` is the byte address of the next free entry. A visit pushes its
// up to three entries unchecked; when fewer than three are left, spill() moves kMoved older ones to
// local memory and leaves a mark in their place. Popping the mark makes kDeepNode the node, and the
// lane waits for the next refill to get them back, which keeps all of this out of the loop: few rays
// ever stack so much. The shared accesses are predicated instructions: as branches they would
// split the warp.
struct StreamStack {
    static constexpr uint32_t kStep  = kStreamBlock * sizeof(int2);
    static constexpr uint32_t kMoved = 8;
    static constexpr uint32_t kFull  = kStackShared - 3;       // more entries than this: spill
    static constexpr uint32_t kMark  = kFull - kMoved;         // entry the mark takes
    uint32_t top, base;

    __device__ __forceinline__ static void store(uint32_t address, int2 e) {
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(address), "r"(e.x), "r"(e.y));
    }
    __device__ __forceinline__ static int2 fetch(uint32_t address) {
        int2 e;
        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(e.x), "=r"(e.y) : "r"(address));
        return e;
    }
    __device__ __forceinline__ void init(void* shared) {
        base = static_cast<uint32_t>(__cvta_generic_to_shared(shared)) + threadIdx.x * static_cast<uint32_t>(sizeof(int2));
        store(base, make_int2(kNoNode, 0));
        clear();
    }
    // Empty but for the end mark.
    __device__ __forceinline__ void clear() { top = base + kStep; }
    __device__ __forceinline__ bool full() const { return top > base + kFull * kStep; }
    // Pushes (ref, t) unless t is +inf.
    __device__ __forceinline__ void push(int ref, float t) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.lt.f32 p, %2, 0f7F800000;\n\t"
            "@p st.shared.v2.b32 [%0], {%1, %3};\n\t"
            "@p add.u32 %0, %0, %4;\n\t}"
            : "+r"(top)
            : "r"(ref), "f"(t), "r"(__float_as_int(t)), "n"(kStep));
    }
    // Where `node` is kPopNode, takes the top entry; it becomes the node unless it lies beyond `far`.
    __device__ __forceinline__ void pop(int& node, float far) {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t.reg .b32 x, y;\n\t"
            "setp.eq.s32 p, %0, %3;\n\t"
            "@p sub.u32 %1, %1, %4;\n\t"
            "@p ld.shared.v2.b32 {x, y}, [%1];\n\t"
            "setp.le.and.f32 q, y, %2, p;\n\t"
            "@q mov.b32 %0, x;\n\t}"
            : "+r"(node), "+r"(top)
            : "f"(far), "n"(kPopNode), "n"(kStep));
    }
};

// The local part of a lane's stack: the moved entries, their count in the first element. spill()
// and restore() take and return `top` by value and are not inlined, so the hot loop keeps the stack
// in registers. Each spill but the first moves the mark of the one before along with kMoved - 1 nodes,
// and the shared part holds kFull - 2 nodes beside the end mark and the newest mark, so kSpills spills
// hold kStackSize nodes.
constexpr uint32_t kSpillNodes = StreamStack::kMoved - 1;
constexpr uint32_t kSpills =
    (kStackSize - 1 - (StreamStack::kFull - 2) + kSpillNodes - 1) / kSpillNodes;
constexpr uint32_t kDeepNodes = kSpills * StreamStack::kMoved;
constexpr uint32_t kDeepSize  = 1 + kDeepNodes;
static_assert(1 + kSpills * kSpillNodes + StreamStack::kFull - 2 >= kStackSize, "spilled nodes and shared ones");

// For a full() stack: entries kMark .. kMark + kMoved - 1 move, the newer ones close up. Returns the
// new top, 0 when the local part is full too.
static __device__ __noinline__ uint32_t spill(uint32_t base, uint32_t top, int2* deep) {
    constexpr uint32_t step = StreamStack::kStep;
    const uint32_t     moved = static_cast<uint32_t>(deep[0].x);
    if (moved + StreamStack::kMoved > kDeepNodes) {
        return 0;
    }
    const uint32_t mark = base + StreamStack::kMark * step;
    for (uint32_t k = 0; k < StreamStack::kMoved; ++k) {
        deep[1 + moved + k] = StreamStack::fetch(mark + k * step);
    }
    deep[0].x = static_cast<int>(moved + StreamStack::kMoved);
    StreamStack::store(mark, make_int2(kDeepNode, 0));
    uint32_t to = mark + step;
    for (uint32_t from = mark + StreamStack::kMoved * step; from < top; from += step, to += step) {
        StreamStack::store(to, StreamStack::fetch(from));
    }
    return to;
}

// When the mark has been popped: the newest moved entries take their places again. Returns the top.
static __device__ __noinline__ uint32_t restore(uint32_t top, int2* deep) {
    constexpr uint32_t step  = StreamStack::kStep;
    const uint32_t     moved = static_cast<uint32_t>(deep[0].x) - StreamStack::kMoved;
    for (uint32_t k = 0; k < StreamStack::kMoved; ++k) {
        StreamStack::store(top + k * step, deep[1 + moved + k]);
    }
    deep[0].x = static_cast<int>(moved);
    return top + StreamStack::kMoved * step;
}

// What a lane keeps of its ray: RayQuery's numbers, with the permutation, the sector offsets and
// the visit count in one word.
struct StreamRay {
    f3       o;
    float    inv_lo[3], inv_hi[3];
    float    sx, sy, sz;
    uint32_t word;  // bits 0-3 near_xy, 4-7 near_z, 8-13 kx ky kz, 14-31 visits
    static constexpr uint32_t kVisit    = 1u << 14;
    static constexpr uint32_t kTooMany  = (kMaxVisits + 1) * kVisit;  // a word that counts more than kMaxVisits
    static_assert(kMaxVisits + 1 < 1u << 18, "the count's bits");
    __device__ __forceinline__ void init(const RayQuery& q) {
        o = q.o;
        for (int a = 0; a < 3; ++a) {
            inv_lo[a] = q.inv_lo[a];
            inv_hi[a] = q.inv_hi[a];
        }
        sx = q.sx, sy = q.sy, sz = q.sz;
        SectorOffsets at;
        at.init(q.neg);
        word = static_cast<uint32_t>(at.near_xy | at.near_z << 4 | q.kx << 8 | q.ky << 10 | q.kz << 12);
    }
    __device__ __forceinline__ SectorOffsets sectors() const {
        return {static_cast<int>(word & 15u), static_cast<int>((word >> 4) & 15u)};
    }
    __device__ __forceinline__ TriangleRay triangle_ray() const {
        return {o, static_cast<int>((word >> 8) & 3u), static_cast<int>((word >> 10) & 3u),
                static_cast<int>((word >> 12) & 3u), sx, sy, sz};
    }
};

// Streams the items [0, n) of `io` through the flattened traversal: nearest hit (ANY_HIT = false)
// or occlusion. Called by all threads of a block of kStreamBlock threads with kStreamSharedBytes of
// shared memory; `work` counts the claimed items. `io` has
//   kBatch                  the lanes' scenes differ
//   load(i, o, d)           item i's ray: origin + tmin, direction + tmax; makes the lane's scene
//                           current. ANY_HIT rays start at 0 and end at o.w.
//   scene() nodes() tris()  the lane's scene and its arrays
//   direction()             the ray's direction again
//   finish(done, ray, hit)  called by all 32 lanes; the lanes with `done` hand on their result
//   fail(bits)              records an error of the lane's item
template <bool ANY_HIT, typename Io>
__device__ __forceinline__ void stream_rays(Io& io, uint32_t n, uint32_t* work, void* shared, TraceCounters& counters) {
    const int      lane  = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (kStreamBlock / 32);
    const uint32_t chunk = min(kStreamChunk, max(32u, n / (4 * warps) & ~31u));
    bool           filled = false;  // the lane has an item
    int            node = kNoNode, leaf = 0;
    float          tmin = 0;
    NearestHit     hit{0, kNone};
    StreamRay      ray;
    uint32_t       next = 0, end = 0;  // the rest of the warp's chunk
    int            refill = kRefill;  // 32 once the queue is empty
    int2           deep[kDeepSize];
    StreamStack    stack;
    stack.init(shared);
    // load() writes the ray before anything reads it. Written here too, it takes another place among the
    // registers: the plain kernel spills 60 bytes instead of 66 (traversal of the room frame 28.2 against
    // 28.6 ms), the multi-job one 160 instead of 124 (24 preview jobs 7.0 against 6.9 ms).
    if constexpr (!Io::kBatch) {
        ray = StreamRay{};
    }
    while (true) {
        stack.pop(node, hit.t);
        if (node < 0 && leaf == 0) {  // postpone the first leaf and keep descending
            leaf = node;
            node = kPopNode;
            ray.word += StreamRay::kVisit;
        }
        const bool     idle      = node >= kDeepNode && leaf == 0;  // finished, or waiting for restore()
        const bool     interior  = static_cast<unsigned>(node) < static_cast<unsigned>(kPopNode);
        const unsigned interiors = __ballot_sync(0xffffffffu, interior);
        const unsigned leaves    = __ballot_sync(0xffffffffu, leaf < 0);
        const unsigned idles     = __ballot_sync(0xffffffffu, idle);
        if (__popc(idles) >= refill) {
            const bool done = idle && node == kNoNode;
            if (done && filled && ray.word >= StreamRay::kTooMany) {  // with its last leaves
                io.fail(kErrorVisits);
            }
            io.finish(done && filled, ray, hit);
            filled = filled && !done;
            if (idle && !done) {
                stack.top = restore(stack.top, deep);
                node      = kPopNode;
            }
            if (refill == 32) {  // the queue is empty
                if (__all_sync(0xffffffffu, done)) {
                    break;
                }
                continue;
            }
            const unsigned dones = __ballot_sync(0xffffffffu, done);
            if (next == end) {
                uint32_t base = 0;
                if (lane == 0) {
                    base = atomicAdd(work, chunk);
                }
                base = __shfl_sync(0xffffffffu, base, 0);
                next = min(base, n);
                end  = min(base + chunk, n);
                refill = next == end ? 32 : kRefill;
            }
            const uint32_t i = next + __popc(dones & ((1u << lane) - 1u));
            next             = min(end, next + __popc(dones));
            if (done && i < end) {
                filled = true;
                float4 o4, d4;
                io.load(i, o4, d4);
                tmin             = ANY_HIT ? 0.0f : o4.w;
                const float tmax = ANY_HIT ? o4.w : d4.w;
                hit              = {tmax, kNone};
                RayQuery q;
                q.init(xyz(o4), xyz(d4));
                ray.init(q);
                const DeviceScene& s = io.scene();
                if (s.has_nodes) {
                    if (!(finite3(q.o) && finite3(q.d))) {
                        io.fail(kErrorRay);
                    } else {
                        counters.bounds++;
                        const float enter =
                            slab_enter(q, make_float4(s.root_lo[0], s.root_hi[0], s.root_lo[1], s.root_hi[1]),
                                       s.root_lo[2], s.root_hi[2], tmin, tmax);
                        if (enter <= tmax) {
                            node = s.root;
                            stack.clear();
                            deep[0].x = 0;
                        }
                    }
                }
            }
            continue;
        }
        if (__popc(interiors) >= __popc(leaves)) {
            if (interior) {
                NodeVisit v;
                v.visit(io.nodes() + kWideNode * static_cast<size_t>(node), ray.sectors(), -ray.o, -ray.o,
                        ray.inv_lo, ray.inv_hi, tmin, hit.t);
                counters.bounds += v.children();
                v.sort();
                node = v.t0 != __int_as_float(0x7f800000) ? v.r0 : kPopNode;
                stack.push(v.r3, v.t3);
                stack.push(v.r2, v.t2);
                stack.push(v.r1, v.t1);
                // Every visit counts and each leaf was pushed by one, so this ends traversal on any
                // tree; the stack, with its local part, holds the kStackSize nodes that cover every
                // accepted tree.
                ray.word += StreamRay::kVisit;
                if (ray.word >= StreamRay::kTooMany || stack.full()) {
                    const bool visits = ray.word >= StreamRay::kTooMany;
                    stack.top         = visits ? 0 : spill(stack.base, stack.top, deep);
                    if (stack.top == 0) {
                        io.fail(visits ? kErrorVisits : kErrorStack);
                        node = kNoNode;
                        leaf = 0;
                    }
                }
            }
        } else if (leaf < 0) {
            const uint32_t slot  = static_cast<uint32_t>(~leaf);
            const float4*  tp    = io.tris() + 3 * static_cast<size_t>(slot);
            const float4   a4    = __ldg(tp + 0);
            const float4   b4    = __ldg(tp + 1);
            const float4   c4    = __ldg(tp + 2);
            const unsigned flags = __float_as_uint(b4.w);
            counters.triangles++;
            leaf = flags & kTriLeafEnd ? 0 : leaf - 1;  // ~(slot + 1)
            float t, ea, eb, ec, det;
            if (triangle_test(ray.triangle_ray(), xyz(a4), xyz(b4), xyz(c4), tmin, hit.t, t, ea, eb, ec, det)) {
                bool visible = true;
                if (flags & kTriSingleSided) {
                    const f3    outward = cross(xyz(b4) - xyz(a4), xyz(c4) - xyz(a4));
                    const float side    = dot(io.direction(), outward);
                    visible             = (flags & kTriMirrored) ? side > 0 : side < 0;
                }
                // t <= hit.t here: nearer, or a tie, which goes to the lower primitive id.
                if (visible && (t < hit.t || hit.slot == kNone ||
                                __float_as_uint(a4.w) <
                                    __float_as_uint(__ldg(io.tris() + 3 * static_cast<size_t>(hit.slot)).w))) {
                    hit.t    = t;
                    hit.slot = slot;
                    if (ANY_HIT) {
                        node = kNoNode;
                        leaf = 0;
                    }
                }
            }
        }
    }
}

}  // namespace mr
