// builder.cu — GPU binned-SAH BVH builder.
//
// The algorithm is the reference's recursive builder (src/render/bvh.cpp:101-196) evaluated
// breadth-first on the GPU: 12 centroid bins per axis, C_T = C_I = 1, a leaf when a node holds at
// most 4 primitives, sits at depth 48, has no split with nonempty sides, or no split cheaper than
// the leaf cost (its primitive count). Ties keep the first axis and split in the reference's
// search order. Partitioning is stable (the reference's std::partition is not; the resulting
// primitive sets, and so the tree topology, are the same).
//
// Two regimes:
//  - nodes with more than kSmallTask primitives are processed one level at a time by the whole
//    GPU: fixed-size chunks of a node's primitive range reduce bounds and bin in shared memory
//    and merge with one atomic per value per chunk; splits are chosen one warp per node;
//    primitives are scattered with a chunk scan so the order is deterministic. One block lists a
//    level's chunks and emits the next level's tasks in order, so the host reads three numbers per
//    level and sorts nothing;
//  - smaller nodes are finished by one warp each, depth-first in shared memory, with node
//    indices taken from a range reserved per subtree (unused indices are squeezed out at the end).
// All arithmetic is FP32. Surface areas are evaluated on extents scaled by a power of two so the
// products cannot overflow (the reference uses double for the same reason, intersection.cpp:44-50).
#include <algorithm>

#include "errors.hpp"
#include "scan.cuh"
#include "scene.cuh"

namespace mr {
namespace {

constexpr int      kBins         = 12;
constexpr uint32_t kMaxDepth     = 48;
constexpr uint32_t kLeafSize     = 4;
constexpr uint32_t kSmallTask    = 256;   // nodes at most this large are built by one warp
constexpr uint32_t kChunk        = 2048;  // primitives per block in the level-wide passes
constexpr int      kSmallWarps   = 4;     // warps per block in the small-task kernel
constexpr uint32_t kUnusedNode   = 0xffffffffu;

__device__ __forceinline__ uint32_t f2o(float f) {  // order-preserving float -> uint
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
constexpr uint32_t kOrderedPosInf = 0xff800000u;  // f2o(+inf)
constexpr uint32_t kOrderedNegInf = 0x007fffffu;  // f2o(-inf)

// bin_index (src/render/bvh.cpp:23-27) in FP32.
__device__ __forceinline__ int bin_of(float c, float lo, float hi) {
    const float coordinate = (c - lo) / (hi - lo);
    const float scaled     = coordinate * static_cast<float>(kBins);
    return min(static_cast<int>(scaled), kBins - 1);
}

// Surface area of a box scaled by `s` (a power of two).
__device__ __forceinline__ float scaled_area(const float* lo, const float* hi, float s) {
    if (lo[0] > hi[0] || lo[1] > hi[1] || lo[2] > hi[2]) {
        return 0.0f;
    }
    const float ex = (hi[0] - lo[0]) * s, ey = (hi[1] - lo[1]) * s, ez = (hi[2] - lo[2]) * s;
    return 2.0f * (ex * ey + ey * ez + ez * ex);
}

__device__ __forceinline__ float area_scale(const float* lo, const float* hi) {
    const float m = fmaxf(fmaxf(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]);
    if (!(m > 0) || !isfinite(m)) {
        return 1.0f;
    }
    int e;
    frexpf(m, &e);
    return ldexpf(1.0f, -e);  // exact power of two, brings the largest extent into [0.5, 1)
}

struct Task {  // a node still to be split
    uint32_t begin, end;
    uint32_t node;
    uint32_t depth;
    uint32_t range;  // small tasks: first node index reserved for descendants
};

struct TaskBounds {  // ordered-uint encoded: bounds lo/hi, centroid lo/hi
    uint32_t v[12];
};

struct TaskBins {  // per axis, per bin: count and bounds (ordered uints)
    uint32_t count[3][kBins];
    uint32_t box[3][kBins][6];
};

struct Chunk {
    uint32_t task;
    uint32_t begin, end;
};

struct Split {
    int      axis;       // -1: leaf
    int      bin;
    uint32_t left_count;
};

__global__ void init_task_state(TaskBounds* bounds, TaskBins* bins, uint32_t count) {
    const uint32_t t = blockIdx.x;
    if (t >= count) {
        return;
    }
    for (int i = threadIdx.x; i < 12; i += blockDim.x) {
        bounds[t].v[i] = (i % 6) < 3 ? kOrderedPosInf : kOrderedNegInf;
    }
    uint32_t* c = &bins[t].count[0][0];
    for (int i = threadIdx.x; i < 3 * kBins; i += blockDim.x) {
        c[i] = 0;
    }
    uint32_t* b = &bins[t].box[0][0][0];
    for (int i = threadIdx.x; i < 3 * kBins * 6; i += blockDim.x) {
        b[i] = (i % 6) < 3 ? kOrderedPosInf : kOrderedNegInf;
    }
}

// Pass 1: node bounds and centroid bounds.
__global__ void reduce_bounds_kernel(const Chunk* chunks, const uint32_t* chunk_total, const uint32_t* order, const float4* plo,
                                     const float4* phi, const float4* pc, TaskBounds* bounds) {
    if (blockIdx.x >= *chunk_total) {
        return;
    }
    __shared__ uint32_t s[12];
    const Chunk ch = chunks[blockIdx.x];
    if (threadIdx.x < 12) {
        s[threadIdx.x] = (threadIdx.x % 6) < 3 ? kOrderedPosInf : kOrderedNegInf;
    }
    __syncthreads();
    float v[12];
    for (int i = 0; i < 12; ++i) {
        v[i] = (i % 6) < 3 ? INFINITY : -INFINITY;
    }
    for (uint32_t i = ch.begin + threadIdx.x; i < ch.end; i += blockDim.x) {
        const uint32_t p = order[i];
        const float4 a = __ldg(plo + p), b = __ldg(phi + p), c = __ldg(pc + p);
        v[0] = fminf(v[0], a.x), v[1] = fminf(v[1], a.y), v[2] = fminf(v[2], a.z);
        v[3] = fmaxf(v[3], b.x), v[4] = fmaxf(v[4], b.y), v[5] = fmaxf(v[5], b.z);
        v[6] = fminf(v[6], c.x), v[7] = fminf(v[7], c.y), v[8] = fminf(v[8], c.z);
        v[9] = fmaxf(v[9], c.x), v[10] = fmaxf(v[10], c.y), v[11] = fmaxf(v[11], c.z);
    }
    for (int i = 0; i < 12; ++i) {
        float x = v[i];
        for (int o = 16; o > 0; o >>= 1) {
            const float y = __shfl_xor_sync(0xffffffffu, x, o);
            x = (i % 6) < 3 ? fminf(x, y) : fmaxf(x, y);
        }
        if ((threadIdx.x & 31) == 0) {
            if ((i % 6) < 3) {
                atomicMin(&s[i], f2o(x));
            } else {
                atomicMax(&s[i], f2o(x));
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        if ((threadIdx.x % 6) < 3) {
            atomicMin(&bounds[ch.task].v[threadIdx.x], s[threadIdx.x]);
        } else {
            atomicMax(&bounds[ch.task].v[threadIdx.x], s[threadIdx.x]);
        }
    }
}

// Pass 2: 12 bins per axis.
__global__ void bin_kernel(const Chunk* chunks, const uint32_t* chunk_total, const uint32_t* order, const float4* plo,
                           const float4* phi, const float4* pc, const TaskBounds* bounds,
                           TaskBins* bins) {
    if (blockIdx.x >= *chunk_total) {
        return;
    }
    __shared__ uint32_t count[3][kBins];
    __shared__ uint32_t box[3][kBins][6];
    const Chunk ch = chunks[blockIdx.x];
    for (int i = threadIdx.x; i < 3 * kBins; i += blockDim.x) {
        (&count[0][0])[i] = 0;
    }
    for (int i = threadIdx.x; i < 3 * kBins * 6; i += blockDim.x) {
        (&box[0][0][0])[i] = (i % 6) < 3 ? kOrderedPosInf : kOrderedNegInf;
    }
    __syncthreads();
    const TaskBounds& tb = bounds[ch.task];
    float clo[3], chi[3];
    for (int a = 0; a < 3; ++a) {
        clo[a] = o2f(tb.v[6 + a]);
        chi[a] = o2f(tb.v[9 + a]);
    }
    for (uint32_t i = ch.begin + threadIdx.x; i < ch.end; i += blockDim.x) {
        const uint32_t p = order[i];
        const float4 a = __ldg(plo + p), b = __ldg(phi + p), c = __ldg(pc + p);
        const float cc[3] = {c.x, c.y, c.z};
        for (int axis = 0; axis < 3; ++axis) {
            if (chi[axis] == clo[axis]) {
                continue;
            }
            const int k = bin_of(cc[axis], clo[axis], chi[axis]);
            atomicAdd(&count[axis][k], 1u);
            atomicMin(&box[axis][k][0], f2o(a.x));
            atomicMin(&box[axis][k][1], f2o(a.y));
            atomicMin(&box[axis][k][2], f2o(a.z));
            atomicMax(&box[axis][k][3], f2o(b.x));
            atomicMax(&box[axis][k][4], f2o(b.y));
            atomicMax(&box[axis][k][5], f2o(b.z));
        }
    }
    __syncthreads();
    TaskBins& out = bins[ch.task];
    for (int i = threadIdx.x; i < 3 * kBins; i += blockDim.x) {
        const uint32_t c = (&count[0][0])[i];
        if (c) {
            atomicAdd(&(&out.count[0][0])[i], c);
        }
    }
    for (int i = threadIdx.x; i < 3 * kBins * 6; i += blockDim.x) {
        const uint32_t v = (&box[0][0][0])[i];
        if ((i % 6) < 3) {
            if (v != kOrderedPosInf) atomicMin(&(&out.box[0][0][0])[i], v);
        } else {
            if (v != kOrderedNegInf) atomicMax(&(&out.box[0][0][0])[i], v);
        }
    }
}

// SAH sweep over the 12 bins of the three axes (src/render/bvh.cpp:131-183) by one warp: each lane
// evaluates one or two of the 33 splits, joining the bins on either side from their ordered-integer
// boxes (an empty bin's box is empty), and the cheapest wins, the first in the reference's order among
// equals. Every lane returns the result. One lane doing the whole sweep, its bins in local memory,
// had been most of the small tasks' time: their launch takes 0.63 ms for a 476k-triangle room with split
// references where it took 2.33 ms, the tree bit for bit the same (B200).
__device__ __forceinline__ Split choose_split(const float* lo, const float* hi, const float* clo, const float* chi,
                                              uint32_t count, const uint32_t* bin_count, const uint32_t* bin_box) {
    constexpr uint32_t kSplits = kBins - 1, kNoCost = 0xffffffffu;
    const uint32_t     lane    = threadIdx.x & 31;
    const float        s       = area_scale(lo, hi);
    const float        parent  = scaled_area(lo, hi, s);
    uint32_t           best_cost = kNoCost, best = 0, best_left = 0;  // costs are positive: their bits order them
    for (uint32_t c = lane; c < 3 * kSplits; c += 32) {
        const uint32_t axis = c / kSplits, split = c - axis * kSplits;
        const float    axis_lo = axis == 0 ? clo[0] : (axis == 1 ? clo[1] : clo[2]);
        const float    axis_hi = axis == 0 ? chi[0] : (axis == 1 ? chi[1] : chi[2]);
        uint32_t       left = 0, right = 0, l[6], r[6];
        for (int d = 0; d < 6; ++d) {
            l[d] = r[d] = d < 3 ? kOrderedPosInf : kOrderedNegInf;
        }
        for (uint32_t k = 0; k < kBins; ++k) {
            const uint32_t  n = bin_count[axis * kBins + k];
            const uint32_t* v = bin_box + (axis * kBins + k) * 6;
            if (k <= split) {
                left += n;
                for (int d = 0; d < 6; ++d) {
                    l[d] = d < 3 ? min(l[d], v[d]) : max(l[d], v[d]);
                }
            } else {
                right += n;
                for (int d = 0; d < 6; ++d) {
                    r[d] = d < 3 ? min(r[d], v[d]) : max(r[d], v[d]);
                }
            }
        }
        if (axis_lo == axis_hi || left == 0 || right == 0) {
            continue;
        }
        float llo[3], lhi[3], rlo[3], rhi[3];
        for (int d = 0; d < 3; ++d) {
            llo[d] = o2f(l[d]), lhi[d] = o2f(l[3 + d]);
            rlo[d] = o2f(r[d]), rhi[d] = o2f(r[3 + d]);
        }
        const float cost = 1.0f + (scaled_area(llo, lhi, s) * static_cast<float>(left) +
                                   scaled_area(rlo, rhi, s) * static_cast<float>(right)) /
                                      parent;
        if (cost < static_cast<float>(count) && __float_as_uint(cost) < best_cost) {
            best_cost = __float_as_uint(cost);
            best      = c;
            best_left = left;
        }
    }
    const uint32_t cheapest = __reduce_min_sync(0xffffffffu, best_cost);
    if (cheapest == kNoCost) {
        return {-1, 0, 0};
    }
    const uint32_t first  = __reduce_min_sync(0xffffffffu, best_cost == cheapest ? best : kNoCost);
    const int      winner = __ffs(__ballot_sync(0xffffffffu, best_cost == cheapest && best == first)) - 1;
    return {static_cast<int>(first / kSplits), static_cast<int>(first % kSplits),
            __shfl_sync(0xffffffffu, best_left, winner)};
}

__device__ __forceinline__ void write_node(mr_bvh_node& n, const float* lo, const float* hi,
                                           uint32_t first, uint32_t right, uint32_t count) {
    for (int a = 0; a < 3; ++a) {
        n.minimum[a] = lo[a];
        n.maximum[a] = hi[a];
    }
    n.first = first;
    n.right = right;
    n.count = count;
}

// Pass 3: one warp per large task decides leaf or split and writes leaves.
__global__ void split_kernel(const Task* tasks, uint32_t count, const TaskBounds* bounds,
                             const TaskBins* bins, Split* splits, mr_bvh_node* nodes,
                             unsigned long long* leaves, unsigned* depth) {
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= count) {
        return;
    }
    const Task& task = tasks[t];
    float lo[3], hi[3], clo[3], chi[3];
    for (int a = 0; a < 3; ++a) {
        lo[a]  = o2f(bounds[t].v[a]);
        hi[a]  = o2f(bounds[t].v[3 + a]);
        clo[a] = o2f(bounds[t].v[6 + a]);
        chi[a] = o2f(bounds[t].v[9 + a]);
    }
    const uint32_t n = task.end - task.begin;
    Split          s{-1, 0, 0};
    if (n > kLeafSize && task.depth < kMaxDepth) {
        s = choose_split(lo, hi, clo, chi, n, &bins[t].count[0][0], &bins[t].box[0][0][0]);
    }
    if (threadIdx.x & 31) {
        return;
    }
    atomicMax(depth, task.depth);
    splits[t] = s;
    if (s.axis < 0) {
        write_node(nodes[task.node], lo, hi, task.begin, 0, n);
        atomicAdd(leaves, 1ull);
    } else {
        write_node(nodes[task.node], lo, hi, 0, 0, 0);  // children filled by emit_children
    }
}

// Pass 4: per chunk, how many primitives go left.
__global__ void count_left_kernel(const Chunk* chunks, const uint32_t* chunk_total, const uint32_t* order, const float4* pc,
                                  const TaskBounds* bounds, const Split* splits, uint32_t* left) {
    if (blockIdx.x >= *chunk_total) {
        return;
    }
    __shared__ uint32_t total;
    const Chunk ch = chunks[blockIdx.x];
    const Split s  = splits[ch.task];
    if (threadIdx.x == 0) {
        total = 0;
    }
    __syncthreads();
    if (s.axis >= 0) {
        const float lo = o2f(bounds[ch.task].v[6 + s.axis]);
        const float hi = o2f(bounds[ch.task].v[9 + s.axis]);
        uint32_t    mine = 0;
        for (uint32_t i = ch.begin + threadIdx.x; i < ch.end; i += blockDim.x) {
            const float4 c  = __ldg(pc + order[i]);
            const float  cc = s.axis == 0 ? c.x : (s.axis == 1 ? c.y : c.z);
            mine += bin_of(cc, lo, hi) <= s.bin ? 1u : 0u;
        }
        for (int o = 16; o > 0; o >>= 1) {
            mine += __shfl_xor_sync(0xffffffffu, mine, o);
        }
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&total, mine);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        left[blockIdx.x] = total;
    }
}

// Pass 5: stable scatter into `out` (chunks of split tasks only; others copy through).
__global__ void scatter_kernel(const Chunk* chunks, const uint32_t* chunk_total, const uint32_t* chunk_left_offset,
                               const uint32_t* task_first_chunk, const Task* tasks,
                               const uint32_t* order, const float4* pc, const TaskBounds* bounds,
                               const Split* splits, uint32_t* out) {
    if (blockIdx.x >= *chunk_total) {
        return;
    }
    const Chunk    ch   = chunks[blockIdx.x];
    const Split    s    = splits[ch.task];
    const Task     task = tasks[ch.task];
    if (s.axis < 0) {
        for (uint32_t i = ch.begin + threadIdx.x; i < ch.end; i += blockDim.x) {
            out[i] = order[i];
        }
        return;
    }
    const float    lo      = o2f(bounds[ch.task].v[6 + s.axis]);
    const float    hi      = o2f(bounds[ch.task].v[9 + s.axis]);
    const uint32_t base_l  = chunk_left_offset[blockIdx.x] - chunk_left_offset[task_first_chunk[ch.task]];
    const uint32_t before  = ch.begin - task.begin;  // primitives of this task in earlier chunks
    uint32_t       left_so_far = 0;
    for (uint32_t start = ch.begin; start < ch.end; start += blockDim.x) {
        const uint32_t i    = start + threadIdx.x;
        bool           goes = false;
        uint32_t       p    = 0;
        if (i < ch.end) {
            p = order[i];
            const float4 c  = __ldg(pc + p);
            const float  cc = s.axis == 0 ? c.x : (s.axis == 1 ? c.y : c.z);
            goes            = bin_of(cc, lo, hi) <= s.bin;
        }
        uint32_t total;
        const uint32_t rank = block_exclusive_scan(goes ? 1u : 0u, total);
        if (i < ch.end) {
            const uint32_t local = i - ch.begin;
            if (goes) {
                out[task.begin + base_l + left_so_far + rank] = p;
            } else {
                const uint32_t right_rank = (before + local) - (base_l + left_so_far + rank);
                out[task.begin + s.left_count + right_rank] = p;
            }
        }
        left_so_far += total;
    }
}

__global__ void copy_kernel(const Chunk* chunks, const uint32_t* chunk_total, const uint32_t* in, uint32_t* out) {
    if (blockIdx.x >= *chunk_total) {
        return;
    }
    const Chunk ch = chunks[blockIdx.x];
    for (uint32_t i = ch.begin + threadIdx.x; i < ch.end; i += blockDim.x) {
        out[i] = in[i];
    }
}

// What the host reads after a level.
struct LevelState {
    uint32_t large;  // tasks of the next level
    uint32_t small;  // small tasks so far
    uint32_t nodes;  // nodes so far
};

// Pass 6, one block: links the children of every split task and lists them as tasks of the next level
// or small tasks, left before right in task order (so tasks stay sorted by where they begin).
__global__ void __launch_bounds__(1024)
emit_children_kernel(const Task* tasks, uint32_t count, const Split* splits, mr_bvh_node* nodes,
                     Task* next_large, Task* small, LevelState* state) {
    uint32_t large_base = 0, small_base = state->small, node_base = state->nodes;
    for (uint32_t base = 0; base < count; base += blockDim.x) {
        const uint32_t t = base + threadIdx.x;
        Task           children[2];
        bool           split = t < count && splits[t].axis >= 0;
        uint32_t       large = 0;
        if (split) {
            const Task     task = tasks[t];
            const uint32_t mid  = task.begin + splits[t].left_count;
            children[0]         = {task.begin, mid, 0, task.depth + 1, 0};
            children[1]         = {mid, task.end, 0, task.depth + 1, 0};
            for (int c = 0; c < 2; ++c) {  // at depth 48 the split pass turns a large one into a leaf
                large += children[c].end - children[c].begin > kSmallTask ? 1u : 0u;
            }
        }
        uint32_t       total;  // children in the low half, large ones in the high half
        const uint32_t rank = block_exclusive_scan(split ? 2u | large << 16 : 0u, total);
        if (split) {
            const uint32_t first = node_base + (rank & 0xffffu);
            uint32_t       l = large_base + (rank >> 16), m = small_base + (rank & 0xffffu) - (rank >> 16);
            nodes[tasks[t].node].first = first;
            nodes[tasks[t].node].right = first + 1;
            for (uint32_t c = 0; c < 2; ++c) {
                children[c].node = first + c;
                if (children[c].end - children[c].begin > kSmallTask) {
                    next_large[l++] = children[c];
                } else {
                    small[m++] = children[c];
                }
            }
        }
        node_base += total & 0xffffu;
        large_base += total >> 16;
        small_base += (total & 0xffffu) - (total >> 16);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        *state = {large_base, small_base, node_base};
    }
}

// One block: the chunks of a level's tasks, and how many there are.
__global__ void __launch_bounds__(1024)
make_chunks_kernel(const Task* tasks, uint32_t count, Chunk* chunks, uint32_t* task_first_chunk,
                   uint32_t* chunk_total) {
    uint32_t running = 0;
    for (uint32_t base = 0; base < count; base += blockDim.x) {
        const uint32_t t = base + threadIdx.x;
        Task           task{};
        if (t < count) {
            task = tasks[t];
        }
        uint32_t total;
        uint32_t k = running + block_exclusive_scan((task.end - task.begin + kChunk - 1) / kChunk, total);
        if (t < count) {
            task_first_chunk[t] = k;
            for (uint32_t b = task.begin; b < task.end; b += kChunk, ++k) {
                chunks[k] = {t, b, min(b + kChunk, task.end)};
            }
        }
        running += total;
    }
    if (threadIdx.x == 0) {
        *chunk_total = running;
    }
}

// One block: exclusive scan of the chunks' left counts.
__global__ void __launch_bounds__(1024)
scan_left_kernel(const uint32_t* left, const uint32_t* chunk_total, uint32_t* offsets) {
    const uint32_t n       = *chunk_total;
    uint32_t       running = 0;
    for (uint32_t base = 0; base < n; base += blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        uint32_t       total;
        const uint32_t rank = block_exclusive_scan(i < n ? left[i] : 0u, total);
        if (i < n) {
            offsets[i] = running + rank;
        }
        running += total;
    }
}

// Small tasks in the order of where they begin: a mark per first primitive, scanned, is their rank.
__global__ void mark_small_kernel(const Task* small, uint32_t count, uint32_t* marks) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < count) {
        marks[small[t].begin] = 1;
    }
}

// Moves each small task to its rank, with the node indices its descendants may take (pre-order).
__global__ void sort_small_kernel(const Task* small, uint32_t count, const uint32_t* ranks, Task* sorted,
                                  uint32_t* sizes) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < count) {
        const Task     task = small[t];
        const uint32_t r    = ranks[task.begin];
        sorted[r]           = task;
        sizes[r]            = 2 * (task.end - task.begin) - 2;  // descendants of a subtree over n primitives
    }
}

// Small subtrees: one warp per task, depth-first in shared memory. Node indices are assigned in
// pre-order from the task's reserved range (the reference's emplacement order, bvh.cpp:104-105).
__global__ void __launch_bounds__(32 * kSmallWarps)
small_build_kernel(const Task* small, uint32_t count, const uint32_t* ranges, const LevelState* state,
                   uint32_t* order, const float4* plo, const float4* phi, const float4* pc,
                   mr_bvh_node* nodes, unsigned long long* leaves, unsigned* max_depth) {
    struct Entry {
        uint32_t begin, end, depth, parent_slot;  // parent_slot: node index*2 + side, or ~0
    };
    __shared__ uint32_t s_idx[kSmallWarps][kSmallTask];
    __shared__ uint32_t s_tmp[kSmallWarps][kSmallTask];
    __shared__ uint32_t s_count[kSmallWarps][3][kBins];
    __shared__ uint32_t s_box[kSmallWarps][3][kBins][6];
    __shared__ Entry    s_stack[kSmallWarps][kMaxDepth + 2];
    const int      warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t t    = blockIdx.x * kSmallWarps + warp;
    if (t >= count) {
        return;
    }
    const Task task = small[t];
    const uint32_t n = task.end - task.begin;
    for (uint32_t i = lane; i < n; i += 32) {
        s_idx[warp][i] = order[task.begin + i];
    }
    __syncwarp();
    uint32_t next_node = state->nodes + ranges[t];
    int      sp        = 0;
    if (lane == 0) {
        s_stack[warp][0] = {0, n, task.depth, kUnusedNode};
    }
    sp = 1;
    bool first = true;
    uint32_t local_leaves = 0, local_depth = 0;
    while (sp > 0) {
        __syncwarp();
        const Entry e = s_stack[warp][--sp];
        __syncwarp();
        const uint32_t node = first ? task.node : next_node++;
        first               = false;
        if (lane == 0 && e.parent_slot != kUnusedNode) {
            mr_bvh_node& parent = nodes[e.parent_slot >> 1];
            if (e.parent_slot & 1u) {
                parent.right = node;
            } else {
                parent.first = node;
            }
        }
        local_depth = max(local_depth, e.depth);
        // Bounds and centroid bounds (warp reduction).
        float v[12];
        for (int i = 0; i < 12; ++i) {
            v[i] = (i % 6) < 3 ? INFINITY : -INFINITY;
        }
        // The lane's first primitive stays in registers for the binning and the partition: most nodes
        // of a small task hold at most 32.
        uint32_t p0 = 0;
        float4   a0 = make_float4(0, 0, 0, 0), b0 = a0, c0 = a0;
        for (uint32_t i = e.begin + lane; i < e.end; i += 32) {
            const uint32_t p = s_idx[warp][i];
            const float4 a = __ldg(plo + p), b = __ldg(phi + p), c = __ldg(pc + p);
            if (i < e.begin + 32) {
                p0 = p, a0 = a, b0 = b, c0 = c;
            }
            v[0] = fminf(v[0], a.x), v[1] = fminf(v[1], a.y), v[2] = fminf(v[2], a.z);
            v[3] = fmaxf(v[3], b.x), v[4] = fmaxf(v[4], b.y), v[5] = fmaxf(v[5], b.z);
            v[6] = fminf(v[6], c.x), v[7] = fminf(v[7], c.y), v[8] = fminf(v[8], c.z);
            v[9] = fmaxf(v[9], c.x), v[10] = fmaxf(v[10], c.y), v[11] = fmaxf(v[11], c.z);
        }
        for (int i = 0; i < 12; ++i) {
            for (int o = 16; o > 0; o >>= 1) {
                const float y = __shfl_xor_sync(0xffffffffu, v[i], o);
                v[i]          = (i % 6) < 3 ? fminf(v[i], y) : fmaxf(v[i], y);
            }
        }
        const float* lo = v;
        const float* hi = v + 3;
        const float* clo = v + 6;
        const float* chi = v + 9;
        const uint32_t m = e.end - e.begin;
        Split s{-1, 0, 0};
        if (m > kLeafSize && e.depth < kMaxDepth) {
            for (int i = lane; i < 3 * kBins; i += 32) {
                (&s_count[warp][0][0])[i] = 0;
            }
            for (int i = lane; i < 3 * kBins * 6; i += 32) {
                (&s_box[warp][0][0][0])[i] = (i % 6) < 3 ? kOrderedPosInf : kOrderedNegInf;
            }
            __syncwarp();
            for (uint32_t i = e.begin + lane; i < e.end; i += 32) {
                float4 a = a0, b = b0, c = c0;
                if (i >= e.begin + 32) {
                    const uint32_t p = s_idx[warp][i];
                    a = __ldg(plo + p), b = __ldg(phi + p), c = __ldg(pc + p);
                }
                const float cc[3] = {c.x, c.y, c.z};
                for (int axis = 0; axis < 3; ++axis) {
                    if (chi[axis] == clo[axis]) {
                        continue;
                    }
                    const int k = bin_of(cc[axis], clo[axis], chi[axis]);
                    atomicAdd(&s_count[warp][axis][k], 1u);
                    atomicMin(&s_box[warp][axis][k][0], f2o(a.x));
                    atomicMin(&s_box[warp][axis][k][1], f2o(a.y));
                    atomicMin(&s_box[warp][axis][k][2], f2o(a.z));
                    atomicMax(&s_box[warp][axis][k][3], f2o(b.x));
                    atomicMax(&s_box[warp][axis][k][4], f2o(b.y));
                    atomicMax(&s_box[warp][axis][k][5], f2o(b.z));
                }
            }
            __syncwarp();
            s = choose_split(lo, hi, clo, chi, m, &s_count[warp][0][0], &s_box[warp][0][0][0]);
        }
        if (s.axis < 0) {
            if (lane == 0) {
                write_node(nodes[node], lo, hi, task.begin + e.begin, 0, m);
            }
            ++local_leaves;
            continue;
        }
        // Stable partition in shared memory.
        uint32_t left_so_far = 0;
        const float plo_axis = s.axis == 0 ? clo[0] : (s.axis == 1 ? clo[1] : clo[2]);
        const float phi_axis = s.axis == 0 ? chi[0] : (s.axis == 1 ? chi[1] : chi[2]);
        for (uint32_t start = e.begin; start < e.end; start += 32) {
            const uint32_t i    = start + lane;
            bool           goes = false;
            uint32_t       p    = 0;
            if (i < e.end) {
                const bool held = i < e.begin + 32;
                p               = held ? p0 : s_idx[warp][i];
                const float4 c  = held ? c0 : __ldg(pc + p);
                const float  cc = s.axis == 0 ? c.x : (s.axis == 1 ? c.y : c.z);
                goes            = bin_of(cc, plo_axis, phi_axis) <= s.bin;
            }
            const unsigned mask = __ballot_sync(0xffffffffu, goes);
            const uint32_t rank = __popc(mask & ((1u << lane) - 1u));
            if (i < e.end) {
                if (goes) {
                    s_tmp[warp][e.begin + left_so_far + rank] = p;
                } else {
                    const uint32_t right_rank = (i - e.begin) - (left_so_far + rank);
                    s_tmp[warp][e.begin + s.left_count + right_rank] = p;
                }
            }
            left_so_far += __popc(mask);
        }
        __syncwarp();
        for (uint32_t i = e.begin + lane; i < e.end; i += 32) {
            s_idx[warp][i] = s_tmp[warp][i];
        }
        if (lane == 0) {
            write_node(nodes[node], lo, hi, 0, 0, 0);
            const uint32_t mid = e.begin + s.left_count;
            s_stack[warp][sp]     = {mid, e.end, e.depth + 1, node * 2 + 1};
            s_stack[warp][sp + 1] = {e.begin, mid, e.depth + 1, node * 2};
        }
        sp += 2;
    }
    __syncwarp();
    for (uint32_t i = lane; i < n; i += 32) {
        order[task.begin + i] = s_idx[warp][i];
    }
    if (lane == 0) {
        atomicAdd(leaves, static_cast<unsigned long long>(local_leaves));
        atomicMax(max_depth, local_depth);
    }
}

__global__ void valid_flag_kernel(const mr_bvh_node* nodes, uint32_t count, uint32_t* flags) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) {
        flags[i] = nodes[i].count == kUnusedNode ? 0u : 1u;
    }
}

__global__ void compact_nodes_kernel(const mr_bvh_node* in, uint32_t count, const uint32_t* index,
                                     mr_bvh_node* out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count || in[i].count == kUnusedNode) {
        return;
    }
    mr_bvh_node n = in[i];
    if (n.count == 0) {
        n.first = index[n.first];
        n.right = index[n.right];
    }
    out[index[i]] = n;
}

__global__ void iota_kernel(uint32_t* out, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        out[i] = i;
    }
}

inline unsigned blocks_for(size_t n, unsigned per = 256) {
    return static_cast<unsigned>((n + per - 1) / per);
}

}  // namespace

BuildResult build_bvh_device(const float4* lo, const float4* hi, const float4* centroid,
                             uint32_t count, cudaStream_t stream) {
    BuildResult result;
    if (count == 0) {
        return result;
    }
    cudaEvent_t start, stop;
    MR_CUDA(cudaEventCreate(&start));
    MR_CUDA(cudaEventCreate(&stop));
    MR_CUDA(cudaEventRecord(start, stream));

    const size_t node_capacity = 2ull * count - 1;
    DeviceBuffer<mr_bvh_node> nodes;
    DeviceBuffer<uint32_t>    order, scratch_order;
    nodes.allocate(node_capacity);
    order.allocate(count);
    scratch_order.allocate(count);
    iota_kernel<<<blocks_for(count), 256, 0, stream>>>(order.ptr, count);

    // Task storage: a level never holds more than count / (kSmallTask + 1) large tasks, the
    // small list never more than count tasks... bounded by count.
    const size_t max_tasks  = std::max<size_t>(1, count / (kSmallTask / 2) + 2);
    const size_t max_chunks = count / kChunk + max_tasks + 1;
    DeviceBuffer<uint8_t> raw;
    const size_t bytes =
        2 * max_tasks * sizeof(Task) + max_tasks * (sizeof(TaskBounds) + sizeof(TaskBins) + sizeof(Split)) +
        max_tasks * sizeof(uint32_t) + max_chunks * (sizeof(Chunk) + 2 * sizeof(uint32_t)) +
        static_cast<size_t>(count) * (sizeof(Task) + 2 * sizeof(uint32_t)) + 64 * 16 +
        (scan_scratch_size(node_capacity) + 8) * sizeof(uint32_t);
    raw.allocate(bytes);
    uint8_t* cursor = raw.ptr;
    const auto take = [&](size_t b) {
        uint8_t* p = cursor;
        cursor += (b + 15) & ~size_t(15);
        return p;
    };
    Task*       tasks[2]      = {reinterpret_cast<Task*>(take(max_tasks * sizeof(Task))),
                                 reinterpret_cast<Task*>(take(max_tasks * sizeof(Task)))};
    TaskBounds* task_bounds   = reinterpret_cast<TaskBounds*>(take(max_tasks * sizeof(TaskBounds)));
    TaskBins*   task_bins     = reinterpret_cast<TaskBins*>(take(max_tasks * sizeof(TaskBins)));
    Split*      splits        = reinterpret_cast<Split*>(take(max_tasks * sizeof(Split)));
    uint32_t*   task_first    = reinterpret_cast<uint32_t*>(take(max_tasks * sizeof(uint32_t)));
    Chunk*      chunks        = reinterpret_cast<Chunk*>(take(max_chunks * sizeof(Chunk)));
    uint32_t*   chunk_left    = reinterpret_cast<uint32_t*>(take(max_chunks * sizeof(uint32_t)));
    uint32_t*   chunk_left_off = reinterpret_cast<uint32_t*>(take(max_chunks * sizeof(uint32_t)));
    Task*       small         = reinterpret_cast<Task*>(take(static_cast<size_t>(count) * sizeof(Task)));
    uint32_t*   small_sizes   = reinterpret_cast<uint32_t*>(take(static_cast<size_t>(count) * sizeof(uint32_t)));
    uint32_t*   small_ranges  = reinterpret_cast<uint32_t*>(take(static_cast<size_t>(count) * sizeof(uint32_t)));
    uint32_t*   counters      = reinterpret_cast<uint32_t*>(take(16 * sizeof(uint32_t)));
    unsigned long long* leaves = reinterpret_cast<unsigned long long*>(take(sizeof(unsigned long long)));
    uint32_t*   scratch       = reinterpret_cast<uint32_t*>(
        take((scan_scratch_size(node_capacity) + 8) * sizeof(uint32_t)));
    // counters: [0-2] LevelState, [3] chunks of the level, [4] maximum depth, [6] nodes in use
    LevelState* state       = reinterpret_cast<LevelState*>(counters);
    uint32_t*   chunk_total = counters + 3;
    MR_CUDA(cudaMemsetAsync(counters, 0, 16 * sizeof(uint32_t), stream));
    MR_CUDA(cudaMemsetAsync(leaves, 0, sizeof(unsigned long long), stream));
    // Every node index is unused (count kUnusedNode) until a node takes it.
    MR_CUDA(cudaMemsetAsync(nodes.ptr, 0xff, node_capacity * sizeof(mr_bvh_node), stream));

    uint32_t level_count = 0;
    uint32_t small_total = 0;
    // Root task (node 0): large unless it is small enough for one warp.
    const Task       root{0, count, 0, 0, 0};
    const LevelState first{0, count > kSmallTask ? 0u : 1u, 1};
    int              cur = 0;
    MR_CUDA(cudaMemcpyAsync(state, &first, sizeof(first), cudaMemcpyHostToDevice, stream));
    if (count > kSmallTask) {
        MR_CUDA(cudaMemcpyAsync(tasks[0], &root, sizeof(Task), cudaMemcpyHostToDevice, stream));
        level_count = 1;
    } else {
        MR_CUDA(cudaMemcpyAsync(small, &root, sizeof(Task), cudaMemcpyHostToDevice, stream));
        small_total = 1;
    }

    while (level_count > 0) {
        Task* level = tasks[cur];
        Task* next  = tasks[cur ^ 1];
        // At most this many chunks; the blocks beyond the level's own count leave at once.
        const unsigned grid = static_cast<unsigned>(std::min<size_t>(max_chunks, count / kChunk + level_count));
        make_chunks_kernel<<<1, 1024, 0, stream>>>(level, level_count, chunks, task_first, chunk_total);
        init_task_state<<<level_count, 128, 0, stream>>>(task_bounds, task_bins, level_count);
        reduce_bounds_kernel<<<grid, 256, 0, stream>>>(chunks, chunk_total, order.ptr, lo, hi, centroid, task_bounds);
        bin_kernel<<<grid, 256, 0, stream>>>(chunks, chunk_total, order.ptr, lo, hi, centroid, task_bounds, task_bins);
        split_kernel<<<blocks_for(level_count, 4), 128, 0, stream>>>(level, level_count, task_bounds, task_bins,
                                                                     splits, nodes.ptr, leaves, counters + 4);
        count_left_kernel<<<grid, 256, 0, stream>>>(chunks, chunk_total, order.ptr, centroid, task_bounds, splits,
                                                    chunk_left);
        scan_left_kernel<<<1, 1024, 0, stream>>>(chunk_left, chunk_total, chunk_left_off);
        scatter_kernel<<<grid, 256, 0, stream>>>(chunks, chunk_total, chunk_left_off, task_first, level, order.ptr,
                                                 centroid, task_bounds, splits, scratch_order.ptr);
        copy_kernel<<<grid, 256, 0, stream>>>(chunks, chunk_total, scratch_order.ptr, order.ptr);
        emit_children_kernel<<<1, 1024, 0, stream>>>(level, level_count, splits, nodes.ptr, next, small, state);
        MR_CUDA(cudaGetLastError());
        LevelState host{};
        MR_CUDA(cudaMemcpyAsync(&host, state, sizeof(host), cudaMemcpyDeviceToHost, stream));
        MR_CUDA(cudaStreamSynchronize(stream));
        level_count = host.large;
        small_total = host.small;
        cur ^= 1;
    }

    DeviceBuffer<Task> sorted;
    if (small_total > 0) {
        uint32_t* marks = scratch_order.ptr;
        sorted.allocate(small_total);
        MR_CUDA(cudaMemsetAsync(marks, 0, count * sizeof(uint32_t), stream));
        mark_small_kernel<<<blocks_for(small_total), 256, 0, stream>>>(small, small_total, marks);
        exclusive_scan(marks, marks, count, scratch, nullptr, stream);
        sort_small_kernel<<<blocks_for(small_total), 256, 0, stream>>>(small, small_total, marks, sorted.ptr,
                                                                        small_sizes);
        exclusive_scan(small_sizes, small_ranges, small_total, scratch, nullptr, stream);
        const unsigned blocks = (small_total + kSmallWarps - 1) / kSmallWarps;
        small_build_kernel<<<blocks, 32 * kSmallWarps, 0, stream>>>(sorted.ptr, small_total, small_ranges, state,
                                                                     order.ptr, lo, hi, centroid, nodes.ptr,
                                                                     leaves, counters + 4);
        MR_CUDA(cudaGetLastError());
    }

    // Squeeze out unused node indices.
    const uint32_t used_capacity = static_cast<uint32_t>(node_capacity);
    DeviceBuffer<uint32_t> valid, index;
    valid.allocate(used_capacity);
    index.allocate(used_capacity);
    valid_flag_kernel<<<blocks_for(used_capacity), 256, 0, stream>>>(nodes.ptr, used_capacity, valid.ptr);
    exclusive_scan(valid.ptr, index.ptr, used_capacity, scratch, counters + 6, stream);
    uint32_t           host_counters[16];
    unsigned long long host_leaves = 0;
    MR_CUDA(cudaMemcpyAsync(host_counters, counters, sizeof(host_counters), cudaMemcpyDeviceToHost, stream));
    MR_CUDA(cudaMemcpyAsync(&host_leaves, leaves, sizeof(host_leaves), cudaMemcpyDeviceToHost, stream));
    MR_CUDA(cudaStreamSynchronize(stream));
    const uint32_t compact    = host_counters[6];
    const uint32_t host_depth = host_counters[4];
    result.nodes.allocate(compact);
    compact_nodes_kernel<<<blocks_for(used_capacity), 256, 0, stream>>>(nodes.ptr, used_capacity, index.ptr,
                                                                         result.nodes.ptr);
    MR_CUDA(cudaGetLastError());
    MR_CUDA(cudaEventRecord(stop, stream));
    MR_CUDA(cudaStreamSynchronize(stream));
    float ms = 0;
    MR_CUDA(cudaEventElapsedTime(&ms, start, stop));
    cudaEventDestroy(start);
    cudaEventDestroy(stop);
    result.order         = std::move(order);
    result.node_count    = compact;
    result.leaves        = host_leaves;
    result.maximum_depth = host_depth;
    result.seconds       = ms * 1e-3;
    return result;
}

}  // namespace mr
