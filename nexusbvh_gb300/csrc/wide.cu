// wide.cu - stage 5: BVH2 -> compressed 8-wide BVH (Ylitie et al. 2017).
//
// Replaces BuildBVH8Kernel (NexusBVH/src/Cuda/WideConverter.cu:225-414).
// The reference launches one thread per work slot (n threads, one work
// item per BVH8 node and one per primitive) and keeps every CTA spinning in
// lock-step on __syncthreads_count until its slots are filled.  Here:
//   * only internal BVH8 nodes are work items; a parent writes its leaf
//     children's primitives into primIdx directly;
//   * a persistent grid (occupancy x SM count) whose lanes each hold one
//     work slot, claimed in increasing order, and poll it with bounded
//     relaxed loads, so no resident lane ever waits on a lane that has not
//     started;
//   * the allocation counters are bumped once per warp iteration with a
//     warp scan instead of once per node;
//   * each thread keeps the children it expands in a slot table in shared
//     memory (BVH2 index, children, box), so popping a child, the slot
//     assignment and the quantisation never reload a node (the reference
//     reloads each child box up to three times);
//   * in a whole-pipeline build the H-PLOC merges also write each internal
//     node's two children side by side (ChildPair, 64 bytes): the collapse
//     then opens a node with one aligned load of its record and reads no
//     BVH2 node at all (a leaf child's box is in its parent's record).
//     Measured on GB300 at 12.58M clustered triangles: BVH8 0.833 ->
//     0.553 ms, H-PLOC 2.16 -> 2.34 ms (the records' stores), build 3.91 ->
//     3.81 ms; the BVH8 kernel's time hardly depends on its occupancy (3 / 6
//     CTAs per SM: 0.898 / 0.833 ms), it follows the random node traffic;
//   * small greedy collapses, which are chains of levels, read every node's
//     children and slots from lists made beforehand, and auctions up to
//     2,000,000 primitives take eight lanes per item (takes_lists,
//     takes_groups).
// The decisions are the reference's:
//   * expansion always re-opens the highest-indexed inner child, the child
//     with the smaller area going to the re-opened position (:284-330);
//   * greedy slot assignment in child order, first strictly best slot
//     (GreedyAssignment, :104-153);
//   * node encoding with 8-bit quantised child boxes (CreateBVH8Node,
//     :156-206; CeilLog2/InvPow2, BuilderUtils.h:335-347);
//   * the one-primitive tree special case (CreateBVH8SingleLeaf, :209-222).
#include <algorithm>

#include "pipeline.h"

namespace nxb {
namespace {

constexpr int kThreads = 128;
constexpr float kQuantStep = 1.0f / 255.0f;  // 1/((1<<NQ)-1), NQ = 8
constexpr uint32_t kQueueSpinLimit = 1u << 20;
constexpr uint32_t kFallback = 0xFFFFFFFEu;  // auction_assign: use the greedy assignment
// Opening a BVH2 node needs its children; the opens of one item form a chain
// of dependent loads.  With prefetching on, loading a child that is itself
// internal also asks L2 for that child's two children (or, with child-pair
// records, for the child's record), so that the next open (or the child's
// own work item) finds them there.
constexpr bool kPrefetch = true;
// Words of a slot: BVH2 index, box (6 floats), and without child-pair records
// also left, right.
template <bool KIDS>
constexpr int kSlotWords = KIDS ? 7 : 9;
template <bool KIDS>
constexpr size_t kSlotSmem = (size_t)kThreads * 8 * kSlotWords<KIDS> * sizeof(uint32_t);

__device__ __forceinline__ uint32_t nib(uint32_t x, uint32_t i) { return (x >> (4 * i)) & 0xFu; }
__device__ __forceinline__ uint32_t popc_below(uint32_t m, uint32_t i) { return __popc(m & ((1u << i) - 1u)); }

__device__ __forceinline__ uint32_t ceil_log2_biased(float x) {
    const uint32_t ix = __float_as_uint(x);
    const uint32_t ex = (ix >> 23) & 0xFFu;
    return ex + ((ix & 0x7FFFFFu) != 0 ? 1u : 0u);
}
__device__ __forceinline__ float inv_pow2(uint8_t e) { return __uint_as_float((uint32_t)(254 - (int)e) << 23); }

// A BVH2 node, through the read-only path (the BVH2 was finished by an
// earlier kernel).
__device__ __forceinline__ Node2 load_node(const Node2* b2, uint32_t i) {
    const uint4* p = reinterpret_cast<const uint4*>(b2 + i);
    const uint4 a = __ldg(p), b = __ldg(p + 1);
    Node2 r;
    r.b.mn = make_float3(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z));
    r.b.mx = make_float3(__uint_as_float(a.w), __uint_as_float(b.x), __uint_as_float(b.y));
    r.left = b.z;
    r.right = b.w;
    return r;
}

// Per-thread table of the (up to 8) children being collected, in shared
// memory, word-interleaved across the CTA's threads (bank-conflict free).
template <bool KIDS>
struct SlotTable {
    uint32_t* base;
    __device__ uint32_t* at(uint32_t slot, uint32_t field) const {
        return base + (slot * kSlotWords<KIDS> + field) * kThreads + threadIdx.x;
    }
    __device__ void put(uint32_t slot, uint32_t idx, const Box& b) const {
        *at(slot, 0) = idx;
        *at(slot, 1) = __float_as_uint(b.mn.x);
        *at(slot, 2) = __float_as_uint(b.mn.y);
        *at(slot, 3) = __float_as_uint(b.mn.z);
        *at(slot, 4) = __float_as_uint(b.mx.x);
        *at(slot, 5) = __float_as_uint(b.mx.y);
        *at(slot, 6) = __float_as_uint(b.mx.z);
    }
    // without child-pair records, an inner child's own children too (with
    // them they come from the node's own record when it is opened)
    __device__ void put(uint32_t slot, uint32_t idx, const Node2& nd) const {
        put(slot, idx, nd.b);
        *at(slot, 7) = nd.left;
        *at(slot, 8) = nd.right;
    }
    __device__ uint32_t idx(uint32_t slot) const { return *at(slot, 0); }
    __device__ uint32_t left(uint32_t slot) const { return *at(slot, 7); }
    __device__ uint32_t right(uint32_t slot) const { return *at(slot, 8); }
    __device__ Box box(uint32_t slot) const {
        Box b;
        b.mn = make_float3(__uint_as_float(*at(slot, 1)), __uint_as_float(*at(slot, 2)), __uint_as_float(*at(slot, 3)));
        b.mx = make_float3(__uint_as_float(*at(slot, 4)), __uint_as_float(*at(slot, 5)), __uint_as_float(*at(slot, 6)));
        return b;
    }
};

// GetCost (WideConverter.cu:25-30): sign pattern of slot s applied to the
// parent-to-child centroid offset.
__device__ __forceinline__ float slot_cost(uint32_t s, float3 o) {
    return ((s >> 2) & 1 ? -1.0f : 1.0f) * o.x + ((s >> 1) & 1 ? -1.0f : 1.0f) * o.y + (s & 1 ? -1.0f : 1.0f) * o.z;
}

template <typename Boxes>
__device__ __forceinline__ uint32_t greedy_assign(float3 pc, const Boxes& boxes, uint32_t count) {
    uint32_t asg = kInvalid;
    for (uint32_t c = 0; c < count; ++c) {
        const Box cb = boxes.box(c);
        const float3 off = make_float3(pc.x - (cb.mx.x + cb.mn.x), pc.y - (cb.mx.y + cb.mn.y),
                                       pc.z - (cb.mx.z + cb.mn.z));
        float best = -3.402823466e+38f;
        uint32_t slot = 0xFu;
#pragma unroll
        for (uint32_t s = 0; s < 8; ++s) {
            if (nib(asg, s) != 0xFu) continue;
            const float cost = slot_cost(s, off);
            if (cost > best) {
                best = cost;
                slot = s;
            }
        }
        if (slot < 8) {
            asg &= ~(0xFu << (4 * slot));
            asg |= c << (4 * slot);
        }
    }
    return asg;
}

// AuctionAssignment (WideConverter.cu:50-102) over the cost table of the
// reference's USE_AUCTION branch (:337-358): child offsets from the parent
// centroid scaled so that the parent's largest extent maps to
// MAX_COST / 2 = 5, prices start at 0, epsilon runs from max(maxCost, 1/n)
// down to 1/n in steps of 1/THETA = 1/8, bidders are taken last-in first-out
// from a nibble stack.  The reference's loop has no bound and indexes
// prices[] with an invalid slot when no reward is finite; here bids are
// capped and both cases fall back to the greedy assignment.
constexpr uint32_t kAuctionBidLimit = 4096;

template <typename Boxes>
__device__ uint32_t auction_assign(const Box& pb, const Boxes& boxes, uint32_t count) {
    const float max_dim = fmaxf(pb.mx.x - pb.mn.x, fmaxf(pb.mx.y - pb.mn.y, pb.mx.z - pb.mn.z));
    float cost_scale = max_dim == 0.0f ? 0.0f : 10.0f / max_dim;
    cost_scale *= 0.5f;
    const float3 pc = make_float3(pb.mn.x + pb.mx.x, pb.mn.y + pb.mx.y, pb.mn.z + pb.mx.z);
    float3 off[8];
    float max_cost = -3.402823466e+38f;
    for (uint32_t c = 0; c < count; ++c) {
        const Box cb = boxes.box(c);
        off[c] = make_float3((pc.x - (cb.mn.x + cb.mx.x)) * cost_scale, (pc.y - (cb.mn.y + cb.mx.y)) * cost_scale,
                             (pc.z - (cb.mn.z + cb.mx.z)) * cost_scale);
        const float cost = fabsf(off[c].x) + fabsf(off[c].y) + fabsf(off[c].z);
        if (cost > max_cost) max_cost = cost;
    }
    float prices[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) prices[i] = 0.0f;
    const float threshold = 1.0f / (float)count;
    float epsilon = fmaxf(max_cost, threshold);
    uint32_t asg = kInvalid, bids = 0;
    while (epsilon >= threshold) {
        asg = kInvalid;
        uint32_t bidders = 0x76543210u, waiting = count;
        while (waiting > 0) {
            const uint32_t c = nib(bidders, --waiting);
            float win = -3.402823466e+38f, second = -3.402823466e+38f;
            uint32_t slot = 0xFu;
#pragma unroll
            for (uint32_t s = 0; s < 8; ++s) {
                const float reward = slot_cost(s, off[c]) - prices[s];
                if (reward > win) {
                    second = win;
                    win = reward;
                    slot = s;
                } else if (reward > second) {
                    second = reward;
                }
            }
            if (slot > 7 || ++bids > kAuctionBidLimit) return kFallback;
            float bump = (win - second) + epsilon;
#pragma unroll
            for (uint32_t s = 0; s < 8; ++s)
                if (s == slot) prices[s] += bump;
            const uint32_t prev = nib(asg, slot);
            asg = (asg & ~(0xFu << (4 * slot))) | (c << (4 * slot));
            if (prev != 0xFu) {
                bidders = (bidders & ~(0xFu << (4 * waiting))) | (prev << (4 * waiting));
                ++waiting;
            }
        }
        epsilon *= 0.125f;
    }
    return asg;
}

template <typename Boxes>
__device__ __forceinline__ void make_node8(uint32_t (&w)[20], const Box& bounds, const Boxes& boxes, uint32_t child_base,
                                           uint32_t prim_base, uint32_t asg, uint32_t inner, uint32_t leaf) {
#pragma unroll
    for (int i = 0; i < 20; ++i) w[i] = 0;
    const float3 diag = make_float3(bounds.mx.x - bounds.mn.x, bounds.mx.y - bounds.mn.y, bounds.mx.z - bounds.mn.z);
    const uint8_t ex = (uint8_t)ceil_log2_biased(diag.x * kQuantStep);
    const uint8_t ey = (uint8_t)ceil_log2_biased(diag.y * kQuantStep);
    const uint8_t ez = (uint8_t)ceil_log2_biased(diag.z * kQuantStep);
    const float3 inv = make_float3(inv_pow2(ex), inv_pow2(ey), inv_pow2(ez));
    w[0] = __float_as_uint(bounds.mn.x);
    w[1] = __float_as_uint(bounds.mn.y);
    w[2] = __float_as_uint(bounds.mn.z);
    uint32_t imask = 0;
    w[4] = child_base;
    w[5] = prim_base;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const uint32_t a = nib(asg, i);
        uint32_t meta;
        if (inner & (1u << i)) {
            imask |= 1u << i;
            meta = 0x20u | (24u + i);
        } else if (a != 0xFu) {
            meta = 0x20u | popc_below(leaf, i);
        } else {
            continue;
        }
        const uint32_t sh = 8u * (i & 3u);
        w[6 + (i >> 2)] |= meta << sh;
        const Box cb = boxes.box(a);
        const uint32_t qlx = (uint8_t)floorf((cb.mn.x - bounds.mn.x) * inv.x);
        const uint32_t qly = (uint8_t)floorf((cb.mn.y - bounds.mn.y) * inv.y);
        const uint32_t qlz = (uint8_t)floorf((cb.mn.z - bounds.mn.z) * inv.z);
        const uint32_t qhx = (uint8_t)ceilf((cb.mx.x - bounds.mn.x) * inv.x);
        const uint32_t qhy = (uint8_t)ceilf((cb.mx.y - bounds.mn.y) * inv.y);
        const uint32_t qhz = (uint8_t)ceilf((cb.mx.z - bounds.mn.z) * inv.z);
        w[8 + (i >> 2)] |= qlx << sh;
        w[10 + (i >> 2)] |= qly << sh;
        w[12 + (i >> 2)] |= qlz << sh;
        w[14 + (i >> 2)] |= qhx << sh;
        w[16 + (i >> 2)] |= qhy << sh;
        w[18 + (i >> 2)] |= qhz << sh;
    }
    w[3] = (uint32_t)ex | ((uint32_t)ey << 8) | ((uint32_t)ez << 16) | (imask << 24);
}
template <typename Boxes>
__device__ __forceinline__ void write_node8(Node8* dst, const Box& bounds, const Boxes& boxes, uint32_t child_base,
                                            uint32_t prim_base, uint32_t asg, uint32_t inner, uint32_t leaf) {
    uint32_t w[20];
    make_node8(w, bounds, boxes, child_base, prim_base, asg, inner, leaf);
    uint4* d = reinterpret_cast<uint4*>(dst);
#pragma unroll
    for (int k = 0; k < 5; ++k) d[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
}

struct LeafZero {
    const Node2* b2;
    __device__ Box box(uint32_t) const { return load_box(b2, 0); }
};

__global__ void bvh8_init_kernel(uint64_t* pairs, uint32_t n, uint32_t* ctr) {
    const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t i = i0; i < n; i += gridDim.x * blockDim.x) pairs[i] = bvh8_queue_slot(i, n);
    if (i0 == 0) bvh8_queue_counters(ctr);
}

// When the collapse is over: as many items have been finished as allocated.
// A warp counts what it finishes and adds it to the queue's count when it has
// nothing ready.  The two counts are never found equal early: an item's
// children are allocated by an atomic whose result the warp waits for (their
// slots follow from it), so that atomic has been performed before the item is
// counted; a warp that looks waits for the finished count before it reads the
// allocated one.  Fences in both places say the same in the memory model's
// words; they take 2 us of a small build's 35 to 50 (they wait for the nodes
// just written).  Counting allocated-but-unfinished items instead, in one
// word, either lets a child be finished before the word knows of it, or has
// every pass wait for a second atomic, on a line that idle warps poll
// (65,536 triangles 39 us instead of 37, 4.19M sphere 242 instead of 236).
constexpr uint32_t kEndCheck = 2;  // idle passes per look: 256,000 triangles 65.5 / 61.4 / 59.4 us at 1 / 2 / 4,
                                   // 16,411 boxes 34.8 / 34.8 / 36.8, 12.58M 517 / 512 / 516
struct FinishedItems {
    uint32_t* ctr;
    uint32_t held = 0, seen = 0;
    __device__ __forceinline__ void add(uint32_t finished) { held += finished; }
    __device__ __forceinline__ void settle() {
        if (held && lane_id() == 0) atomicAdd(ctr + kBvh8Finished, held);
        held = 0;
    }
    // Whether every item is finished.  The allocated count, which every pass
    // bumps, is only read again once as many items have been finished as had
    // been allocated at its last reading (reading it at every look: 12.58M
    // 512 -> 527 us).  Its address depends on the finished count, which is
    // below 2^31.
    __device__ __forceinline__ bool all() {
        const uint32_t finished = ld_relaxed_u32(ctr + kBvh8Finished);
        if (finished < seen) return false;
        seen = ld_relaxed_u32(ctr + kBvh8Alloc + (finished >> 31));
        return finished == seen;
    }
};

// Work items are the internal BVH8 nodes only: a parent writes the
// primitive of each leaf child straight into primIdx (it holds the leaf's
// node in its slot table), instead of queueing a work item per leaf as the
// reference does (one per primitive, each re-reading the leaf node).  Every
// inner child gets a fresh slot (breadth-first), so a slot is always written
// by an item in a lower slot.  Each lane holds one slot at a time and claims
// the next one (warp-aggregated: one atomic on the claim counter) once its
// item is done, whether or not a parent has allocated it yet, and polls it
// until its item arrives; a slot is only ever waited on by its own lane, so
// lanes that wait hold no other lane up.  The kernel ends when the count of
// allocated-but-unfinished items drops to zero (the slots still held then
// are never allocated).  Claiming without first reading the allocation
// counter keeps two loads per warp pass off the counters' cache lines,
// which every warp of the grid hits (measured on GB300: BVH8 0.858 ->
// 0.836 ms at 12.58M clustered triangles, 0.340 -> 0.320 ms at 4.19M).
// An item is (mesh-local BVH2 index << 32 | BVH8 index in `out`).  In the
// batched form (Seg = MeshBatch) the items of all meshes share the queue,
// the BVH8 index names the mesh, and nodes and leaves are counted per mesh
// in mesh_nodes / mesh_leaves.
template <typename Seg, bool AUCTION, bool KIDS>
__global__ __launch_bounds__(kThreads) void bvh8_kernel(const Node2* __restrict__ b2, Seg seg, Node8* out,
                                                        uint32_t cap, uint32_t slots, uint32_t* prim_idx,
                                                        uint64_t* pairs, uint32_t* ctr, uint32_t* mesh_nodes,
                                                        uint32_t* mesh_leaves, uint32_t* err,
                                                        const ChildPair* __restrict__ kids) {
    extern __shared__ uint32_t s_slots[];
    const SlotTable<KIDS> tab{s_slots};
    __shared__ uint4 s_stage[kThreads / 32][5 * 32];  // a warp's nodes, written out together
    uint4* stage = s_stage[threadIdx.x >> 5];
    const uint32_t lane = lane_id();
    if constexpr (!Seg::kBatch) {
        if (seg.n == 1) {
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                write_node8(out, load_box(b2, 0), LeafZero{b2}, 0, 0, 0xFFFFFFF0u, 0u, 1u);
                prim_idx[0] = 0;
                ctr[kBvh8Leaves] = 1;
                ctr[kBvh8Finished] = 1;
            }
            return;
        }
    }
    uint32_t slot = kInvalid;
    bool retired = false;
    uint32_t idle = 0;
    FinishedItems items{ctr};
    for (;;) {
        // lanes without a slot claim the next ones, in increasing order; a
        // slot past the queue's end is never allocated and retires the lane
        const bool want = !retired && slot == kInvalid;
        const uint32_t wmask = __ballot_sync(kFullMask, want);
        if (wmask) {
            const uint32_t leader = __ffs(wmask) - 1;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(ctr + kBvh8Claim, (uint32_t)__popc(wmask));
            base = __shfl_sync(kFullMask, base, leader);
            if (want) {
                const uint32_t claimed = base + __popc(wmask & lanemask_lt());
                if (claimed < slots && claimed >= base)
                    slot = claimed;
                else
                    retired = true;
            }
        }
        if (__all_sync(kFullMask, retired)) {
            items.settle();
            return;
        }
        uint64_t pr = 0;
        bool ready = false;
        if (slot != kInvalid) {
            pr = ld_relaxed_u64(pairs + slot);
            ready = (uint32_t)(pr >> 32) != kInvalid;
        }
        if (!__any_sync(kFullMask, ready)) {
            items.settle();
            if (++idle % kEndCheck == 0 && items.all()) return;
            if (idle > kQueueSpinLimit) {
                if (lane == 0) set_error(err, NXB_DEVERR_BVH8_QUEUE_TIMEOUT);
                return;
            }
            __nanosleep(min(32u << min(idle, 5u), 1024u));  // back off: idle warps poll the counters
            continue;
        }
        idle = 0;
        const uint32_t b2i = (uint32_t)(pr >> 32), b8i = (uint32_t)pr;
        // the item's mesh: its BVH2 nodes, BVH8 range and primitive range
        MeshSpan me{0, 0, 0};
        const Node2* mb2 = b2;
        uint32_t base8 = 0, cap8 = cap;
        bool internal = false;
        Node2 nd;
        ChildPair kp;  // KIDS: the item node's children
        if (ready) {
            if constexpr (Seg::kBatch) {
                me = seg.span(owner_of(seg.off8, 0, seg.meshes - 1, b8i));
                mb2 = b2 + 2ull * me.start;
                base8 = __ldg(seg.off8 + me.m);
                cap8 = __ldg(seg.off8 + me.m + 1) - base8;
            } else {
                me.count = seg.n;
            }
            const uint32_t node_limit = 2 * me.count - 1;
            if (Seg::kBatch && me.count <= 1) {
                // an empty mesh has no tree; a one-primitive mesh gets the
                // single-leaf node (CreateBVH8SingleLeaf, WideConverter.cu:209-222)
                if (me.count == 1) {
                    write_node8(out + b8i, load_box(mb2, 0), LeafZero{mb2}, 0, 0, 0xFFFFFFF0u, 0u, 1u);
                    prim_idx[me.start] = 0;
                    mesh_leaves[me.m] = 1;
                }
            } else if (b2i >= node_limit || b8i - base8 >= cap8) {
                set_error(err, NXB_DEVERR_BVH8_OVERFLOW);
            } else if constexpr (KIDS) {
                // an item is an internal node; its box is the union of its children's
                if (b2i < me.count) {
                    set_error(err, NXB_DEVERR_BVH8_OVERFLOW);
                } else {
                    kp = load_child_pair(kids + me.start + (b2i - me.count));
                    if (kp.li >= node_limit || kp.ri >= node_limit) {
                        set_error(err, NXB_DEVERR_BVH8_OVERFLOW);
                    } else {
                        nd.b = kp.l;
                        grow(nd.b, kp.r);
                        internal = true;
                    }
                }
            } else {
                nd = load_node(mb2, b2i);
                if (nd.left >= node_limit || nd.right >= node_limit)
                    set_error(err, NXB_DEVERR_BVH8_OVERFLOW);
                else
                    internal = true;
            }
            if (!internal) slot = kInvalid;  // done (or reported); the item counts as finished
        }
        const uint32_t node_limit = 2 * me.count - 1;
        uint32_t inner = 0, count = 0, asg = kInvalid, leaf = 0;
        if (internal) {
            // open BVH2 nodes top-down until 8 children or no inner child
            uint32_t l0, l1;
            if constexpr (KIDS) {
                l0 = kp.li;
                l1 = kp.ri;
            } else {
                l0 = nd.left;
                l1 = nd.right;
            }
            uint32_t msb = 0;
            while (true) {
                bool in0, in1, first;
                if constexpr (KIDS) {
                    // the children of the opened node and their boxes are in
                    // its record; an internal child's own record is the next
                    // load of its chain
                    in0 = l0 >= me.count;
                    in1 = l1 >= me.count;
                    if (kPrefetch) {
                        if (in0) prefetch_l2(kids + me.start + (l0 - me.count));
                        if (in1) prefetch_l2(kids + me.start + (l1 - me.count));
                    }
                    first = !(half_area(kp.l) < half_area(kp.r));
                    tab.put(msb, first ? l1 : l0, first ? kp.r : kp.l);
                    tab.put(count + 1, first ? l0 : l1, first ? kp.l : kp.r);
                } else {
                    const Node2 c0 = load_node(mb2, l0), c1 = load_node(mb2, l1);
                    if (kPrefetch) {
                        if (c0.left < node_limit && c0.right < node_limit) {
                            prefetch_l2(mb2 + c0.left);
                            prefetch_l2(mb2 + c0.right);
                        }
                        if (c1.left < node_limit && c1.right < node_limit) {
                            prefetch_l2(mb2 + c1.left);
                            prefetch_l2(mb2 + c1.right);
                        }
                    }
                    first = !(half_area(c0.b) < half_area(c1.b));
                    // the smaller-area child takes the re-opened position
                    tab.put(msb, first ? l1 : l0, first ? c1 : c0);
                    tab.put(count + 1, first ? l0 : l1, first ? c0 : c1);
                    in0 = c0.left != kInvalid;
                    in1 = c1.left != kInvalid;
                }
                if (first ? in1 : in0) inner |= 1u << msb;
                if (first ? in0 : in1) inner |= 1u << (count + 1);
                count += 2;
                if (inner == 0 || count == 8) break;
                msb = 31 - __clz(inner);
                inner &= ~(1u << msb);
                count--;
                if constexpr (KIDS) {
                    kp = load_child_pair(kids + me.start + (tab.idx(msb) - me.count));
                    l0 = kp.li;
                    l1 = kp.ri;
                } else {
                    l0 = tab.left(msb);
                    l1 = tab.right(msb);
                }
                if (l0 >= node_limit || l1 >= node_limit) {  // corrupt BVH2: report, stop expanding
                    set_error(err, NXB_DEVERR_BVH8_OVERFLOW);
                    inner |= 1u << msb;
                    count++;
                    break;
                }
            }
            const float3 pc = make_float3(nd.b.mn.x + nd.b.mx.x, nd.b.mn.y + nd.b.mx.y, nd.b.mn.z + nd.b.mx.z);
            if constexpr (AUCTION) {
                asg = auction_assign(nd.b, tab, count);
                if (asg == kFallback) asg = greedy_assign(pc, tab, count);
            } else {
                asg = greedy_assign(pc, tab, count);
            }
            uint32_t ninner = 0;
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const uint32_t a = nib(asg, i);
                if (a == 0xFu) continue;
                const uint32_t bit = (inner >> a) & 1u;
                ninner |= bit << i;
                leaf |= (bit ^ 1u) << i;
            }
            inner = ninner;
        }
        // warp-aggregated allocation of work slots (and, for one mesh, of
        // BVH8 nodes and leaves; a batch counts those per mesh)
        const uint32_t ic = internal ? (uint32_t)__popc(inner) : 0u;
        const uint32_t lc = internal ? count - ic : 0u;
        const uint32_t wc = ic;  // every inner child becomes a work item of its own
        const uint32_t packed = Seg::kBatch ? (wc << 20) : (ic | (lc << 10) | (wc << 20));
        uint32_t incl = packed;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        const uint32_t done = __popc(__ballot_sync(kFullMask, ready));
        // one 64-bit atomic: work slots (one mesh: = BVH8 nodes) low, leaves high
        uint64_t bases = 0;
        if (lane == 31) {
            const uint64_t tl = (incl >> 10) & 0x3FFu, tw = incl >> 20;
            if (tl | tw)
                bases = atomicAdd(reinterpret_cast<unsigned long long*>(ctr + kBvh8Alloc),
                                  (unsigned long long)((tl << 32) | tw));
        }
        bases = __shfl_sync(kFullMask, bases, 31);
        items.add(done);
        const uint32_t wb = (uint32_t)bases, nb = wb, lb = (uint32_t)(bases >> 32);
        bool wrote = false;
        __syncwarp();
        if (internal) {
            const uint32_t excl = incl - packed;
            uint32_t child_base, prim_base;
            if constexpr (Seg::kBatch) {
                child_base = ic ? atomicAdd(mesh_nodes + me.m, ic) : 0u;
                prim_base = lc ? atomicAdd(mesh_leaves + me.m, lc) : 0u;
            } else {
                child_base = nb + (excl & 0x3FFu);
                prim_base = lc ? lb + ((excl >> 10) & 0x3FFu) : 0u;
            }
            const uint32_t work_base = wb + (excl >> 20);
            if (child_base + ic > cap8 || work_base + wc > slots || prim_base + lc > me.count) {
                set_error(err, NXB_DEVERR_BVH8_OVERFLOW);
            } else {
#pragma unroll
                for (uint32_t i = 0; i < 8; ++i) {
                    const uint32_t a = nib(asg, i);
                    if ((inner >> i) & 1u) {
                        const uint32_t k = popc_below(inner, i);
                        const uint64_t pair = ((uint64_t)tab.idx(a) << 32) | (base8 + child_base + k);
                        st_relaxed_u64(pairs + work_base + k, pair);
                    } else if ((leaf >> i) & 1u) {
                        // leaf i of the BVH2 is primitive i (its node's right field)
                        prim_idx[me.start + prim_base + popc_below(leaf, i)] = KIDS ? tab.idx(a) : tab.right(a);
                    }
                }
                uint32_t w[20];
                make_node8(w, nd.b, tab, child_base, prim_base, asg, inner, leaf);
#pragma unroll
                for (int k = 0; k < 5; ++k)
                    stage[5 * lane + k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
                wrote = true;
            }
            slot = kInvalid;
        }
        // the warp's nodes (mostly neighbours in `out`, as its slots are) in
        // consecutive 16-byte units: written by their own lanes, 80 bytes
        // apart, they filled no memory sector at once (12.58M clustered
        // triangles 553 -> 528 us, 4.19M sphere 256 -> 242)
        const uint32_t wm = __ballot_sync(kFullMask, wrote);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const uint32_t u = 32 * k + lane, item = u / 5, part = u - 5 * item;
            const uint32_t to = __shfl_sync(kFullMask, b8i, item);
            if ((wm >> item) & 1u)
                reinterpret_cast<uint4*>(out + to)[part] = stage[u];
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------- groups
// The same collapse with eight lanes per work item: lane c of a group holds
// child c while the node is opened, and slot c when slots are assigned,
// quantised and written.  What bounds it is the chain of levels: without
// lists, per level 3.3 us of dependent record loads (up to eight), 1.3 us of
// assignment and allocation and 0.6 us until a child is seen; the write, 2 us
// in one lane, is 0.45 and off that chain.
constexpr uint32_t kGroupsPerCta = kThreads / 8;

// Monotone key of a cost for comparing as uint32; 0 for one that the
// sequential search would never take (not above -FLT_MAX, or NaN).  -0 and
// +0 compare equal, so both get +0's key.
__device__ __forceinline__ uint32_t cost_key(float cost) {
    const uint32_t u = __float_as_uint(cost);
    return cost > -3.402823466e+38f ? f2ord(u == 0x80000000u ? 0.0f : cost) : 0u;
}

// The first lane of the group with the largest key (a slot index), or 0xF.
__device__ __forceinline__ uint32_t group_first(uint32_t key, uint32_t best, uint32_t base) {
    const uint32_t m = __ballot_sync(kFullMask, key == best) >> base & 0xFFu;
    return best ? (uint32_t)__ffs(m) - 1u : 0xFu;
}

// greedy_assign over a group: lane s returns the child of slot s (0xF: none).
// Every lane rates the slots for its own child; then the children choose in
// order, lane c telling the others its first best slot among those left.
__device__ __forceinline__ uint32_t group_greedy(float3 off, uint32_t count, uint32_t sub) {
    uint32_t key[8];
#pragma unroll
    for (uint32_t s = 0; s < 8; ++s) key[s] = cost_key(slot_cost(s, off));
    uint32_t mine = 0xFu, taken = 0;
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) {
        uint32_t k[8], at[8];
#pragma unroll
        for (uint32_t s = 0; s < 8; ++s) {
            k[s] = (taken >> s) & 1u ? 0u : key[s];
            at[s] = s;
        }
#pragma unroll
        for (uint32_t w = 1; w < 8; w *= 2)
#pragma unroll
            for (uint32_t s = 0; s < 8; s += 2 * w) {
                const bool t = k[s + w] > k[s];
                k[s] = t ? k[s + w] : k[s];
                at[s] = t ? at[s + w] : at[s];
            }
        const uint32_t slot = __shfl_sync(kFullMask, k[0] ? at[0] : 0xFu, c, 8);
        if (c < count && slot < 8) {
            taken |= 1u << slot;
            if (sub == slot) mine = c;
        }
    }
    return mine;
}

// auction_assign over a group; kFallback in every lane where the sequential
// form falls back.
__device__ __forceinline__ uint32_t group_auction(const Box& pb, const Box& cb, uint32_t count, bool run, uint32_t sub,
                                                  uint32_t base, float (*costs)[8]) {
    const float max_dim = fmaxf(pb.mx.x - pb.mn.x, fmaxf(pb.mx.y - pb.mn.y, pb.mx.z - pb.mn.z));
    float cost_scale = max_dim == 0.0f ? 0.0f : 10.0f / max_dim;
    cost_scale *= 0.5f;
    const float3 pc = make_float3(pb.mn.x + pb.mx.x, pb.mn.y + pb.mx.y, pb.mn.z + pb.mx.z);
    const float3 off = make_float3((pc.x - (cb.mn.x + cb.mx.x)) * cost_scale, (pc.y - (cb.mn.y + cb.mx.y)) * cost_scale,
                                   (pc.z - (cb.mn.z + cb.mx.z)) * cost_scale);
    float max_cost = sub < count ? fmaxf(-3.402823466e+38f, fabsf(off.x) + fabsf(off.y) + fabsf(off.z))
                                 : -3.402823466e+38f;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) max_cost = fmaxf(max_cost, __shfl_xor_sync(kFullMask, max_cost, o));
    const float threshold = 1.0f / (float)count;
    float epsilon = fmaxf(max_cost, threshold);
    float price = 0.0f;
    uint32_t mine = 0xFu, bids = 0, bidders = 0x76543210u, waiting = count;
    run = run && epsilon >= threshold;
    // lane c rates the slots for its child once; a bid reads its row (1.05M
    // triangles 506 -> 492 us; it was three shuffles and the rating per bid)
    __syncwarp();
#pragma unroll
    for (uint32_t s = 0; s < 8; ++s) costs[sub][s] = slot_cost(s, off);
    __syncwarp();
    while (__any_sync(kFullMask, run)) {
        // one bid per group
        const uint32_t c = nib(bidders, (waiting - 1u) & 7u) & 7u;
        const uint32_t key = cost_key(costs[c][sub] - price);
        uint32_t first = key, second = 0;
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {
            const uint32_t f = __shfl_xor_sync(kFullMask, first, d), g = __shfl_xor_sync(kFullMask, second, d);
            second = max(min(first, f), max(second, g));
            first = max(first, f);
        }
        const uint32_t slot = group_first(key, first, base);
        const uint32_t prev = __shfl_sync(kFullMask, mine, slot, 8);
        if (run) {
            if (slot > 7 || ++bids > kAuctionBidLimit) {
                mine = kFallback;
                run = false;
            } else {
                --waiting;
                if (sub == slot) {
                    price += (ord2f(first) - (second ? ord2f(second) : -3.402823466e+38f)) + epsilon;
                    mine = c;
                }
                if (prev != 0xFu) {
                    bidders = (bidders & ~(0xFu << (4 * waiting))) | (prev << (4 * waiting));
                    ++waiting;
                }
                if (waiting == 0) {
                    epsilon *= 0.125f;
                    run = epsilon >= threshold;
                    if (run) {
                        mine = 0xFu;
                        bidders = 0x76543210u;
                        waiting = count;
                    }
                }
            }
        }
    }
    return mine;
}

// ---------------------------------------------------------------- lists
// What a BVH8 node made of BVH2 node X would hold, for every internal X: its
// up to eight children, by slot, as one thread per X opens and assigns them.
// It does not depend on X's place in the BVH8, so it needs no order, and it
// leaves the collapse a shorter chain per level: a level of opening and
// assigning takes 5.3 us (seven dependent record loads 2.9, the assignment
// 1.3), one that reads its list 1.7.  Four nodes of five are never made, so
// this pays as long as the chain is what a collapse takes (takes_lists).
// A list is three words of three 21-bit child indices (kNoChild: none); their
// top bits hold the number of children less one (0: the BVH2 is corrupt).
constexpr uint32_t kNoChild = (1u << 21) - 1u;

template <typename Seg>
__global__ __launch_bounds__(kThreads) void bvh8_lists_kernel(Seg seg, uint32_t records,
                                                              const ChildPair* kids, uint64_t* lists) {
    after_previous();
    extern __shared__ uint32_t s_slots[];
    const SlotTable<true> tab{s_slots};
    const uint32_t r = blockIdx.x * kThreads + threadIdx.x;
    if (r >= records) return;
    MeshSpan me{0, 0, 0};
    if constexpr (Seg::kBatch)
        me = seg.of_prim(r);
    else
        me.count = seg.n;
    if (r - me.start + 1 >= me.count) return;  // a mesh has a record less than primitives
    const uint32_t node_limit = 2 * me.count - 1;
    ChildPair kp = load_child_pair(kids + r);
    Box nb = kp.l;
    grow(nb, kp.r);
    uint32_t inner = 0, count = 0, msb = 0;
    bool ok = true;
    while (true) {
        ok = kp.li < node_limit && kp.ri < node_limit;
        if (!ok) break;
        const bool in0 = kp.li >= me.count, in1 = kp.ri >= me.count;
        const bool first = !(half_area(kp.l) < half_area(kp.r));
        // the smaller-area child takes the re-opened position
        tab.put(msb, first ? kp.ri : kp.li, first ? kp.r : kp.l);
        tab.put(count + 1, first ? kp.li : kp.ri, first ? kp.l : kp.r);
        if (first ? in1 : in0) inner |= 1u << msb;
        if (first ? in0 : in1) inner |= 1u << (count + 1);
        count += 2;
        if (inner == 0 || count == 8) break;
        msb = 31 - __clz(inner);
        inner &= ~(1u << msb);
        count--;
        kp = load_child_pair(kids + me.start + (tab.idx(msb) - me.count));
    }
    uint64_t w[3] = {~0ull >> 1, ~0ull >> 1, ~0ull >> 1};
    if (ok) {
        const uint32_t asg = greedy_assign(
            make_float3(nb.mn.x + nb.mx.x, nb.mn.y + nb.mx.y, nb.mn.z + nb.mx.z), tab, count);
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            const uint32_t a = nib(asg, i), sh = 21 * (i % 3);
            const uint32_t id = a == 0xFu ? kNoChild : tab.idx(a);
            w[i / 3] = (w[i / 3] & ~((uint64_t)kNoChild << sh)) | ((uint64_t)id << sh);
        }
#pragma unroll
        for (uint32_t k = 0; k < 3; ++k) w[k] |= (uint64_t)(((count - 1) >> k) & 1u) << 63;
    }
#pragma unroll
    for (uint32_t k = 0; k < 3; ++k) lists[3ull * r + k] = w[k];
}

template <typename Seg, bool AUCTION, bool LISTS>
__global__ __launch_bounds__(kThreads) void bvh8_group_kernel(const Node2* b2, Seg seg, Node8* out,
                                                              uint32_t cap, uint32_t slots, uint32_t* prim_idx,
                                                              uint64_t* pairs, uint32_t* ctr, uint32_t* mesh_nodes,
                                                              uint32_t* mesh_leaves, uint32_t* err,
                                                              const ChildPair* kids,
                                                              const uint64_t* lists) {
    after_previous();
    __shared__ __align__(8) uint8_t s_rows[kGroupsPerCta][64];  // meta and quantised bytes of a group's node
    __shared__ __align__(16) float s_costs[AUCTION ? kGroupsPerCta : 1][8][8];  // by child and slot
    const uint32_t lane = lane_id(), sub = lane & 7u, base = lane & 24u;
    uint8_t* rows = s_rows[threadIdx.x >> 3];
    if constexpr (!Seg::kBatch) {
        if (seg.n == 1) {
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                write_node8(out, load_box(b2, 0), LeafZero{b2}, 0, 0, 0xFFFFFFF0u, 0u, 1u);
                prim_idx[0] = 0;
                ctr[kBvh8Leaves] = 1;
                ctr[kBvh8Finished] = 1;
            }
            return;
        }
    }
    uint32_t slot = kInvalid;
    bool retired = false;
    uint32_t idle = 0;
    FinishedItems items{ctr};
    for (;;) {
        // groups without a slot claim the next ones (see bvh8_kernel)
        const bool want = !retired && slot == kInvalid;
        const uint32_t wmask = __ballot_sync(kFullMask, want && sub == 0);
        if (wmask) {
            uint32_t first = 0;
            if (lane == 0) first = atomicAdd(ctr + kBvh8Claim, (uint32_t)__popc(wmask));
            first = __shfl_sync(kFullMask, first, 0);
            if (want) {
                const uint32_t claimed = first + __popc(wmask & ((1u << base) - 1u));
                if (claimed < slots && claimed >= first)
                    slot = claimed;
                else
                    retired = true;
            }
        }
        if (__all_sync(kFullMask, retired)) {
            items.settle();
            return;
        }
        uint64_t pr = ~0ull;
        if (slot != kInvalid) pr = ld_relaxed_u64(pairs + slot);
        pr = __shfl_sync(kFullMask, pr, 0, 8);  // one lane's view for the whole group
        const bool ready = (uint32_t)(pr >> 32) != kInvalid;
        if (!__any_sync(kFullMask, ready)) {
            items.settle();
            if (++idle % kEndCheck == 0 && items.all()) return;
            if (idle > kQueueSpinLimit) {
                if (lane == 0) set_error(err, NXB_DEVERR_BVH8_QUEUE_TIMEOUT);
                return;
            }
            __nanosleep(min(32u << min(idle, 5u), 128u));
            continue;
        }
        idle = 0;
        const uint32_t b2i = (uint32_t)(pr >> 32), b8i = (uint32_t)pr;
        MeshSpan me{0, 0, 0};
        const Node2* mb2 = b2;
        uint32_t base8 = 0, cap8 = cap;
        bool internal = false;
        ChildPair kp;
        Box nb;  // the node's box
        uint64_t list = 0;
        if (ready) {
            if constexpr (Seg::kBatch) {
                me = seg.span(owner_of(seg.off8, 0, seg.meshes - 1, b8i));
                mb2 = b2 + 2ull * me.start;
                base8 = __ldg(seg.off8 + me.m);
                cap8 = __ldg(seg.off8 + me.m + 1) - base8;
            } else {
                me.count = seg.n;
            }
            if (Seg::kBatch && me.count <= 1) {
                if (me.count == 1 && sub == 0) {
                    write_node8(out + b8i, load_box(mb2, 0), LeafZero{mb2}, 0, 0, 0xFFFFFFF0u, 0u, 1u);
                    prim_idx[me.start] = 0;
                    mesh_leaves[me.m] = 1;
                }
            } else if (b2i >= 2 * me.count - 1 || b8i - base8 >= cap8 || b2i < me.count) {
                if (sub == 0) set_error(err, NXB_DEVERR_BVH8_OVERFLOW);
            } else {
                const uint32_t record = me.start + (b2i - me.count);
                if constexpr (LISTS) {
                    list = lists[3ull * record + sub / 3];
                    nb = load_box(mb2, b2i);
                    internal = true;
                } else {
                    kp = load_child_pair(kids + record);
                    internal = kp.li < 2 * me.count - 1 && kp.ri < 2 * me.count - 1;
                    if (!internal && sub == 0) set_error(err, NXB_DEVERR_BVH8_OVERFLOW);
                }
            }
            if (!internal) slot = kInvalid;  // done (or reported); the item counts as finished
        }
        uint32_t count = 0, child;  // of the node; in slot `sub`
        bool used, is_inner;
        Box qb;  // the child's box
        if (!internal) nb.mn = nb.mx = make_float3(0.f, 0.f, 0.f);
        if constexpr (LISTS) {
            const uint32_t bits = __ballot_sync(kFullMask, list >> 63) >> base;
            count = 1u + ((bits & 1u) | (bits >> 2 & 2u) | (bits >> 4 & 4u));
            if (internal && count == 1) {
                if (sub == 0) set_error(err, NXB_DEVERR_BVH8_OVERFLOW);
                internal = false;
                slot = kInvalid;
            }
            child = (uint32_t)(list >> (21 * (sub % 3))) & kNoChild;
            used = internal && child != kNoChild;
            is_inner = used && child >= me.count;
            qb = nb;
            if (used) qb = load_box(mb2, child);
        } else {
            const uint32_t node_limit = 2 * me.count - 1;
            Box cb;  // this lane's child's box
            cb.mn = cb.mx = make_float3(0.f, 0.f, 0.f);
            uint32_t idx = 0, inner = 0, msb = 0;
            if (internal) {
                nb = kp.l;
                grow(nb, kp.r);
            }
            // open BVH2 nodes top-down until 8 children or no inner child; every
            // lane of the group has the record, the two lanes concerned keep a child
            bool open = internal;
            while (__any_sync(kFullMask, open)) {
                if (open) {
                    const bool in0 = kp.li >= me.count, in1 = kp.ri >= me.count;
                    const bool first = !(half_area(kp.l) < half_area(kp.r));
                    // the smaller-area child takes the re-opened position
                    const bool low = sub == msb, high = sub == count + 1;
                    if (low || high) {
                        const bool right = low == first;
                        cb = right ? kp.r : kp.l;
                        idx = right ? kp.ri : kp.li;
                        if (idx >= me.count) prefetch_l2(kids + me.start + (idx - me.count));
                    }
                    if (first ? in1 : in0) inner |= 1u << msb;
                    if (first ? in0 : in1) inner |= 1u << (count + 1);
                    count += 2;
                    if (inner == 0 || count == 8) {
                        open = false;
                    } else {
                        msb = 31 - __clz(inner);
                        inner &= ~(1u << msb);
                        count--;
                    }
                }
                const uint32_t next = __shfl_sync(kFullMask, idx, msb, 8);
                if (open) {
                    kp = load_child_pair(kids + me.start + (next - me.count));
                    if (kp.li >= node_limit || kp.ri >= node_limit) {  // corrupt BVH2: report, stop expanding
                        if (sub == 0) set_error(err, NXB_DEVERR_BVH8_OVERFLOW);
                        inner |= 1u << msb;
                        count++;
                        open = false;
                    }
                }
            }
            const float3 pc = make_float3(nb.mn.x + nb.mx.x, nb.mn.y + nb.mx.y, nb.mn.z + nb.mx.z);
            const float3 off = make_float3(pc.x - (cb.mx.x + cb.mn.x), pc.y - (cb.mx.y + cb.mn.y),
                                           pc.z - (cb.mx.z + cb.mn.z));
            uint32_t mine;  // the child of slot `sub`
            if constexpr (AUCTION) {
                mine = group_auction(nb, cb, max(count, 1u), internal, sub, base, s_costs[threadIdx.x >> 3]);
                const bool failed = mine == kFallback;
                if (__any_sync(kFullMask, failed)) {
                    const uint32_t g = group_greedy(off, count, sub);
                    if (failed) mine = g;
                }
            } else {
                mine = group_greedy(off, count, sub);
            }
            used = internal && mine != 0xFu;
            is_inner = used && ((inner >> mine) & 1u);
            child = __shfl_sync(kFullMask, idx, mine, 8);
            qb.mn.x = __shfl_sync(kFullMask, cb.mn.x, mine, 8);
            qb.mn.y = __shfl_sync(kFullMask, cb.mn.y, mine, 8);
            qb.mn.z = __shfl_sync(kFullMask, cb.mn.z, mine, 8);
            qb.mx.x = __shfl_sync(kFullMask, cb.mx.x, mine, 8);
            qb.mx.y = __shfl_sync(kFullMask, cb.mx.y, mine, 8);
            qb.mx.z = __shfl_sync(kFullMask, cb.mx.z, mine, 8);
        }
        const uint32_t imask = __ballot_sync(kFullMask, is_inner) >> base & 0xFFu;
        const uint32_t lmask = __ballot_sync(kFullMask, used && !is_inner) >> base & 0xFFu;
        // allocation of work slots (one mesh: = BVH8 nodes) and leaves, one
        // atomic for the warp's four groups
        const uint32_t ic = internal ? (uint32_t)__popc(imask) : 0u;
        const uint32_t lc = internal ? count - (uint32_t)__popc(imask) : 0u;
        const uint32_t packed = ic | (lc << 16);
        uint32_t excl = 0, total = 0;
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            const uint32_t v = __shfl_sync(kFullMask, packed, 8 * q);
            if (8 * q < base) excl += v;
            total += v;
        }
        const uint32_t done = __popc(__ballot_sync(kFullMask, ready && sub == 0));
        const uint32_t new_items = total & 0xFFFFu;
        const uint64_t tl = Seg::kBatch ? 0u : total >> 16;
        uint64_t bases = 0;
        if (lane == 0 && (tl | new_items))
            bases = atomicAdd(reinterpret_cast<unsigned long long*>(ctr + kBvh8Alloc),
                              (unsigned long long)((tl << 32) | new_items));
        uint32_t child_base = 0, prim_base = 0;
        if (Seg::kBatch && internal && sub == 0) {
            child_base = ic ? atomicAdd(mesh_nodes + me.m, ic) : 0u;
            prim_base = lc ? atomicAdd(mesh_leaves + me.m, lc) : 0u;
        }
        bases = __shfl_sync(kFullMask, bases, 0);
        items.add(done);
        const uint32_t work_base = (uint32_t)bases + (excl & 0xFFFFu);
        if constexpr (Seg::kBatch) {
            child_base = __shfl_sync(kFullMask, child_base, 0, 8);
            prim_base = __shfl_sync(kFullMask, prim_base, 0, 8);
        } else {
            child_base = work_base;
            prim_base = lc ? (uint32_t)(bases >> 32) + (excl >> 16) : 0u;
        }
        bool write = internal;
        if (write && (child_base + ic > cap8 || work_base + ic > slots || prim_base + lc > me.count)) {
            if (sub == 0) set_error(err, NXB_DEVERR_BVH8_OVERFLOW);
            write = false;
        }
        if (write) {
            if (is_inner) {
                const uint32_t k = popc_below(imask, sub);
                st_relaxed_u64(pairs + work_base + k, ((uint64_t)child << 32) | (base8 + child_base + k));
            } else if (used) {
                prim_idx[me.start + prim_base + popc_below(lmask, sub)] = child;  // leaf i is primitive i
            }
        }
        if (internal) slot = kInvalid;
        // the node: lane s quantises slot s (write_node8)
        if (__any_sync(kFullMask, write)) {
            const uint8_t ex = (uint8_t)ceil_log2_biased((nb.mx.x - nb.mn.x) * kQuantStep);
            const uint8_t ey = (uint8_t)ceil_log2_biased((nb.mx.y - nb.mn.y) * kQuantStep);
            const uint8_t ez = (uint8_t)ceil_log2_biased((nb.mx.z - nb.mn.z) * kQuantStep);
            const float3 inv = make_float3(inv_pow2(ex), inv_pow2(ey), inv_pow2(ez));
            rows[sub] = (uint8_t)(!used ? 0u : is_inner ? 0x20u | (24u + sub) : 0x20u | popc_below(lmask, sub));
            rows[8 + sub] = used ? (uint8_t)floorf((qb.mn.x - nb.mn.x) * inv.x) : (uint8_t)0;
            rows[16 + sub] = used ? (uint8_t)floorf((qb.mn.y - nb.mn.y) * inv.y) : (uint8_t)0;
            rows[24 + sub] = used ? (uint8_t)floorf((qb.mn.z - nb.mn.z) * inv.z) : (uint8_t)0;
            rows[32 + sub] = used ? (uint8_t)ceilf((qb.mx.x - nb.mn.x) * inv.x) : (uint8_t)0;
            rows[40 + sub] = used ? (uint8_t)ceilf((qb.mx.y - nb.mn.y) * inv.y) : (uint8_t)0;
            rows[48 + sub] = used ? (uint8_t)ceilf((qb.mx.z - nb.mn.z) * inv.z) : (uint8_t)0;
            __syncwarp();
            if (write) {
                uint2* d = reinterpret_cast<uint2*>(out + b8i);
                if (sub == 0) d[0] = make_uint2(__float_as_uint(nb.mn.x), __float_as_uint(nb.mn.y));
                if (sub == 1)
                    d[1] = make_uint2(__float_as_uint(nb.mn.z), (uint32_t)ex | ((uint32_t)ey << 8) |
                                                                   ((uint32_t)ez << 16) | (imask << 24));
                if (sub == 2) d[2] = make_uint2(child_base, prim_base);
                if (sub < 7) d[3 + sub] = reinterpret_cast<const uint2*>(rows)[sub];
            }
            __syncwarp();
        }
    }
}

template <typename Seg, bool AUCTION, bool LISTS = false>
cudaError_t launch_group(const Node2* bvh2, Seg seg, uint32_t items, Node8* out, uint32_t cap, uint32_t slots,
                         uint32_t* prim_idx, uint64_t* pairs, uint32_t* ctr, uint32_t* mesh_nodes,
                         uint32_t* mesh_leaves, uint32_t* err, cudaStream_t s, const ChildPair* kids,
                         uint64_t* lists = nullptr) {
    if constexpr (LISTS) {
        const cudaError_t e = once_per_device([] {
            return cudaFuncSetAttribute(bvh8_lists_kernel<Seg>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                        cudaSharedmemCarveoutMaxShared);
        });
        if (e) return e;
        const uint32_t ctas = (items + kThreads - 1) / kThreads;
        if constexpr (Seg::kBatch) {
            bvh8_lists_kernel<Seg><<<ctas, kThreads, (kSlotSmem<true>), s>>>(seg, items, kids, lists);
        } else {
            const cudaError_t le =
                launch_after(items, bvh8_lists_kernel<Seg>, ctas, kThreads, kSlotSmem<true>, s, seg, items, kids, lists);
            if (le) return le;
        }
    }
    int per_sm = resident_ctas<bvh8_group_kernel<Seg, AUCTION, LISTS>>(kThreads, 0);
    // Groups that wait poll the finished count, and too many of them saturate
    // its L2 line.  With lists, a group per 16 primitives and, above 4,096
    // groups, per 32: 1,021 triangles 27 us (33 at 32), 65,536 39 (47 at 8),
    // 128,000 49 (53 at 16), 256,000 68 (70); at 8 CTAs per SM instead of 4,
    // 256,000 take 109 and 512,000 137 (98).  Auctions keep their groups
    // busy: 1.05M triangles 631 us at 4, 512 at 8.
    if (!AUCTION) per_sm = std::min(per_sm, 4);
    uint32_t groups = (items + 15) / 16;
    if (LISTS) groups = std::max(std::min(groups, 4096u), (items + 31) / 32);
    const uint32_t want = (groups + kGroupsPerCta - 1) / kGroupsPerCta;
    const uint32_t grid = std::max(1u, std::min(want, (uint32_t)(device_info().sms * per_sm)));
    if constexpr (LISTS && !Seg::kBatch)
        return launch_after(items, bvh8_group_kernel<Seg, AUCTION, LISTS>, grid, kThreads, 0, s, bvh2, seg, out, cap, slots,
                            prim_idx, pairs, ctr, mesh_nodes, mesh_leaves, err, kids, lists);
    bvh8_group_kernel<Seg, AUCTION, LISTS><<<grid, kThreads, 0, s>>>(bvh2, seg, out, cap, slots, prim_idx, pairs, ctr,
                                                                     mesh_nodes, mesh_leaves, err, kids, lists);
    return cudaGetLastError();
}

// Which form of the collapse a build with child-pair records takes.  Small
// greedy collapses are a chain of levels (12 at 65,536 triangles), which
// lists make shortest; large ones are bound by random memory traffic, where
// one lane per item keeps eight times the items in flight, and where the
// lists of nodes never made cost more than the chain.  Measured (one lane / a
// group per item / a group with lists): 1,021 soup triangles - / 45 / 27 us,
// 16,411 clustered boxes 98 / 76 / 37, 65,536 soup 100 / 70 / 39, 256,000
// 129 / 100 / 72, 512,000 143 / 131 / 98, 1.0M 154 / 184 / 160, 1.0M
// clustered 180 / - / 166, 4.19M sphere 237 / 473 / -.  Groups of a batch
// that overlaps its stages have no room for lists.  An auction is a long
// sequential search per item, eight times shorter in a group, so it takes the
// groups further, up to where the items in flight count (group / one lane):
// 100,000 soup triangles 256 / 457 us, 1.0M 510 / 674, 2.0M 756 / 748, 3.0M
// 1,026 / 817, 12.58M 3,565 / 1,655; 2.0M clustered 746 / 776.  The lists would
// take it for every node.
constexpr uint32_t kListMaxPrims = 800000;  // at most 2^20: a list holds 21-bit indices
constexpr uint32_t kGroupMaxPrims = 600000;
constexpr uint32_t kAuctionGroupMaxPrims = 2000000;
inline bool takes_lists(uint32_t prims, bool auction) { return !auction && prims <= kListMaxPrims; }
inline bool takes_groups(uint32_t prims, bool auction) {
    return prims <= (auction ? kAuctionGroupMaxPrims : kGroupMaxPrims);
}

template <typename Seg, bool AUCTION, bool KIDS>
cudaError_t configure_smem() {
    return once_per_device([] {
        return cudaFuncSetAttribute(bvh8_kernel<Seg, AUCTION, KIDS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kSlotSmem<KIDS>);
    });
}

template <typename Seg, bool AUCTION, bool KIDS>
uint32_t persistent_grid(uint32_t items) {
    const int per_sm = resident_ctas<bvh8_kernel<Seg, AUCTION, KIDS>>(kThreads, kSlotSmem<KIDS>);
    const uint32_t want = (items + kThreads - 1) / kThreads;
    return std::max(1u, std::min(want, (uint32_t)(device_info().sms * per_sm)));
}

template <typename Seg, bool AUCTION, bool KIDS = false>
cudaError_t launch_wide(const Node2* bvh2, Seg seg, uint32_t items, Node8* out, uint32_t cap, uint32_t slots,
                        uint32_t* prim_idx, uint64_t* pairs, uint32_t* ctr, uint32_t* mesh_nodes,
                        uint32_t* mesh_leaves, uint32_t* err, cudaStream_t s, const ChildPair* kids = nullptr) {
    cudaError_t e = configure_smem<Seg, AUCTION, KIDS>();
    if (e) return e;
    bvh8_kernel<Seg, AUCTION, KIDS><<<persistent_grid<Seg, AUCTION, KIDS>(items), kThreads, (kSlotSmem<KIDS>), s>>>(
        bvh2, seg, out, cap, slots, prim_idx, pairs, ctr, mesh_nodes, mesh_leaves, err, kids);
    return cudaGetLastError();
}

}  // namespace

// Bounded-wait check: a two-primitive BVH2 whose work queue is never seeded,
// so every slot poll expires.  Returns the error word.
cudaError_t run_bvh8_stall_probe(uint32_t* err_out) {
    const uint32_t n = 2;
    unsigned char* buf = nullptr;
    const size_t bytes = 4 * (kBvh8CtrWords + 32) + 3 * sizeof(Node2) + 2 * sizeof(Node8) + 8 * n + 4 * n;
    cudaError_t e = configure_smem<SingleMesh, false, false>();
    if (!e) e = cudaMalloc(&buf, bytes);
    if (e) return e;
    uint32_t* ctr = (uint32_t*)buf;  // 256-byte aligned
    uint32_t* err = ctr + kBvh8CtrWords;
    Node2* b2 = (Node2*)(buf + 4 * (kBvh8CtrWords + 32));
    Node8* out = (Node8*)(b2 + 3);
    uint64_t* pairs = (uint64_t*)(out + 2);
    uint32_t* prim = (uint32_t*)(pairs + n);
    e = cudaMemset(buf, 0, bytes);
    if (!e) e = cudaMemset(pairs, 0xFF, 8 * n);
    uint32_t c[kBvh8CtrWords] = {};
    c[kBvh8Alloc] = 1;  // slot 0 is allocated, but its pair is never written
    if (!e) e = cudaMemcpy(ctr, c, sizeof(c), cudaMemcpyHostToDevice);
    if (!e) {
        bvh8_kernel<SingleMesh, false, false><<<1, kThreads, (kSlotSmem<false>)>>>(b2, SingleMesh{n}, out, 2, n, prim, pairs,
                                                                          ctr, nullptr, nullptr, err, nullptr);
        e = cudaGetLastError();
    }
    if (!e) e = cudaMemcpy(err_out, err, 4, cudaMemcpyDeviceToHost);
    cudaFree(buf);
    return e;
}

cudaError_t launch_bvh8_init(uint64_t* pairs, uint32_t n, uint32_t* ctr, cudaStream_t s) {
    uint32_t grid = std::min<uint32_t>((n + 255) / 256, (uint32_t)device_info().sms * 8);
    bvh8_init_kernel<<<grid, 256, 0, s>>>(pairs, n, ctr);
    return cudaGetLastError();
}

uint32_t bvh8_launches(uint32_t prims, bool auction, bool lists) { return lists && takes_lists(prims, auction) ? 2 : 1; }

cudaError_t launch_bvh8(const Node2* bvh2, uint32_t n, Node8* out, uint32_t cap, uint32_t* prim_idx, uint64_t* pairs,
                        uint32_t* ctr, uint32_t* err, bool auction, cudaStream_t s, const ChildPair* child_pairs,
                        uint64_t* lists) {
    const SingleMesh seg{n};
    if (child_pairs && lists && takes_lists(n, auction))
        return launch_group<SingleMesh, false, true>(bvh2, seg, n, out, cap, n, prim_idx, pairs, ctr, nullptr,
                                                     nullptr, err, s, child_pairs, lists);
    if (child_pairs && auction && takes_groups(n, true))
        return launch_group<SingleMesh, true>(bvh2, seg, n, out, cap, n, prim_idx, pairs, ctr, nullptr, nullptr, err,
                                              s, child_pairs);
    if (child_pairs && auction)
        return launch_wide<SingleMesh, true, true>(bvh2, seg, n, out, cap, n, prim_idx, pairs, ctr, nullptr, nullptr,
                                                   err, s, child_pairs);
    if (child_pairs)
        return launch_wide<SingleMesh, false, true>(bvh2, seg, n, out, cap, n, prim_idx, pairs, ctr, nullptr,
                                                    nullptr, err, s, child_pairs);
    if (auction)
        return launch_wide<SingleMesh, true>(bvh2, seg, n, out, cap, n, prim_idx, pairs, ctr, nullptr, nullptr, err,
                                             s);
    return launch_wide<SingleMesh, false>(bvh2, seg, n, out, cap, n, prim_idx, pairs, ctr, nullptr, nullptr, err, s);
}

cudaError_t launch_bvh8_batch(const Node2* bvh2, const MeshBatch& batch, uint32_t total, Node8* out, uint32_t slots,
                              uint32_t* prim_idx, uint64_t* pairs, uint32_t* ctr, uint32_t* mesh_nodes,
                              uint32_t* mesh_leaves, uint32_t* err, bool auction, cudaStream_t s,
                              const ChildPair* child_pairs, uint64_t* lists) {
    if (lists && takes_lists(total, auction))
        return launch_group<MeshBatch, false, true>(bvh2, batch, total, out, 0u, slots, prim_idx, pairs, ctr,
                                                    mesh_nodes, mesh_leaves, err, s, child_pairs, lists);
    if (takes_groups(total, auction) && auction)
        return launch_group<MeshBatch, true>(bvh2, batch, total, out, 0u, slots, prim_idx, pairs, ctr, mesh_nodes,
                                             mesh_leaves, err, s, child_pairs);
    if (takes_groups(total, auction))
        return launch_group<MeshBatch, false>(bvh2, batch, total, out, 0u, slots, prim_idx, pairs, ctr, mesh_nodes,
                                              mesh_leaves, err, s, child_pairs);
    if (auction)
        return launch_wide<MeshBatch, true, true>(bvh2, batch, total, out, 0u, slots, prim_idx, pairs, ctr, mesh_nodes,
                                                  mesh_leaves, err, s, child_pairs);
    return launch_wide<MeshBatch, false, true>(bvh2, batch, total, out, 0u, slots, prim_idx, pairs, ctr, mesh_nodes,
                                               mesh_leaves, err, s, child_pairs);
}

cudaError_t load_collapse_kernels() {
    return load_kernels(bvh8_kernel<SingleMesh, false, true>, bvh8_kernel<MeshBatch, false, true>);
}

}  // namespace nxb
