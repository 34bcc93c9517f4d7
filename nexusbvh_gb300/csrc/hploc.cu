// hploc.cu - stage 4: H-PLOC binary BVH (Benthin et al. 2024).
//
// Replaces BuildBVH2Kernel (NexusBVH/src/Cuda/BinaryBuilder.cu:200-273).
// The decisions are the reference's, so the topology and every box are
// identical; how they are computed on the GPU differs:
//   * the bottom-up LBVH climb (Apetrei 2014; FindParentId/Delta,
//     BinaryBuilder.cu:14-40) is cut into tiles of consecutive sorted leaves.
//     A warp loads a tile's key deltas, ids and leaf boxes into shared
//     memory once, and every LBVH node whose range lies inside the tile is
//     climbed to, merged and handed over there; only subtrees that touch the
//     tile's edge publish their clusters and climb on through global
//     hand-over slots (see hploc_kernel).  All cross-CTA data is read
//     through L2 after an acquire fence (the reference reads cluster ids and
//     node boxes with plain, L1-cacheable loads, which can return stale
//     lines written by another SM);
//   * LoadIndices (:42-57): a window inside a tile is read from shared
//     memory, its cluster count carried by the hand-over; a published window
//     is read as 16 {box, id, token} records in one round trip;
//   * FindNearestNeighbor (:126-163) is evaluated as what it computes: for
//     lane i, the first minimum of the union area (compared as uint32 bit
//     patterns) over candidates i+1, i-1, i+2, i-2, ..., i+R, i-R, every
//     pair's area computed by one lane and shuffled to the lanes it belongs
//     to (see nearest_neighbour);
//   * the merge and the order-preserving compaction follow
//     MergeClustersCreateBVH2Node (:71-124); internal nodes are numbered
//     from the tokens of the clusters they absorb instead of from a global
//     atomic counter (see merge_step), and the root still lands at 2n-2.
// A published window whose valid ids are not a prefix (impossible for a
// correct climb) sets NXB_DEVERR_HPLOC_INVALID_CLUSTER instead of reading
// out of bounds.
#include <algorithm>

#include "pipeline.h"

namespace nxb {
namespace {

constexpr uint32_t kMergeThreshold = 16;  // MERGING_THRESHOLD, BinaryBuilder.cu:10

// Delta (BinaryBuilder.cu:16-28) of sorted positions a and b of the mesh
// whose first position is s; the index tie-break uses mesh-local positions.
__device__ __forceinline__ uint64_t delta(const uint32_t* k, uint32_t a, uint32_t b, uint32_t s) {
    return (((uint64_t)k[a] << 32) | (a - s)) ^ (((uint64_t)k[b] << 32) | (b - s));
}
__device__ __forceinline__ uint64_t delta(const uint64_t* k, uint32_t a, uint32_t b, uint32_t s) {
    const uint64_t d = k[a] ^ k[b];
    return d ? d : (uint64_t)((a - s) ^ (b - s));
}
// Batched 30-bit keys: mesh << 32 | code, sorted as one key; the delta is
// the 32-bit one of the code.
__device__ __forceinline__ uint64_t delta(const MeshKey* k, uint32_t a, uint32_t b, uint32_t s) {
    const uint32_t ka = (uint32_t)k[a].v, kb = (uint32_t)k[b].v;
    return (((uint64_t)ka << 32) | (a - s)) ^ (((uint64_t)kb << 32) | (b - s));
}
// The mesh of sorted position p (the high half of its key).
__device__ __forceinline__ uint32_t mesh_of(const MeshKey* k, uint32_t p) { return (uint32_t)(k[p].v >> 32); }
template <typename K>
__device__ __forceinline__ uint32_t mesh_of(const K*, uint32_t) {
    return 0;
}
template <typename K, typename Seg>
__device__ __forceinline__ MeshSpan span_at(const K* keys, const Seg& seg, uint32_t p) {
    if constexpr (Seg::kBatch)
        return seg.span(mesh_of(keys, p));
    else
        return seg.of_prim(p);
}

// A run of clusters in shared memory: min xyz and max x, max yz, {id,
// token}.  Three arrays, so that consecutive lanes read each of them without
// a bank conflict (8-byte reads out of 16-byte records took two wavefronts
// where one suffices: 21 % of the kernel's shared-memory load wavefronts).
struct Row {
    uint32_t a, b, c;  // shared-memory addresses
    __device__ __forceinline__ Row at(int32_t k) const { return {a + 16 * k, b + 8 * k, c + 8 * k}; }
    __device__ __forceinline__ void put(int32_t k, const Box& x, uint32_t cid, uint32_t ctok) const {
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a + 16 * k), "f"(x.mn.x), "f"(x.mn.y),
                     "f"(x.mn.z), "f"(x.mx.x)
                     : "memory");
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(b + 8 * k), "f"(x.mx.y), "f"(x.mx.z) : "memory");
        asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(c + 8 * k), "r"(cid), "r"(ctok) : "memory");
    }
    template <int K = 0>
    __device__ __forceinline__ Box box() const {
        Box r;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4 + %5];"
                     : "=f"(r.mn.x), "=f"(r.mn.y), "=f"(r.mn.z), "=f"(r.mx.x)
                     : "r"(a), "n"(16 * K));
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2 + %3];" : "=f"(r.mx.y), "=f"(r.mx.z) : "r"(b), "n"(8 * K));
        return r;
    }
    __device__ __forceinline__ Box box(int32_t k) const { return at(k).box<0>(); }
    __device__ __forceinline__ uint2 ids(int32_t k) const {
        uint2 r;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(c + 8 * k));
        return r;
    }
};

// Slots a row reaches before its first cluster (marks -2, -1) and past its
// 32nd lane (the highest mark is lane + 3, 6 and 15 at radius 4, 8 and 16).
constexpr int kRowFront = 2;
constexpr int row_back(int radius) { return 32 + (radius / 3) * 3; }

// half_area of the unions of two pairs.
__device__ __forceinline__ void pair_areas(const Box& lo0, const Box& hi0, const Box& lo1, const Box& hi1, uint32_t& r0,
                                           uint32_t& r1) {
    Box a = hi0, b = hi1;
    grow(a, lo0);
    grow(b, lo1);
    float f0, f1;
    half_area2(a, b, f0, f1);
    r0 = __float_as_uint(f0);
    r1 = __float_as_uint(f1);
}
__device__ __forceinline__ uint32_t pair_area(const Box& lo, const Box& hi) {
    Box u = hi;
    grow(u, lo);
    return __float_as_uint(half_area(u));
}

// The better of two candidates; the first one wins a tie.
struct Pick {
    uint32_t area;
    int32_t code;
};
__device__ __forceinline__ Pick first_min(Pick a, Pick b) {
    const bool t = b.area < a.area;
    return {t ? b.area : a.area, t ? b.code : a.code};
}
__device__ __forceinline__ Pick both_ways(uint32_t fwd, uint32_t back, int32_t d) {
    return first_min({fwd, d}, {back, -d});
}

// The candidates at distances H, H+1, H+2 and beyond, from the mark lane + H.
// The comparisons form a tree, not a chain of 2R: 285 -> 270 million ALU
// instructions at 4.19M clustered triangles, and a shorter round for a warp
// that runs alone.
template <int R, int H>
__device__ __forceinline__ Pick pick_group(uint32_t num, const Box& cb, const Box& b1, const Box& b0, const Row& own) {
    const uint32_t lane = lane_id();
    const Box hi = own.box<H>();
    const bool in = lane + H < num;
    const int down = (int)(lane - H);  // (taken modulo 32)
    Pick group;
    if constexpr (H + 1 <= R) {
        uint32_t f0, f1;
        pair_areas(cb, hi, b1, hi, f0, f1);
        f0 = in ? f0 : kInvalid;
        f1 = in && lane >= 1 ? f1 : kInvalid;
        group = first_min(both_ways(f0, __shfl_sync(kFullMask, f0, down), H),
                          both_ways(__shfl_down_sync(kFullMask, f1, 1), __shfl_sync(kFullMask, f1, down), H + 1));
    } else {
        const uint32_t f0 = in ? pair_area(cb, hi) : kInvalid;
        group = both_ways(f0, __shfl_sync(kFullMask, f0, down), H);
    }
    if constexpr (H + 2 <= R) {
        const uint32_t a2 = pair_area(b0, hi);
        const uint32_t f2 = in && lane >= 2 ? a2 : kInvalid;
        group = first_min(group, both_ways(__shfl_down_sync(kFullMask, f2, 2), __shfl_sync(kFullMask, f2, down), H + 2));
    }
    if constexpr (H + 3 <= R)
        return first_min(group, pick_group<R, H + 3>(num, cb, b1, b0, own));
    else
        return group;
}

// The nearest neighbour of every lane's cluster, as a signed lane distance
// (0: none); `own` is the lane's place in the row of the window's clusters,
// cb its own box.
// Each lane reads the boxes at lane-2, lane-1 and lane + 3k and computes the
// pairs (lane-1, lane), (lane-2, lane) and, for each k, (lane, lane+3k),
// (lane-1, lane+3k), (lane-2, lane+3k): every distance 1..R once, every pair
// of the window by exactly one lane, with four box reads instead of eight at
// radius 8 (three at radius 4, seven instead of sixteen at radius 16) and no
// wrap-around: a pair is valid if its lower lane is not negative and its
// upper one below num, which depends only on the two marks.  Each area then
// goes to its two lanes (12 shuffles at radius 8).  The union is grown in
// the operand order of the reference (upper box grown by the lower one).
template <int R>
__device__ __forceinline__ int32_t nearest_neighbour(uint32_t num, const Box& cb, const Row& own) {
    const uint32_t lane = lane_id();
    const Box b1 = own.box<-1>(), b0 = own.box<-2>();
    Pick best;
    {
        uint32_t f1, f2;
        pair_areas(b1, cb, b0, cb, f1, f2);
        f1 = lane >= 1 && lane < num ? f1 : kInvalid;
        f2 = lane >= 2 && lane < num ? f2 : kInvalid;
        best = first_min(both_ways(__shfl_sync(kFullMask, f1, (lane + 1) & 31u), f1, 1),
                         both_ways(__shfl_sync(kFullMask, f2, (lane + 2) & 31u), f2, 2));
    }
    return first_min(best, pick_group<R, 3>(num, cb, b1, b0, own)).code;
}

struct Outputs {
    Node2* nodes;
    ChildPair* kids;           // if not null: each internal node's two children, at node - n
    uint32_t* parent_of_last;  // per mesh: the node whose child is node 2n-2 (root fix-up)
    uint32_t* err;
};
// The mesh a merge works on: node i is out.nodes[2 * start + i], its
// child-pair record out.kids[start + i - n].
struct MergeCtx {
    const Outputs& out;
    uint32_t mesh, start, n;
    __device__ __forceinline__ uint32_t limit() const { return 2 * n - 1; }
    __device__ __forceinline__ Node2* node(uint32_t i) const { return out.nodes + (2ull * start + i); }
    __device__ __forceinline__ ChildPair* kid(uint32_t i) const { return out.kids + (start + (i - n)); }
};

// One round of PLOC merging (MergeClustersCreateBVH2Node,
// BinaryBuilder.cu:71-124).  Node numbering: every cluster carries the
// sorted position of its first leaf (its token); merging lanes i < j keeps
// token i, and token j is never seen again.  The n-1 merges therefore
// absorb the tokens 1..n-1 exactly once, and node n-1+token(j) is a
// collision-free index in [n, 2n-1) that needs no global counter (the
// reference takes one atomicAdd on a single counter per merge round).
// The row holds the clusters at the start of every round: the merge reads
// its partner there, and the order-preserving compaction goes through it
// (each kept cluster that moved or merged is written at its rank, every
// lane reads its own slot).
__device__ __forceinline__ uint32_t merge_step(const MergeCtx& m, uint32_t num, int32_t code, uint32_t& cid,
                                               uint32_t& ctok, Box& cb, const Row& row) {
    const uint32_t lane = lane_id();
    const uint32_t nn = (lane + code) & 31u;
    const int32_t back = __shfl_sync(kFullMask, code, nn);
    const bool mutual = lane < num && back == -code;
    const bool merge = mutual && code > 0;
    const bool keep = lane < num && !(mutual && code < 0);
    const uint32_t kmask = __ballot_sync(kFullMask, keep);
    const uint32_t rank = __popc(kmask & lanemask_lt());
    const uint32_t left = __popc(kmask);
    if (merge) {
        const Box nb = row.box(nn);
        const uint2 it = row.ids(nn);
        const uint32_t idx = m.n - 1 + it.y;
        const bool ok = idx < m.limit() && it.y != 0;
        if (ok && m.out.kids) store_child_pair(m.kid(idx), cb, nb, cid, it.x);
        grow(cb, nb);
        if (ok) {
            store_node(m.node(idx), 0, cb, cid, it.x);
            if (cid == m.limit() - 1 || it.x == m.limit() - 1) atomicExch(m.out.parent_of_last + m.mesh, idx);
        } else {
            set_error(m.out.err, NXB_DEVERR_HPLOC_INVALID_CLUSTER);
        }
        cid = idx;
    }
    __syncwarp();  // every read of the row is done
    if (keep && (merge || rank != lane)) row.put(rank, cb, cid, ctok);
    __syncwarp();
    if (lane < left) {
        cb = row.box(lane);
        const uint2 it = row.ids(lane);
        cid = it.x;
        ctok = it.y;
    }
    return left;
}

// The last merge of the build (the root, two clusters left in lanes 0 and
// 1).  The root must sit at node 2n-2, like the reference's; if the token
// numbering put another node there, that node moves to the root's own
// slot n-1+token(lane 1) and its parent's child index is patched.
__device__ __forceinline__ void merge_root(const MergeCtx& m, uint32_t& cid, uint32_t& ctok, Box& cb) {
    const uint32_t lane = lane_id();
    const uint32_t b_cid = __shfl_sync(kFullMask, cid, 1);
    const uint32_t b_tok = __shfl_sync(kFullMask, ctok, 1);
    const Box b_box = shfl_box(cb, 1);
    __syncwarp();
    if (lane == 0) {
        const uint32_t root = m.limit() - 1;
        const uint32_t natural = m.n - 1 + b_tok;
        uint32_t a = cid, b = b_cid;
        if (natural != root) {
            if (natural >= m.limit()) {
                set_error(m.out.err, NXB_DEVERR_HPLOC_INVALID_CLUSTER);
            } else {
                const uint4* src = reinterpret_cast<const uint4*>(m.node(root));
                uint4* dst = reinterpret_cast<uint4*>(m.node(natural));
                const uint4 lo = __ldcg(src), hi = __ldcg(src + 1);
                __stcg(dst, lo);
                __stcg(dst + 1, hi);
                if (m.out.kids) {  // the moved node's child pair moves with it
                    const uint4* ks = reinterpret_cast<const uint4*>(m.kid(root));
                    uint4* kd = reinterpret_cast<uint4*>(m.kid(natural));
                    const uint4 k0 = __ldcg(ks), k1 = __ldcg(ks + 1), k2 = __ldcg(ks + 2), k3 = __ldcg(ks + 3);
                    __stcg(kd, k0);
                    __stcg(kd + 1, k1);
                    __stcg(kd + 2, k2);
                    __stcg(kd + 3, k3);
                }
                if (a == root) {
                    a = natural;
                } else if (b == root) {
                    b = natural;
                } else {
                    const uint32_t p = __ldcg(m.out.parent_of_last + m.mesh);
                    if (p < m.limit() && p >= m.n) {
                        uint32_t* pl = reinterpret_cast<uint32_t*>(m.node(p)) + 6;
                        const uint32_t side = __ldcg(pl) == root ? 0u : 1u;
                        __stcg(pl + side, natural);
                        if (m.out.kids) __stcg(&m.kid(p)->li + side, natural);
                    } else {
                        set_error(m.out.err, NXB_DEVERR_HPLOC_INVALID_CLUSTER);
                    }
                }
            }
        }
        if (m.out.kids) store_child_pair(m.kid(root), cb, b_box, a, b);
        grow(cb, b_box);
        store_node(m.node(root), 0, cb, a, b);
        cid = root;
    }
}

// Merges the window's clusters (in the registers of lanes 0..num-1 and in
// the row) down to at most 16, or to one for the last node of a mesh;
// returns how many are left, in the same places.  Every round merges a pair,
// whatever the boxes hold (areas compare as uint32): of the pairs with the
// least area, then the least distance, the one with the highest lanes is
// mutual, as its lower lane prefers forward and its upper lane has no such
// pair ahead of it.
template <int R>
__device__ __forceinline__ uint32_t merge_window(const MergeCtx& m, uint32_t num, bool fin, uint32_t& cid,
                                                 uint32_t& ctok, Box& cb, const Row& row) {
    const uint32_t threshold = fin ? 1u : kMergeThreshold;
    while (num > threshold) {
        if (fin && num == 2) {
            merge_root(m, cid, ctok, cb);
            return 1;
        }
        const int32_t code = nearest_neighbour<R>(num, cb, row.at(lane_id()));
        num = merge_step(m, num, code, cid, ctok, cb, row);
    }
    return num;
}

// Subtrees that leave their tile store their clusters as {box, id, token}
// records at the window's positions, so that the next merge reads 16
// consecutive records in one round trip.
__device__ __forceinline__ void publish(Node2* rec, uint32_t pos, const Box& b, uint32_t cid, uint32_t ctok) {
    uint4* p = reinterpret_cast<uint4*>(rec + pos);
    __stcg(p, make_uint4(__float_as_uint(b.mn.x), __float_as_uint(b.mn.y), __float_as_uint(b.mn.z),
                         __float_as_uint(b.mx.x)));
    __stcg(p + 1, make_uint4(__float_as_uint(b.mx.y), __float_as_uint(b.mx.z), cid, ctok));
}

// ---------------------------------------------------------------- tiles
// A tile is a run of consecutive sorted leaves held in shared memory by one
// warp.  Gap j of a tile lies between its positions j-1 and j (0..cnt).
// Largest tile and resident warps, measured on GB300 (H-PLOC of 12.58M
// clustered triangles, 63-bit): 128 leaves x 31 warps (64 registers, spills)
// 2.23 ms, 144 x 28 (72 registers; a few spilled at radius 16 and in the
// batched forms) 2.12, 160 x 26 2.16, 176 x 24 2.17, 192 x 22 2.22.  Four CTAs
// of 7 warps and one of 28 measure the same; the small CTA leaves room beside
// it on the SM.
constexpr int kTile = 144;
constexpr int kTileWarps = 7;  // per CTA
constexpr int kTileCtas = 4;   // per SM
constexpr uint64_t kEdge = ~0ull;  // the delta across a mesh's end
template <int R>
struct __align__(16) WarpTile {
    static constexpr int kRows = kTile + kRowFront + row_back(R);
    uint4 a[kRows];
    uint2 b[kRows];
    uint2 c[kRows];
    uint64_t gap[kTile + 2];   // deltas; then the list of subtrees that leave the tile
    uint32_t hand[kTile + 4];  // hand-over slots: the range's other end | clusters << 16
    uint4 mesh;                // batches: the mesh, its start and count if the tile lies in one, else count 0
    __device__ __forceinline__ Row rows() {
        return {(uint32_t)__cvta_generic_to_shared(a + kRowFront), (uint32_t)__cvta_generic_to_shared(b + kRowFront),
                (uint32_t)__cvta_generic_to_shared(c + kRowFront)};
    }
};

template <typename K, typename Seg>
struct Climb {
    // the mesh of the leaf at position p, which lies in the tile (or in a
    // range that reaches into it)
    template <int R>
    __device__ __forceinline__ MeshSpan span(const WarpTile<R>& t, uint32_t p) const {
        if constexpr (Seg::kBatch) {
            const uint4 m = t.mesh;
            if (m.z) return {m.x, m.y, m.z};
            return span_at(keys, seg, p);
        } else {
            return seg.of_prim(p);
        }
    }
    const K* keys;
    const uint32_t* cluster;
    uint32_t* parent;
    Seg seg;
    Outputs out;
    Node2* rec;
    uint32_t begin, end, tile;  // tile: leaves per tile
    uint64_t* bvh8_pairs;
};

// LoadIndices (BinaryBuilder.cu:42-57): one lane's entry k of a published
// window of `size` leaves at `pos`.
template <typename K, typename Seg>
__device__ __forceinline__ void load_entry(const Climb<K, Seg>& g, uint32_t pos, uint32_t k, uint32_t size, uint32_t& v,
                                           uint32_t& t, Box& b) {
    v = kInvalid;
    t = 0;
    b.mn = b.mx = make_float3(0.f, 0.f, 0.f);
    if (k >= min(size, kMergeThreshold)) return;
    const uint4* p = reinterpret_cast<const uint4*>(g.rec + pos + k);
    const uint4 lo = __ldcg(p), hi = __ldcg(p + 1);
    b.mn = make_float3(__uint_as_float(lo.x), __uint_as_float(lo.y), __uint_as_float(lo.z));
    b.mx = make_float3(__uint_as_float(lo.w), __uint_as_float(hi.x), __uint_as_float(hi.y));
    v = hi.z;
    t = hi.w;
}

// FindParentId (BinaryBuilder.cu:30-40): whether the range [l, r] of the mesh
// of n leaves at `start` (not all of them) hands over at its right end.
template <typename K>
__device__ __forceinline__ bool hands_right(const K* keys, uint32_t l, uint32_t r, uint32_t start, uint32_t n) {
    return l == start || (r != start + n - 1 && delta(keys, r, r + 1, start) < delta(keys, l - 1, l, start));
}

// PlocMerge (BinaryBuilder.cu:200-273, the merge part) between tiles, for
// the range of lane `owner`, whose two children were published; then on up
// the tree for as long as the sibling has already arrived: its hand-over
// slot is read (acquire) instead of exchanged, and the range's own clusters
// stay in the row, so such a level has no fence, no exchange and one window
// to load.  Returns the range reached and whether it is a whole mesh; the
// clusters of a range that is not are stored (StoreIndices, :59-69).
template <int R, typename K, typename Seg>
__device__ __forceinline__ bool merge_between(const Climb<K, Seg>& g, const WarpTile<R>& t, uint32_t owner,
                                              uint32_t& left, uint32_t& right, uint32_t split, const Row& row) {
    const uint32_t lane = lane_id();
    uint32_t l = __shfl_sync(kFullMask, left, owner), r = __shfl_sync(kFullMask, right, owner);
    const uint32_t mid = __shfl_sync(kFullMask, split, owner);
    const MeshSpan me = g.span(t, l);
    const uint32_t start = me.start;
    const MergeCtx m{g.out, me.m, start, me.count};
    uint32_t cid, ctok, num, first;
    Box cb;
    bool bad;  // a window's valid ids must be a prefix of it, and in range
    {
        const bool lo = lane < 16;
        load_entry(g, lo ? l : mid, lane & 15u, lo ? mid - l : r + 1 - mid, cid, ctok, cb);
        const uint32_t vb = __ballot_sync(kFullMask, cid != kInvalid);
        first = __popc(vb & 0xFFFFu);
        num = __popc(vb);
        bad = (vb & 0xFFFFu) != (1u << first) - 1u || vb >> 16 != (1u << (num - first)) - 1u;
        __syncwarp();  // the row's last readers are done
        if (cid != kInvalid) row.put(lo ? lane : first + lane - 16, cb, cid, ctok);
    }
    bool fin = false;
    for (;;) {
        __syncwarp();
        cid = kInvalid;
        if (lane < num) {
            cb = row.box(lane);
            const uint2 it = row.ids(lane);
            cid = it.x;
            ctok = it.y;
        }
        if (bad || __any_sync(kFullMask, lane < num && (cid >= m.limit() || ctok >= m.n))) {
            if (lane == 0) set_error(m.out.err, NXB_DEVERR_HPLOC_INVALID_CLUSTER);
            fin = true;
            break;
        }
        fin = r - l + 1 == m.n;
        // where the range hands over (its keys are read before the merge, so
        // that only the slot is waited for after it)
        const bool go_right = !fin && hands_right(g.keys, l, r, start, m.n);
        num = merge_window<R>(m, num, fin, cid, ctok, cb, row);
        if (fin) break;
        const uint32_t other = __shfl_sync(kFullMask, ld_acquire_u32(g.parent + (go_right ? r : l - 1)), 0);
        if (other == kInvalid) break;
        __syncwarp();  // acquired by all
        uint32_t v, vt;
        Box b;
        load_entry(g, go_right ? r + 1 : other, lane, go_right ? other - r : l - other, v, vt, b);
        const uint32_t vb = __ballot_sync(kFullMask, v != kInvalid);
        const uint32_t ns = __popc(vb);
        bad = (vb & (vb + 1)) != 0;
        __syncwarp();
        if (!go_right && lane < num) row.put(ns + lane, cb, cid, ctok);
        if (v != kInvalid) row.put((go_right ? num : 0u) + lane, b, v, vt);
        num += ns;
        if (go_right)
            r = other;
        else
            l = other;
    }
    if (!fin && lane < min(r - l + 1, kMergeThreshold)) publish(g.rec, l + lane, cb, lane < num ? cid : kInvalid, ctok);
    if (lane == owner) {
        left = l;
        right = r;
    }
    return fin;
}

// Loads leaves [base, base + cnt) into the warp's tile: the gaps' deltas,
// the leaves' ids and boxes.
template <int R, typename K, typename Seg>
__device__ __forceinline__ void load_tile(const Climb<K, Seg>& g, WarpTile<R>& t, uint32_t base, uint32_t cnt) {
    constexpr int kPer = (kTile + 31) / 32;
    const uint32_t lane = lane_id();
    const Row rows = t.rows();
    // most tiles of a batch lie inside one mesh
    MeshSpan first = span_at(g.keys, g.seg, base);
    const bool one = !Seg::kBatch || base + cnt <= first.start + first.count;
    if (Seg::kBatch && lane == 0) t.mesh = make_uint4(first.m, first.start, one ? first.count : 0u, 0u);
    uint32_t id[kPer];
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const uint32_t j = lane + 32 * q;
        id[q] = j < cnt ? g.cluster[base + j] : kInvalid;
    }
#pragma unroll
    for (int q = 0; q <= kPer; ++q) {
        const uint32_t j = lane + 32 * q;
        if (j > cnt) break;
        const uint32_t p = base + j;
        uint32_t start = first.start;
        bool edge;
        if (one) {
            edge = p == start || p == start + first.count;
        } else {
            edge = p == g.begin || p == g.end || mesh_of(g.keys, p - 1) != mesh_of(g.keys, p);
            if (!edge) start = span_at(g.keys, g.seg, p).start;
        }
        uint64_t d = kEdge;
        if (!edge) {
            d = delta(g.keys, p - 1, p, start);
            d = d < kEdge ? d : kEdge - 1;  // only a mesh's end is an edge
        }
        t.gap[j] = d;
        t.hand[j] = kInvalid;
    }
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
        const uint32_t j = lane + 32 * q;
        if (j < cnt) {
            const MeshSpan me = one ? first : span_at(g.keys, g.seg, base + j);
            Box b;
            b.mn = b.mx = make_float3(0.f, 0.f, 0.f);
            if (id[q] < me.count)
                b = load_box(g.out.nodes + 2ull * me.start, id[q]);
            else
                set_error(g.out.err, NXB_DEVERR_HPLOC_INVALID_CLUSTER);
            rows.put(j, b, id[q], base + j - me.start);
            if (!Seg::kBatch && g.bvh8_pairs) g.bvh8_pairs[base + j] = bvh8_queue_slot(base + j, g.end);
        }
    }
}

// The climb inside the tile.  Each lane climbs from a leaf as in the
// reference (FindParentId: a range hands over at the smaller of its two
// bounding deltas; the second to arrive continues), with the hand-over slots
// in shared memory: the value is the range's other end and its cluster
// count.  A lane that stops takes the tile's next leaf.  A node of more than
// 16 leaves is merged by the whole warp, and the warp goes on up the tree
// while the sibling is there; the clusters stay in the rows at the range's
// first positions, where the next merge finds them, so nothing in global
// memory is waited for.  A range that arrives at a slot alone waits there:
// its sibling reaches past the tile.
template <int R, typename K, typename Seg>
__device__ __forceinline__ void climb_tile(const Climb<K, Seg>& g, WarpTile<R>& t, uint32_t base, uint32_t cnt) {
    const uint32_t lane = lane_id();
    const Row rows = t.rows();
    uint32_t range = 0;  // left | right << 16
    uint32_t parts = 0;  // split | left clusters << 16 | right clusters << 24
    uint32_t next = 0;
    bool active = false;
    for (;;) {
        const uint32_t need = __ballot_sync(kFullMask, !active);
        if (next < cnt && need) {
            const uint32_t mine = next + __popc(need & lanemask_lt());
            if (!active && mine < cnt) {
                range = mine | mine << 16;
                parts = 1u << 16;
                active = true;
            }
            next += __popc(need);
        }
        if (!__any_sync(kFullMask, active)) break;
        bool second = false, final = false;
        if (active) {
            uint32_t left = range & 0xFFFFu, right = range >> 16;
            const uint64_t dl = t.gap[left], dr = t.gap[right + 1];
            active = false;
            if (dl != kEdge || dr != kEdge) {  // else a mesh's root
                const bool go_right = dr < dl;
                const uint32_t gp = go_right ? right + 1 : left;
                const uint32_t have = (parts >> 16 & 0xFFu) + (parts >> 24);
                const uint32_t prev = atomicExch(&t.hand[gp], (go_right ? left : right) | have << 16);
                if (prev != kInvalid) {
                    t.hand[gp] = kInvalid;
                    const uint32_t sib = prev >> 16;
                    if (go_right) {
                        right = prev & 0xFFFFu;
                        parts = gp | have << 16 | sib << 24;
                    } else {
                        left = prev & 0xFFFFu;
                        parts = gp | sib << 16 | have << 24;
                    }
                    range = left | right << 16;
                    active = second = true;
                    final = t.gap[left] == kEdge && t.gap[right + 1] == kEdge;
                }
            }
        }
        uint32_t todo =
            __ballot_sync(kFullMask, second && ((range >> 16) - (range & 0xFFFFu) >= kMergeThreshold || final));
        while (todo) {
            const uint32_t owner = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t lr = __shfl_sync(kFullMask, range, owner), ps = __shfl_sync(kFullMask, parts, owner);
            uint32_t l = lr & 0xFFFFu, r = lr >> 16, mid = ps & 0xFFFFu, cl = ps >> 16 & 0xFFu, num = cl + (ps >> 24);
            bool fin = t.gap[l] == kEdge && t.gap[r + 1] == kEdge;
            const MeshSpan me = g.span(t, base + l);
            const MergeCtx m{g.out, me.m, me.start, me.count};
            uint32_t cid, ctok = 0;
            Box cb;
            for (;;) {
                // both windows, side by side at the range's first positions
                const Row row = rows.at(l);
                cid = kInvalid;
                __syncwarp();
                if (lane < num) {
                    const uint32_t k = lane < cl ? lane : mid - l + lane - cl;
                    cb = row.box(k);
                    const uint2 it = row.ids(k);
                    cid = it.x;
                    ctok = it.y;
                }
                __syncwarp();
                if (mid - l != cl && lane >= cl && lane < num) row.put(lane, cb, cid, ctok);
                __syncwarp();
                num = merge_window<R>(m, num, fin, cid, ctok, cb, row);
                // on up the tree while the sibling is there
                const uint64_t dl = t.gap[l], dr = t.gap[r + 1];
                if (dl == kEdge && dr == kEdge) break;
                const bool go_right = dr < dl;
                const uint32_t gp = go_right ? r + 1 : l;
                const uint32_t prev = t.hand[gp];
                if (prev == kInvalid) break;
                __syncwarp();
                if (lane == 0) t.hand[gp] = kInvalid;
                mid = gp;
                if (go_right) {
                    r = prev & 0xFFFFu;
                    cl = num;
                } else {
                    l = prev & 0xFFFFu;
                    cl = prev >> 16;
                }
                num += prev >> 16;
                fin = t.gap[l] == kEdge && t.gap[r + 1] == kEdge;
            }
            if (lane == owner) {
                range = l | r << 16;
                parts = num << 16;
            }
        }
        __syncwarp();
    }
}

// The subtrees left alone in a hand-over slot reach past the tile: lists
// them (in t.gap) and stores their clusters; returns how many.
template <int R, typename K, typename Seg>
__device__ __forceinline__ uint32_t leave_tile(const Climb<K, Seg>& g, WarpTile<R>& t, uint32_t base, uint32_t cnt) {
    const uint32_t lane = lane_id();
    const Row rows = t.rows();
    uint32_t leaving = 0;
    __syncwarp();
    for (uint32_t g0 = 0; g0 <= cnt; g0 += 32) {
        const uint32_t gap = g0 + lane;
        const uint32_t v = gap <= cnt ? t.hand[gap] : kInvalid;
        const uint32_t mask = __ballot_sync(kFullMask, v != kInvalid);
        if (v != kInvalid) {
            const uint32_t other = v & 0xFFFFu;
            const bool is_left = other < gap;  // the range ends at the gap, else it starts there
            const uint32_t l = is_left ? other : gap, r = is_left ? gap - 1 : other;
            t.gap[leaving + __popc(mask & lanemask_lt())] =
                (uint64_t)(l | r << 16) | ((uint64_t)(v >> 16 | (is_left ? 0x100u : 0u)) << 32);
        }
        leaving += __popc(mask);
    }
    __syncwarp();
    for (uint32_t i = lane >> 4; i < leaving; i += 2) {
        const uint64_t e = t.gap[i];
        const uint32_t l = (uint32_t)e & 0xFFFFu, size = (((uint32_t)e >> 16) & 0xFFFFu) - l + 1;
        const uint32_t num = (uint32_t)(e >> 32) & 0xFFu, k = lane & 15u;
        if (k < min(size, kMergeThreshold)) {
            const uint2 it = rows.ids(l + k);
            publish(g.rec, base + l + k, rows.box(l + k), k < num ? it.x : kInvalid, it.y);
        }
    }
    __syncwarp();
    return leaving;
}

// The climb between tiles, for the `leaving` subtrees listed in t.gap: their
// lanes hand over through slots in global memory (parent[g] for the gap
// after position g; the value is the range's other end).  The exchanges are
// relaxed; a pass that found siblings fences (acquire) after its exchanges,
// before reading the siblings' clusters, and (release) before the next
// pass's exchanges.  A join of less than 17 leaves has nothing to merge or to
// store, and above it the next sibling has often arrived (a tile's edge is
// crossed by a chain of such joins), so its lane goes on with an acquiring
// read of the next slot (0.9 us a level, 2.5 with two fences and an exchange);
// it exchanges only where that is empty.  Nothing waits on another warp.
// With merge_between reading its keys early, H-PLOC of 1,021 triangles 41 ->
// 34 us, 65,536 72 -> 65, 16,411 boxes 84 -> 77, 4.19M sphere 469 -> 453.
template <int R, typename K, typename Seg>
__device__ __forceinline__ void climb_between(const Climb<K, Seg>& g, WarpTile<R>& t, uint32_t base,
                                              uint32_t leaving) {
    const uint32_t lane = lane_id();
    const Row row = t.rows();
    uint32_t item = lane;
    uint32_t left = 0, right = 0, split = 0;
    bool active = false, peek = false;
    MeshSpan me = Seg::kBatch ? MeshSpan{0, 0, 0} : g.seg.of_prim(0);
    bool release_due = true;  // warp-uniform: stores or acquired clusters since the last release fence
    for (;;) {
        bool fresh = false, go_right = false;
        if (!active && item < leaving) {
            const uint64_t e = t.gap[item];
            item += 32;
            left = base + ((uint32_t)e & 0xFFFFu);
            right = base + (((uint32_t)e >> 16) & 0xFFFFu);
            go_right = (e >> 40) & 1u;
            active = fresh = true;
            peek = false;
        }
        if (!__any_sync(kFullMask, active)) break;
        if (Seg::kBatch && fresh) me = g.span(t, left);
        if (active && !fresh) go_right = hands_right(g.keys, left, right, me.start, me.count);
        uint32_t* slot = g.parent + (go_right ? right : left - 1);
        uint32_t sib = kInvalid;  // the sibling's other end
        if (active && peek) sib = ld_acquire_u32(slot);
        const bool put = active && sib == kInvalid;
        if (__any_sync(kFullMask, put)) {
            if (release_due) {
                __syncwarp();
                fence_acq_rel_gpu();
                release_due = false;
            }
            if (put) sib = atomicExch(slot, go_right ? left : right);
            if (__any_sync(kFullMask, put && sib != kInvalid)) fence_acq_rel_gpu();  // acquire: the siblings' clusters
        }
        active = active && sib != kInvalid;
        peek = active;
        if (active) {
            split = go_right ? right + 1 : left;
            if (go_right)
                right = sib;
            else
                left = sib;
        }
        uint32_t todo = __ballot_sync(
            kFullMask, active && (right - left >= kMergeThreshold || right - left + 1 == me.count));
        if (todo >> lane & 1u) peek = false;  // merge_between has looked
        if (__any_sync(kFullMask, active)) release_due = true;
        __syncwarp();  // acquired by all
        while (todo) {
            const uint32_t owner = __ffs(todo) - 1;
            todo &= todo - 1;
            if (merge_between<R>(g, t, owner, left, right, split, row) && lane == owner) active = false;
        }
    }
    __syncwarp();
}

// Persistent warps, each with a tile of its own in shared memory; nothing
// waits on another warp.
//
// What bounds it: the ALU (62 % busy while active at 4.19M clustered
// triangles; a round of neighbour search takes about 130 ALU instructions of
// 240), the shared-memory pipe (59 %) and, for small or deep trees, the chain
// of merges from a leaf to the root, one after another.  A climb through
// global hand-over slots alone (a persistent grid whose warps take leaves)
// costs two fences, an exchange and two dependent loads at every level; with
// most levels inside a tile a merge takes 6 us of a warp instead of 9.
// Measured against that form (H-PLOC, before -> now): 12.58M clustered
// triangles 2.33 -> 2.12 ms, 4.19M sphere 0.576 -> 0.470, 3.0M at radius 16
// 1.14 -> 0.95, 500,009 clustered boxes 0.38 -> 0.20, 65,536 soup triangles
// 0.092 -> 0.071 ms.  A tile shared by the four warps of a CTA (512 leaves)
// left 45 % of the warp time at its barrier (clustered trees are chains, with
// about two merges ready at a time), and one-warp CTAs that are not
// persistent start too slowly (one per 27 ns).
template <typename K, int R, typename Seg>
__global__ __launch_bounds__(32 * kTileWarps, kTileCtas) void hploc_kernel(Climb<K, Seg> g, uint32_t tiles, uint32_t* tile_ctr,
                                                            uint32_t* bvh8_ctr) {
    after_previous();
    extern __shared__ __align__(16) unsigned char smem[];
    WarpTile<R>& t = reinterpret_cast<WarpTile<R>*>(smem)[threadIdx.x >> 5];
    if (!Seg::kBatch && bvh8_ctr && blockIdx.x == 0 && threadIdx.x == 0) bvh8_queue_counters(bvh8_ctr);
    // the first tile of each warp spreads small builds over the SMs
    uint32_t tile = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    while (tile < tiles) {
        const uint32_t base = g.begin + tile * g.tile, cnt = min(g.tile, g.end - base);
        load_tile<R>(g, t, base, cnt);
        __syncwarp();
        climb_tile<R>(g, t, base, cnt);
        const uint32_t leaving = leave_tile<R>(g, t, base, cnt);
        if (leaving) climb_between<R>(g, t, base, leaving);
        if (lane_id() == 0) tile = gridDim.x * (blockDim.x >> 5) + atomicAdd(tile_ctr, 1u);
        tile = __shfl_sync(kFullMask, tile, 0);
    }
}

template <typename K, int R, typename Seg>
cudaError_t launch_r(const Climb<K, Seg>& g, uint32_t* tile_ctr, uint32_t* bvh8_ctr, uint32_t max_per_sm,
                     cudaStream_t s) {
    constexpr size_t smem = sizeof(WarpTile<R>) * kTileWarps;
    static_assert(kTileCtas * (smem + 1024) <= 228 * 1024, "shared memory of an SM");
    const cudaError_t e = once_per_device([] {
        cudaError_t r = cudaFuncSetAttribute(hploc_kernel<K, R, Seg>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (!r)
            r = cudaFuncSetAttribute(hploc_kernel<K, R, Seg>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        return r;
    });
    if (e) return e;
    const uint32_t sms = (uint32_t)device_info().sms;
    const uint32_t tiles = (g.end - g.begin + g.tile - 1) / g.tile;
    // resident warps per SM; the batch tuning's cap counts CTAs of four warps
    uint32_t per_sm = std::min((tiles + sms - 1) / sms, (uint32_t)(kTileWarps * kTileCtas));
    if (max_per_sm) per_sm = std::min(per_sm, 4 * max_per_sm);
    const uint32_t ctas = (per_sm + kTileWarps - 1) / kTileWarps, warps = (per_sm + ctas - 1) / ctas;
    const uint32_t grid = std::min(tiles, sms * ctas);
    if constexpr (!Seg::kBatch)
        return launch_after(g.end, hploc_kernel<K, R, Seg>, grid, 32 * warps, sizeof(WarpTile<R>) * warps, s, g, tiles, tile_ctr,
                            bvh8_ctr);
    hploc_kernel<K, R, Seg><<<grid, 32 * warps, sizeof(WarpTile<R>) * warps, s>>>(g, tiles, tile_ctr, bvh8_ctr);
    return cudaGetLastError();
}

template <typename K, typename Seg>
cudaError_t launch_t(const K* keys, const uint32_t* cluster, uint32_t* parent, Node2* nodes, Seg seg, uint32_t begin,
                     uint32_t end, uint32_t radius, uint32_t* pol, uint32_t* tile_ctr, uint32_t* err,
                     uint32_t max_per_sm, cudaStream_t s, Node2* rec, uint64_t* pairs, uint32_t* ctr,
                     ChildPair* kids) {
    if (begin == end) return cudaSuccess;  // a batch's group of empty meshes has nothing to climb
    // one tile per resident warp while that is at most kTile leaves, so that
    // small builds use every SM: 65,536 triangles take 71 us with 32 leaves
    // per tile, 88 with 144.  The smallest tile is a window and a little: whole
    // builds of 1,021 / 8,000 / 16,411 / 32,000 / 65,536 primitives with 16
    // leaves 68 / 96 / 161 / 124 / 143 us, 20: 68 / 92 / 159 / 120 / 143, 24:
    // 69 / 93 / 158 / 120 / 145, 32: 72 / 94 / 163 / 119 / 146
    const uint32_t warps = (uint32_t)device_info().sms * kTileWarps * kTileCtas;
    const uint32_t tile = std::max(20u, std::min((end - begin + warps - 1) / warps, (uint32_t)kTile));
    const Climb<K, Seg> g{keys, cluster, parent, seg, {nodes, kids, pol, err}, rec, begin, end, tile, pairs};
    switch (radius) {
        case 4: return launch_r<K, 4, Seg>(g, tile_ctr, ctr, max_per_sm, s);
        case 16: return launch_r<K, 16, Seg>(g, tile_ctr, ctr, max_per_sm, s);
        default: return launch_r<K, 8, Seg>(g, tile_ctr, ctr, max_per_sm, s);
    }
}

}  // namespace

cudaError_t launch_hploc(uint32_t key_bytes, const void* keys, uint32_t* cluster_idx, uint32_t* parent, Node2* nodes,
                         uint32_t n, uint32_t radius, uint32_t* parent_of_last, uint32_t* ctr, uint32_t* err,
                         cudaStream_t s, Node2* records, uint64_t* bvh8_pairs, uint32_t* bvh8_ctr,
                         ChildPair* child_pairs) {
    const SingleMesh seg{n};
    if (!bvh8_pairs != !bvh8_ctr) return cudaErrorInvalidValue;
    if (key_bytes == 4)
        return launch_t((const uint32_t*)keys, cluster_idx, parent, nodes, seg, 0u, n, radius, parent_of_last, ctr,
                        err, 0u, s, records, bvh8_pairs, bvh8_ctr, child_pairs);
    return launch_t((const uint64_t*)keys, cluster_idx, parent, nodes, seg, 0u, n, radius, parent_of_last, ctr,
                    err, 0u, s, records, bvh8_pairs, bvh8_ctr, child_pairs);
}

cudaError_t launch_hploc_batch(const uint64_t* keys, uint32_t* cluster_idx, uint32_t* parent, Node2* nodes,
                               const MeshBatch& batch, uint32_t begin, uint32_t end, uint32_t radius,
                               Node2* records, uint32_t* parent_of_last, uint32_t* ctr, uint32_t* err,
                               uint32_t ctas_per_sm, cudaStream_t s, ChildPair* child_pairs) {
    return launch_t(reinterpret_cast<const MeshKey*>(keys), cluster_idx, parent, nodes, batch, begin, end, radius,
                    parent_of_last, ctr, err, ctas_per_sm, s, records, nullptr, nullptr, child_pairs);
}

}  // namespace nxb
