// Stage 4 of a conjunction step: broad phase, i.e. every object's box tested
// against the step's BVH (mizuba/detect_conjunctions_broad_phase.cpp:153-339).
//
// The reference walks the tree once per object in Morton order with an
// explicit stack and emits (orig_p, orig_q) for every member q of every
// overlapped leaf with orig_p < orig_q and otype[p] + otype[q] <= 3, then sorts
// the step's pairs lexicographically.  Here one thread handles one Morton
// position (so a warp's boxes are neighbours in space and its walks stay
// coherent) and walks the tree without a stack by following ropes.  Each
// pair is examined once (the half traversal below) and appended to the batch's
// pair queue with its rank among the pairs of the same (step, lower index);
// an exclusive scan of the counts gives every object its offset in the step's
// list, a scatter pass puts the queue's pairs there and every object's
// partners are sorted, so the lexicographic order comes out directly.  Overlap
// is the reference's closed-interval test on the four dimensions
// (broad_phase.cpp:269-271).
#include <algorithm>

#include "block.cuh"
#include "common.cuh"
#include "kernels.cuh"

namespace mzb
{

// ---- Half traversal (one pass).
//
// Every pair is considered once, from the object x with the lower Morton
// position p.  x's query box is Q = box of x's leaf (equal to x's own box
// unless x sits in a multi-object leaf).  The walk starts at x's own leaf,
// whose members after p are tested first, and then follows the ropes: in
// the depth-first order of the tree the subtrees reached from a leaf by its
// rope chain hold exactly the positions after that leaf, so the walk never
// visits the root-to-leaf path or anything at or before p.  At a leaf L it
// tests each member y at a position q > p with the reference's rule for the
// pair (a, b) = (min, max) of the two indices, "box(a) overlaps the box of
// b's leaf": box(x) vs box(L) when x < y, box(y) vs Q when y < x.  A pair of
// the reference's set is reached by this walk because Q contains box(x) and
// b's leaf box contains box(b), so the exact rule gives the reference's pair
// set with half the node visits.  Partners are filed under a = min(x, y).
//
// Pair queue: entry k is pair[k] = (slot, partner), slot = step * N + a, and
// rank[k], the pair's number among its slot's.  Entries past the capacity are
// counted, not stored (the host grows the queue and walks again).
struct pair_queue {
    uint2 *pair;
    uint32_t *rank;
    uint64_t cap;
    unsigned long long *count;
    uint32_t *counts; // per slot
};

__device__ __forceinline__ bool overlap4(float4 al, float4 au, float4 bl, float4 bu)
{
    return (au.x >= bl.x && al.x <= bu.x) && (au.y >= bl.y && al.y <= bu.y) && (au.z >= bl.z && al.z <= bu.z)
           && (au.w >= bl.w && al.w <= bu.w);
}

// The reference's rule for the pair of x (position p, leaf own) and the member
// at position q of leaf cur, and the object types.
__device__ __forceinline__ bool half_pair(const float *__restrict__ rows, const bvh_node *__restrict__ tree,
                                          const int32_t *__restrict__ otypes, uint32_t p, uint32_t x, int32_t own,
                                          int32_t cur, uint32_t q, uint32_t y)
{
    bool ok;
    if (x < y) {
        const float4 *rx = reinterpret_cast<const float4 *>(rows + uint64_t(p) * 8);
        const float4 *ln = reinterpret_cast<const float4 *>(tree + cur);
        ok = overlap4(rx[0], rx[1], ln[1], ln[2]);
    } else {
        const float4 *ry = reinterpret_cast<const float4 *>(rows + uint64_t(q) * 8);
        const float4 *lq = reinterpret_cast<const float4 *>(tree + own);
        ok = overlap4(ry[0], ry[1], lq[1], lq[2]);
    }
    return ok && otypes[x] + otypes[y] <= 3;
}

// One pair appended by one lane (the alternative walks).
__device__ __forceinline__ void queue_pair(const pair_queue &Q, uint32_t slot0, uint32_t x, uint32_t y)
{
    const uint32_t a = x < y ? x : y, o = x < y ? y : x;
    const uint32_t r = atomicAdd(Q.counts + slot0 + a, 1u);
    const unsigned long long w = atomicAdd(Q.count, 1ull);
    if (w < Q.cap) {
        Q.pair[w] = make_uint2(slot0 + a, o);
        Q.rank[w] = r;
    }
}

// The half walk, one position (gid % N of batch step gid / N) per thread.
//
// A lane keeps the partners it finds in its own column of a shared-memory
// buffer (HITS entries) and walks on; the warp meets when every lane's walk
// has ended or its column is full, and empties the columns together: one
// atomic on the queue's counter for the warp, the ranks' atomics independent
// of one another.  Appended one by one from inside the divergent walk, every
// partner cost its warp two dependent L2 round trips, and dense catalogues
// serialised on the counter.  Broad phase of 48 steps of a 60,000-object
// catalogue at 20 km (24 M pairs) 16.9 -> 4.3 ms, 192 steps of 20,000 objects
// with shells at 10 km (9.8 M) 5.4 -> 2.2 ms, of which the second, full walk
// that the older spill list took on overflow was 11.7 and 2.9 ms; the
// 20,000-object day (4.5 M) is unchanged (2.55 ms): bound by the latency of its
// dependent node loads.  HITS 16 keeps the buffer at 8 KB per CTA, so that the
// walk nodes keep the L1 (the same broad phases with 8, 16 and 24: 4.67, 4.34,
// 4.46; 2.30, 2.19, 2.32; day 2.54, 2.55, 2.70 ms).  Ten CTAs an SM (48 registers): at 72
// registers the day took 3.2 ms, at 40 with spills 3.3 ms.
constexpr int WALK_T = 128;
constexpr int HITS = 16;

__global__ void __launch_bounds__(WALK_T, 10) k_broad_half(const float *__restrict__ srt_aabbs,
                                                       const bvh_node *__restrict__ trees, uint64_t cap,
                                                       const walk_node *__restrict__ walks,
                                                       const uint32_t *__restrict__ leaf_of,
                                                       const uint32_t *__restrict__ srt_idx,
                                                       const uint32_t *__restrict__ tree_size,
                                                       const int32_t *__restrict__ otypes, uint32_t s_first,
                                                       uint32_t nb, uint64_t N, pair_queue Q,
                                                       unsigned long long *visits)
{
    __shared__ uint32_t hit[HITS][WALK_T];
    const unsigned tid = threadIdx.x, lane = tid & 31;
    const uint64_t gid = blockIdx.x * uint64_t(WALK_T) + tid;
    uint32_t n_visits = 0;
    int n_hits = 0;
    const bool in = gid < N * nb;
    const uint32_t b = in ? uint32_t(gid / N) : 0;
    const uint32_t p = in ? uint32_t(gid % N) : 0;
    const uint64_t s = uint64_t(s_first) + b;
    const float *rows = srt_aabbs + s * (N + 1) * 8;
    const bvh_node *tree = trees + s * cap;
    const walk_node *wk = walks + uint64_t(b) * cap;
    const uint32_t *sidx = srt_idx + s * N;
    const uint32_t slot0 = uint32_t(uint64_t(b) * N);
    int32_t cur = -1, own = -1;
    uint32_t x = 0;
    uint32_t first = p + 1; // positions before it are done
    // The walk prunes with the quantised query box; the exact query box and
    // x's own box are read at leaves only (about 1.5 leaves per walk).
    uint4 qq = make_uint4(0, 0, 0, 0);
    if (in && isfinite(rows[uint64_t(p) * 8]) && tree_size[s] != 0) {
        x = sidx[p];
        cur = own = int32_t(leaf_of[uint64_t(b) * N + p]);
        qq = reinterpret_cast<const uint4 *>(wk + own)[0];
    }
    for (;;) {
        while (cur >= 0) {
            // One 32-byte sector per visit: quantised box, left child, rope
            // and member range.
            const uint4 nq = reinterpret_cast<const uint4 *>(wk + cur)[0];
            const int4 m = reinterpret_cast<const int4 *>(wk + cur)[1];
            ++n_visits;
            if (!walk_overlap(qq, nq)) {
                cur = m.y;
                continue;
            }
            if (m.x != -1) {
                cur = m.x;
                continue;
            }
            // Leaf: the reference's exact rule on each member after p (the
            // member tests imply the exact query-box / leaf-box overlap, so
            // the conservative test above changes no pair).
            for (uint32_t q = max(first, uint32_t(m.z)); q < uint32_t(m.w); ++q) {
                const uint32_t y = sidx[q];
                if (!half_pair(rows, tree, otypes, p, x, own, cur, q, y)) continue;
                hit[n_hits++][tid] = y;
                if (n_hits == HITS) {
                    first = q + 1;
                    break;
                }
            }
            if (n_hits == HITS) { // this leaf again, from first on
                --n_visits;
                break;
            }
            cur = m.y;
        }
        const bool alive = __any_sync(0xffffffffu, cur >= 0);
        {
            uint32_t pre = uint32_t(n_hits);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, pre, o);
                if (lane >= unsigned(o)) pre += u;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, pre, 31);
            if (total) {
                unsigned long long base = 0;
                if (lane == 31) base = atomicAdd(Q.count, (unsigned long long)total);
                base = __shfl_sync(0xffffffffu, base, 31) + (pre - uint32_t(n_hits));
                // Two ranks in flight a lane: more cost the walk registers.
#pragma unroll 1
                for (int k = 0; k < n_hits; k += 2) {
                    const bool two = k + 1 < n_hits;
                    const uint32_t y0 = hit[k][tid], y1 = two ? hit[k + 1][tid] : 0;
                    const uint32_t a0 = slot0 + min(x, y0), a1 = slot0 + min(x, y1);
                    const uint32_t r0 = atomicAdd(Q.counts + a0, 1u), r1 = two ? atomicAdd(Q.counts + a1, 1u) : 0;
                    if (base + k < Q.cap) {
                        Q.pair[base + k] = make_uint2(a0, max(x, y0));
                        Q.rank[base + k] = r0;
                    }
                    if (two && base + k + 1 < Q.cap) {
                        Q.pair[base + k + 1] = make_uint2(a1, max(x, y1));
                        Q.rank[base + k + 1] = r1;
                    }
                }
                n_hits = 0;
            }
        }
        if (!alive) break;
    }
    // Node visits of the block's walks, one atomic per warp (the walk's
    // work unit for the roofline).
    const unsigned long long w = __reduce_add_sync(0xffffffffu, n_visits);
    if (lane == 0 && w) atomicAdd(visits, w);
}

// ---- Half traversal with work refill.
//
// The walk and pair rule of k_broad_half, but a lane whose walk has ended
// takes the next position at once instead of waiting for the slowest walk of
// its warp (walk lengths vary several-fold between neighbours, so a warp
// with fixed positions spends most of its time with a third of its lanes
// active).  Each warp draws pools of WALK_POOL consecutive positions from a
// global counter with one atomic; every loop iteration hands the pool's next
// positions to the lanes without a walk and advances every other lane by one
// node.  The set of live lanes is kept explicitly and the warp reconverges on
// it at the top of each iteration, so the pool bookkeeping is warp-uniform.
// On the 20k-object catalogue it loses to fixed positions (3.57 ms against
// 2.81 ms for a day): the per-visit reconvergence and ballot cost more than
// the idle lanes did.  It is kept for inputs with more skewed walks and is
// measured by the autotuner.
constexpr uint32_t WALK_POOL = 64;

__global__ void __launch_bounds__(128) k_broad_pool(const float *__restrict__ srt_aabbs,
                                                    const bvh_node *__restrict__ trees, uint64_t cap,
                                                    const walk_node *__restrict__ walks,
                                                    const uint32_t *__restrict__ leaf_of,
                                                    const uint32_t *__restrict__ srt_idx,
                                                    const uint32_t *__restrict__ tree_size,
                                                    const int32_t *__restrict__ otypes, uint32_t s_first,
                                                    uint32_t nb, uint64_t N, pair_queue Q,
                                                    unsigned long long *next)
{
    const unsigned lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
    const uint64_t total = N * nb;
    unsigned alive = 0xffffffffu;
    uint64_t pool = 0, pool_end = 0; // warp-uniform
    int32_t cur = -1, own = 0;
    uint32_t b = 0, p = 0, x = 0;
    uint64_t s = 0;
    uint4 qq = make_uint4(0, 0, 0, 0);
    for (;;) {
        __syncwarp(alive);
        const unsigned need = __ballot_sync(alive, cur < 0);
        if (need) {
            if (pool == pool_end) {
                const int leader = __ffs(alive) - 1;
                unsigned long long base = 0;
                if (int(lane) == leader) base = atomicAdd(next, (unsigned long long)WALK_POOL);
                base = __shfl_sync(alive, base, leader);
                pool = base < total ? base : total;
                pool_end = base + WALK_POOL < total ? base + WALK_POOL : total;
            }
            const uint64_t avail = pool_end - pool;
            if (avail == 0) { // every position has been handed out
                alive &= ~need;
                if (cur < 0) break;
                continue;
            }
            if (cur < 0) {
                const uint32_t rank = __popc(need & lt);
                if (rank < avail) {
                    const uint64_t gid = pool + rank;
                    b = uint32_t(gid / N);
                    p = uint32_t(gid % N);
                    s = uint64_t(s_first) + b;
                    const float *row = srt_aabbs + (s * (N + 1) + p) * 8;
                    if (isfinite(row[0]) && tree_size[s] != 0) {
                        x = srt_idx[s * N + p];
                        own = int32_t(leaf_of[uint64_t(b) * N + p]);
                        qq = reinterpret_cast<const uint4 *>(walks + uint64_t(b) * cap + own)[0];
                        cur = own;
                    }
                }
            }
            const uint32_t k = __popc(need);
            pool += (k < avail) ? k : avail;
            continue; // lanes given a position start walking next iteration
        }
        // Every live lane has a walk: advance it by one node.
        const walk_node *wk = walks + uint64_t(b) * cap;
        const uint4 nq = reinterpret_cast<const uint4 *>(wk + cur)[0];
        const int4 m = reinterpret_cast<const int4 *>(wk + cur)[1];
        if (!walk_overlap(qq, nq)) {
            cur = m.y;
        } else if (m.x != -1) {
            cur = m.x;
        } else {
            for (uint32_t q = (uint32_t(m.z) > p + 1 ? uint32_t(m.z) : p + 1); q < uint32_t(m.w); ++q) {
                const uint32_t y = srt_idx[s * N + q];
                if (half_pair(srt_aabbs + s * (N + 1) * 8, trees + s * cap, otypes, p, x, own, cur, q, y))
                    queue_pair(Q, uint32_t(uint64_t(b) * N), x, y);
            }
            cur = m.y;
        }
    }
}

// ---- Warp-coherent half traversal.
//
// The same walk and pair rule as k_broad_half, made warp-uniform.  A warp
// holds 32 consecutive Morton positions p of one step (warps never straddle
// two steps), i.e. 32 spatial neighbours whose walks largely coincide.  The
// warp starts at the leaf of its first position and follows the ropes; it
// descends into a node when any lane wants it (an overlap of the lane's
// query box with the node box, and positions after the lane's own in the
// node), otherwise it takes the rope.  Every lane's own leaf and every
// subtree holding positions after it come after the first lane's leaf in
// the depth-first order, so each lane meets every node its own walk would;
// at a leaf each interested lane tests only the members after its own
// position, with the exact rule of k_broad_half, so the pairs are the same.
// Node and rope loads are the same address across the warp (broadcasts) and
// the loop has no divergence except inside leaves.
__global__ void __launch_bounds__(128) k_broad_warp(const float *__restrict__ srt_aabbs,
                                                    const bvh_node *__restrict__ trees, uint64_t cap,
                                                    const int32_t *__restrict__ ropes,
                                                    const uint32_t *__restrict__ leaf_of,
                                                    const uint32_t *__restrict__ srt_idx,
                                                    const uint32_t *__restrict__ tree_size,
                                                    const int32_t *__restrict__ otypes, uint32_t s_first,
                                                    uint32_t nb, uint64_t N, pair_queue Q)
{
    const uint64_t warps_per_step = (N + 31) / 32;
    const uint64_t gw = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) / 32;
    const unsigned lane = threadIdx.x & 31;
    if (gw >= warps_per_step * nb) return; // whole warps only
    const uint32_t b = uint32_t(gw / warps_per_step);
    const uint64_t p64 = (gw % warps_per_step) * 32 + lane;
    const uint64_t s = uint64_t(s_first) + b;
    if (tree_size[s] == 0) return; // uniform over the warp
    bool active = p64 < N;
    const uint32_t p = uint32_t(p64);
    float4 xl = make_float4(0, 0, 0, 0), xu = xl, ql = xl, qu = xl;
    uint32_t x = 0;
    int32_t otx = 0;
    int32_t own = -1;
    if (active) {
        const float4 *row = reinterpret_cast<const float4 *>(srt_aabbs + (s * (N + 1) + p) * 8);
        xl = row[0];
        xu = row[1];
        active = isfinite(xl.x);
    }
    const bvh_node *tree = trees + s * cap;
    const int32_t *rope = ropes + uint64_t(b) * cap;
    const uint32_t *sidx = srt_idx + s * N;
    if (active) {
        x = sidx[p];
        otx = otypes[x];
        own = int32_t(leaf_of[uint64_t(b) * N + p]);
        const float4 *lq = reinterpret_cast<const float4 *>(tree + own);
        ql = lq[1];
        qu = lq[2];
    }
    // No-data boxes sort last: the active lanes are a prefix of the warp.
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (act == 0) return;
    int32_t cur = __shfl_sync(0xffffffffu, own, __ffs(act) - 1);
    while (cur >= 0) {
        const float4 *np = reinterpret_cast<const float4 *>(tree + cur);
        const float4 h = np[0], nl = np[1], nu = np[2];
        const int32_t next = rope[cur];
        const uint32_t qb = __float_as_uint(h.x), qe = __float_as_uint(h.y);
        const bool want = active && qe > p + 1 && overlap4(ql, qu, nl, nu);
        const int32_t left = __float_as_int(h.z);
        if (left != -1) {
            cur = __any_sync(0xffffffffu, want) ? left : next;
            continue;
        }
        // The members one by one, the whole warp together: the pairs found
        // at a member are appended with one atomic on the queue's counter.
        for (uint32_t q = qb; q < qe; ++q) {
            const uint32_t y = sidx[q];
            bool ok = want && q > p;
            if (ok) {
                if (x < y) {
                    ok = overlap4(xl, xu, nl, nu);
                } else {
                    const float4 *ry = reinterpret_cast<const float4 *>(srt_aabbs + (s * (N + 1) + q) * 8);
                    ok = overlap4(ry[0], ry[1], ql, qu);
                }
                ok = ok && otx + otypes[y] <= 3;
            }
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            if (m == 0) continue;
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(Q.count, (unsigned long long)__popc(m));
            base = __shfl_sync(0xffffffffu, base, 0) + __popc(m & lanemask_lt());
            if (ok) {
                const uint32_t sl = uint32_t(uint64_t(b) * N) + (x < y ? x : y);
                const uint32_t r = atomicAdd(Q.counts + sl, 1u);
                if (base < Q.cap) {
                    Q.pair[base] = make_uint2(sl, x < y ? y : x);
                    Q.rank[base] = r;
                }
            }
        }
        cur = next;
    }
}

// The queue's pairs to their places: the step's and the slot's offset plus the
// pair's rank.
__global__ void __launch_bounds__(256) k_broad_scatter(const uint2 *__restrict__ qpair,
                                                       const uint32_t *__restrict__ qrank, uint64_t n, uint32_t N,
                                                       const uint32_t *__restrict__ offs,
                                                       const uint64_t *__restrict__ step_off,
                                                       uint2 *__restrict__ pairs)
{
    const uint64_t k = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    if (k >= n) return;
    const uint2 e = qpair[k];
    const uint32_t b = e.x / N;
    pairs[step_off[b] + offs[e.x] + qrank[k]] = make_uint2(e.x - b * N, e.y);
}

// Sorts the partner lists: those of up to LIST_K partners here, one thread
// each in registers, the longer ones by k_broad_sort_long.
constexpr int LIST_K = 8;

__global__ void __launch_bounds__(256) k_broad_sort_lists(const uint32_t *__restrict__ counts,
                                                          const uint32_t *__restrict__ offs,
                                                          const uint64_t *__restrict__ step_off, uint32_t N,
                                                          uint64_t n,
                                                          uint2 *__restrict__ pairs, uint32_t *__restrict__ longer,
                                                          unsigned long long *n_longer)
{
    const uint64_t slot = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    const uint32_t cnt = slot < n ? counts[slot] : 0;
    const unsigned m = __ballot_sync(0xffffffffu, cnt > LIST_K);
    if (m) {
        unsigned long long base = 0;
        if ((threadIdx.x & 31) == 0) base = atomicAdd(n_longer, (unsigned long long)__popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (cnt > LIST_K) longer[base + __popc(m & lanemask_lt())] = uint32_t(slot);
    }
    if (cnt < 2 || cnt > LIST_K) return;
    uint2 *out = pairs + step_off[uint32_t(slot) / N] + offs[slot];
    uint32_t v[LIST_K];
    const uint32_t a = out[0].x;
#pragma unroll
    for (int k = 0; k < LIST_K; ++k) v[k] = uint32_t(k) < cnt ? out[k].y : 0xffffffffu;
    // Odd-even transposition: LIST_K rounds sort LIST_K values; a list of cnt
    // values behind which only larger ones stand is sorted after cnt rounds.
#pragma unroll
    for (int r = 0; r < LIST_K; ++r) {
        if (uint32_t(r) >= cnt) break;
#pragma unroll
        for (int k = r & 1; k + 1 < LIST_K; k += 2) {
            const uint32_t lo = min(v[k], v[k + 1]), hi = max(v[k], v[k + 1]);
            v[k] = lo;
            v[k + 1] = hi;
        }
    }
#pragma unroll
    for (int k = 0; k < LIST_K; ++k)
        if (uint32_t(k) < cnt) out[k] = make_uint2(a, v[k]);
}

// One warp per longer list.  Up to LONG_CAP partners: every lane counts the
// smaller partners of its own in a shared-memory copy (the partners of one
// object are distinct), which is the partner's place.  Beyond: bitonic merges
// in place whose first round pairs mirrored places, so that every exchange is
// ascending and the places past the end (which would hold +inf) are skipped.
constexpr int LONG_T = 128;
constexpr uint32_t LONG_CAP = 1024;

__global__ void __launch_bounds__(LONG_T) k_broad_sort_long(const uint32_t *__restrict__ longer,
                                                            const unsigned long long *n_longer,
                                                            const uint32_t *__restrict__ counts,
                                                            const uint32_t *__restrict__ offs,
                                                            const uint64_t *__restrict__ step_off, uint32_t N,
                                                            uint2 *pairs)
{
    __shared__ __align__(16) uint32_t sm[LONG_T / 32][LONG_CAP];
    const unsigned lane = threadIdx.x & 31;
    uint32_t *val = sm[threadIdx.x >> 5];
    const uint64_t n = *n_longer;
    for (uint64_t w = (blockIdx.x * uint64_t(LONG_T) + threadIdx.x) >> 5; w < n;
         w += (uint64_t(gridDim.x) * LONG_T) >> 5) {
        const uint32_t slot = longer[w], cnt = counts[slot];
        uint2 *out = pairs + step_off[slot / N] + offs[slot];
        const uint32_t a = out[0].x;
        if (cnt <= LONG_CAP) {
            const uint32_t c4 = (cnt + 3) & ~3u;
            for (uint32_t k = lane; k < c4; k += 32) val[k] = k < cnt ? out[k].y : 0xffffffffu;
            __syncwarp();
            for (uint32_t k = lane; k < cnt; k += 32) {
                const uint32_t v = val[k];
                uint32_t r = 0;
                for (uint32_t j = 0; j < c4; j += 4) {
                    const uint4 u = *reinterpret_cast<const uint4 *>(val + j);
                    r += (u.x < v) + (u.y < v) + (u.z < v) + (u.w < v);
                }
                out[r] = make_uint2(a, v);
            }
            __syncwarp();
        } else {
            for (uint64_t size = 2; size < 2ull * cnt; size <<= 1)
                for (uint64_t stride = size >> 1; stride > 0; stride >>= 1) {
                    const bool mirror = stride == size >> 1;
                    for (uint64_t t = lane;; t += 32) {
                        const uint64_t blk = t / stride, in = t % stride;
                        const uint64_t i = blk * 2 * stride + in;
                        if (blk * 2 * stride >= cnt) break;
                        const uint64_t j = mirror ? blk * 2 * stride + 2 * stride - 1 - in : i + stride;
                        if (j < cnt) {
                            const uint2 u = out[i], v = out[j];
                            if (u.y > v.y) {
                                out[i] = v;
                                out[j] = u;
                            }
                        }
                    }
                    __syncwarp();
                }
        }
    }
}

// ---- Offsets of the partner lists: within each step (one CTA per step, 8
// counts a thread and tile), then the steps' own (one CTA), which also writes
// the host's copies into its mapped memory.  Two launches; the batch-wide scan
// before it took four and one more for the read-back (97 -> 49 us for the
// 20,000-object day's 9.6 M counts, 45 -> 30 us for 60,000 objects x 48 steps).
constexpr int SCAN_T = 1024;
constexpr int SCAN_K = 8;

__global__ void __launch_bounds__(SCAN_T) k_scan_steps(const uint32_t *__restrict__ counts, uint64_t N,
                                                       uint32_t *__restrict__ offs, uint64_t *__restrict__ step_tot)
{
    __shared__ uint32_t sm[33];
    const uint64_t row = uint64_t(blockIdx.x) * N;
    // 32-bit sums: a batch of 2^32 pairs or more is refused by the host, which
    // reads the queue's 64-bit count (a tile's sum alone can wrap).
    uint64_t carry = 0;
    for (uint64_t t0 = 0; t0 < N; t0 += SCAN_T * SCAN_K) {
        const uint64_t i0 = t0 + uint64_t(threadIdx.x) * SCAN_K;
        uint32_t c[SCAN_K], sum = 0;
#pragma unroll
        for (int k = 0; k < SCAN_K; ++k) {
            c[k] = i0 + k < N ? counts[row + i0 + k] : 0;
            sum += c[k];
        }
        uint32_t tot;
        uint32_t run = uint32_t(carry) + block_excl_scan(sum, sm, &tot);
#pragma unroll
        for (int k = 0; k < SCAN_K; ++k) {
            if (i0 + k < N) offs[row + i0 + k] = run;
            run += c[k];
        }
        carry += tot;
    }
    if (threadIdx.x == 0) step_tot[blockIdx.x] = carry;
}

// step_off[b], b <= nb: the pairs of the batch before step b.  host_off,
// host_count and host_visits: device addresses of mapped host memory.
__global__ void __launch_bounds__(SCAN_T) k_step_offsets(const uint64_t *__restrict__ step_tot, uint32_t nb,
                                                         uint64_t *__restrict__ step_off, uint64_t *host_off,
                                                         const unsigned long long *qcount,
                                                         unsigned long long *host_count,
                                                         const unsigned long long *visits,
                                                         unsigned long long *host_visits)
{
    __shared__ uint64_t wsum[SCAN_T / 32];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t carry = 0;
    for (uint32_t b0 = 0; b0 < nb; b0 += SCAN_T) {
        const uint32_t b = b0 + threadIdx.x;
        const uint64_t v = b < nb ? step_tot[b] : 0;
        uint64_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= unsigned(o)) x += y;
        }
        if (lane == 31) wsum[warp] = x;
        __syncthreads();
        uint64_t before = carry, tot = 0;
        for (unsigned w = 0; w < SCAN_T / 32; ++w) {
            if (w < warp) before += wsum[w];
            tot += wsum[w];
        }
        if (b < nb) step_off[b] = host_off[b] = before + x - v;
        carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        step_off[nb] = host_off[nb] = carry;
        *host_count = *qcount;
        *host_visits = *visits;
    }
}

void launch_pair_offsets(const uint32_t *counts, uint64_t N, uint32_t nb, uint32_t *offs, uint64_t *step_tot,
                         uint64_t *step_off, uint64_t *host_off, const unsigned long long *qcount,
                         unsigned long long *host_count, const unsigned long long *visits,
                         unsigned long long *host_visits, cudaStream_t stream)
{
    k_scan_steps<<<nb, SCAN_T, 0, stream>>>(counts, N, offs, step_tot);
    k_step_offsets<<<1, SCAN_T, 0, stream>>>(step_tot, nb, step_off, host_off, qcount, host_count, visits,
                                             host_visits);
}

// counts, *qcount, *walk_next and *visits start at zero.
void launch_broad_half(const float *srt_aabbs, const bvh_node *trees, uint64_t cap, const int32_t *ropes,
                       const walk_node *walks, const uint32_t *leaf_of, const uint32_t *srt_idx,
                       const uint32_t *tree_size, const int32_t *otypes, uint32_t s_first, uint32_t nb, uint64_t N,
                       uint32_t *counts, uint2 *qpair, uint32_t *qrank, uint64_t qcap, unsigned long long *qcount,
                       unsigned long long *walk_next, int walk, unsigned long long *visits, cudaStream_t stream)
{
    const uint64_t n = N * nb;
    const pair_queue Q{qpair, qrank, qcap, qcount, counts};
    if (walk == 2) {
        // Enough warps to fill every SM; each keeps drawing positions.
        k_broad_pool<<<148 * 16, 128, 0, stream>>>(srt_aabbs, trees, cap, walks, leaf_of, srt_idx, tree_size, otypes,
                                                   s_first, nb, N, Q, walk_next);
    } else if (walk == 0) {
        k_broad_half<<<unsigned((n + WALK_T - 1) / WALK_T), WALK_T, 0, stream>>>(
            srt_aabbs, trees, cap, walks, leaf_of, srt_idx, tree_size, otypes, s_first, nb, N, Q, visits);
    } else {
        const uint64_t threads = (N + 31) / 32 * 32 * nb;
        k_broad_warp<<<unsigned((threads + 127) / 128), 128, 0, stream>>>(srt_aabbs, trees, cap, ropes, leaf_of,
                                                                          srt_idx, tree_size, otypes, s_first, nb, N,
                                                                          Q);
    }
}

// n_pairs: the queue's length, which its capacity held.  *n_longer starts at
// zero.
void launch_broad_lists(uint32_t nb, uint64_t N, const uint32_t *counts, const uint32_t *offs,
                        const uint64_t *step_off, const uint2 *qpair, const uint32_t *qrank, uint64_t n_pairs,
                        uint2 *pairs, uint32_t *longer, unsigned long long *n_longer, cudaStream_t stream)
{
    const uint64_t n = N * nb;
    if (n_pairs == 0) return;
    k_broad_scatter<<<unsigned((n_pairs + 255) / 256), 256, 0, stream>>>(qpair, qrank, n_pairs, uint32_t(N), offs,
                                                                         step_off, pairs);
    k_broad_sort_lists<<<unsigned((n + 255) / 256), 256, 0, stream>>>(counts, offs, step_off, uint32_t(N), n, pairs,
                                                                      longer, n_longer);
    k_broad_sort_long<<<unsigned(std::min<uint64_t>(148 * 12, (n + 3) / 4)), LONG_T, 0, stream>>>(
        longer, n_longer, counts, offs, step_off, uint32_t(N), pairs);
}

} // namespace mzb
