// Stage 5 of a conjunction step: narrow phase
// (mizuba/detect_conjunctions_narrow_phase.cpp:167-769).
//
// k_items: one thread per broad-phase pair walks the two objects' segment
//   boundaries (narrow.cpp:345-418) and appends every overlapping
//   sub-interval to a device queue of items.
// k_narrow_filter: one thread per item (persistent grid pulling from that
//   queue) settles the items whose outcome a cheap FMA formulation proves:
//   those whose enclosure clears the threshold, and those with one interior
//   minimum that clears it.  In the mixed form a distance screen inside the
//   merge walk drops most items before it.
// k_narrow: one thread per item that is left
//   translates both position polynomials to the sub-interval start
//   (conjunctions_jit.cpp:68-140), evaluates them at the order+1 Chebyshev
//   nodes, interpolates the squared distance with Bjorck-Pereyra
//   (narrow.cpp:95-152, poly_utils.cpp:467-535) and encloses it with
//   Cargo-Shisha (narrow.cpp:502-517).  Sub-intervals whose enclosure does not
//   reach below threshold^2 are dropped; the others go to a device queue with
//   their distance polynomial.
// k_roots: one thread per queued sub-interval (persistent grid pulling from the
//   device queue) runs the minimum search on the
//   derivative (poly_utils.cpp:272-460): fast exclusion, Descartes/VCA
//   isolation with the reference's LIFO working list (in global scratch,
//   at most 251 entries as in the reference), TOMS 748 polishing, the
//   threshold test on the interpolant, the trajectory-boundary minima
//   (narrow.cpp:629-714) and the state vectors at TCA (narrow.cpp:542-575).
// k_conj_*: per-step ordering by (tca, record) (narrow.cpp:751-757).
#include <algorithm>
#include <cmath>

#include "block.cuh"
#include "common.cuh"
#include "filter_margin.cuh"
#include "kernels.cuh"

namespace mzb
{

// ------------------------------------------------------------- k_narrow

__device__ __forceinline__ double dmax_ref(double a, double b) { return (a < b) ? b : a; } // std::max(a, b)
__device__ __forceinline__ double dmin_ref(double a, double b) { return (b < a) ? b : a; } // std::min(a, b)

__device__ __forceinline__ void warp_add(unsigned long long *ctr, unsigned long long v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(ctr, v);
}

// The sums of a and b over the CTA, added to *pa (and *pa2, when given) and
// *pb: one atomic each per CTA.  Every thread of the CTA takes part.
__device__ __forceinline__ void block_add2(unsigned long long *pa, unsigned long long *pa2, unsigned a,
                                           unsigned long long *pb, unsigned b)
{
    __shared__ unsigned sa, sb;
    if (threadIdx.x == 0) sa = sb = 0;
    __syncthreads();
    a = __reduce_add_sync(0xffffffffu, a);
    b = __reduce_add_sync(0xffffffffu, b);
    if ((threadIdx.x & 31) == 0) {
        if (a) atomicAdd(&sa, a);
        if (b) atomicAdd(&sb, b);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (sa) atomicAdd(pa, (unsigned long long)sa);
        if (sa && pa2) atomicAdd(pa2, (unsigned long long)sa);
        if (sb) atomicAdd(pb, (unsigned long long)sb);
    }
}

// Warp-aggregated append of one slot per active lane; returns this lane's
// slot.
__device__ __forceinline__ unsigned long long warp_append(unsigned long long *counter, bool want)
{
    const unsigned mask = __ballot_sync(0xffffffffu, want);
    if (!want) return 0;
    const unsigned lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    unsigned long long base = 0;
    if (int(lane) == leader) base = atomicAdd(counter, (unsigned long long)__popc(mask));
    base = __shfl_sync(mask, base, leader);
    return base + __popc(mask & lanemask_lt());
}

// One thread per broad-phase pair: the merge walk over both objects' segment
// boundaries (narrow.cpp:345-418) appends every overlapping sub-interval to
// the item queue.  Items are re-sorted per step at the end, so queue order is
// free.  With increasing time points every live iteration advances at least
// one cursor, so a walk ends within (ei - it_i) + (ej - it_j) iterations; a
// walk that reaches that bound (time points out of order on the device)
// stops and reports ERR_NP_INTERVAL instead of spinning.
__global__ void __launch_bounds__(128) k_items(const dev_pj pj, const double2 *__restrict__ cd_bounds,
                                               uint32_t s_first, uint32_t nb, const uint2 *__restrict__ pairs,
                                               const uint64_t *__restrict__ step_off,
                                               const uint2 *__restrict__ srange, np_item *__restrict__ items,
                                               uint64_t cap, unsigned long long *item_count,
                                               unsigned long long *counters, dev_status *st)
{
    const uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    const uint64_t n_pairs = step_off[nb];
    bool active = p < n_pairs;
    uint32_t b = 0, i = 0, j = 0, it_i = 0, it_j = 0, ei = 0, ej = 0;
    const double *ti = nullptr, *tj = nullptr;
    double cb = 0, ce = 0;
    if (active) {
        uint32_t lo = 0, hi = nb;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (step_off[mid] <= p) lo = mid;
            else hi = mid;
        }
        b = lo;
        const double2 cbe = cd_bounds[s_first + b];
        cb = cbe.x;
        ce = cbe.y;
        const uint2 pr = pairs[p];
        i = pr.x;
        j = pr.y;
        ti = pj.time + pj.time_off[i];
        tj = pj.time + pj.time_off[j];
        // The segment ranges found by the AABB pass (step_range over the
        // same step bounds).
        const uint2 ri = srange[uint64_t(b) * pj.n_objs + i], rj = srange[uint64_t(b) * pj.n_objs + j];
        it_i = ri.x, ei = ri.y;
        it_j = rj.x, ej = rj.y;
    }
    unsigned n_cand = 0;
    uint32_t budget = (ei - it_i) + (ej - it_j);
    // Warp-synchronous loop: every lane iterates until all lanes are done.
    for (;;) {
        bool live = active && it_i != ei && it_j != ej;
        if (live && budget == 0) {
            set_error(st, ERR_NP_INTERVAL, i, j, 0.0, 0.0);
            live = false;
            active = false;
        }
        if (!__any_sync(0xffffffffu, live)) break;
        bool emit = false;
        double ti_e = 0, tj_e = 0;
        if (live) {
            const double si = ti[it_i - 1], sj = tj[it_j - 1];
            ti_e = ti[it_i];
            tj_e = tj[it_j];
            const double lb_i = dmax_ref(cb, si), ub_i = dmin_ref(ce, ti_e);
            const double lb_j = dmax_ref(cb, sj), ub_j = dmin_ref(ce, tj_e);
            emit = ub_i > lb_j && lb_i < ub_j;
        }
        const unsigned long long slot = warp_append(item_count, emit);
        if (emit) {
            ++n_cand;
            if (slot < cap) items[slot] = np_item{i, j, b, it_i, it_j, 0};
        }
        if (live) {
            it_i += (ti_e <= tj_e);
            it_j += (tj_e <= ti_e);
            --budget;
        }
    }
    block_add2(counters + 0, nullptr, n_cand, counters + 1, 0u);
}

// The reference formulation of one item, operation for operation.  Persistent
// grid over the device-side item count: one thread per item, or, for few
// items, one warp.
//
// The filter leaves 1 % of a day's items and 2 % of dense catalogues'.  The
// 11,000 dependent FP64 operations of an item take one thread 63 us however
// few the items, which is 6 % of a small call.  With a warp per item (lane I
// computes translated coefficient I, node I, divided difference I; every
// value by the same operations in the same order, so bit for bit the same)
// they take 19 us; the warp keeps 19 of 32 lanes busy at order 18 and repeats
// the powers, so beyond WARP_ITEMS items, three or four a resident warp, the
// thread per item is faster (13,000 items: 67 against 105 us; 517,000 of
// 60,000 objects x 48 steps at 20 km: 0.65 ms).  That path keeps node values and
// squared distances in a shared-memory column per thread, so that its loops
// over objects, coordinates, nodes and divided differences stay loops (14,000
// instructions unrolled, 0.71 ms).
constexpr int NARROW_T = 64;
constexpr uint64_t WARP_ITEMS = 6144;

// The sub-interval of an item: false (with the reference's error) when it is
// not a valid one.
struct sub_interval {
    double lb_rf, ub_rf, rf_int, di, dj;
    uint64_t gsi, gsj;
    uint32_t flags; // 1 = end of trajectory data, 2 = start
};
__device__ __forceinline__ bool item_interval(const dev_pj &pj, const double2 *__restrict__ cd_bounds,
                                              uint32_t s_first, const np_item &it, sub_interval &v)
{
    const double2 cbe = cd_bounds[s_first + it.b];
    const double cb = cbe.x, ce = cbe.y;
    const double *ti = pj.time + pj.time_off[it.i];
    const double *tj = pj.time + pj.time_off[it.j];
    const double si = ti[it.it_i - 1], sj = tj[it.it_j - 1];
    const double ti_e = ti[it.it_i], tj_e = tj[it.it_j];
    const double lb_i = dmax_ref(cb, si), ub_i = dmin_ref(ce, ti_e);
    const double lb_j = dmax_ref(cb, sj), ub_j = dmin_ref(ce, tj_e);
    v.lb_rf = dmax_ref(lb_i, lb_j);
    v.ub_rf = dmin_ref(ub_i, ub_j);
    v.di = v.lb_rf - si;
    v.dj = v.lb_rf - sj;
    v.rf_int = v.ub_rf - v.lb_rf;
    v.gsi = pj.seg_off[it.i] + it.it_i - 1;
    v.gsj = pj.seg_off[it.j] + it.it_j - 1;
    const uint32_t nsi = pj.nseg[it.i], nsj = pj.nseg[it.j];
    v.flags = 0;
    if ((it.it_i == nsi && ti_e == v.ub_rf) || (it.it_j == nsj && tj_e == v.ub_rf)) v.flags |= 1u;
    if ((it.it_i == 1 && v.lb_rf == ti[0]) || (it.it_j == 1 && v.lb_rf == tj[0])) v.flags |= 2u;
    return isfinite(v.di) && isfinite(v.dj) && isfinite(v.rf_int) && v.di >= 0 && v.dj >= 0 && v.rf_int >= 0;
}

__device__ __forceinline__ void fill_root_item(root_item &q, const np_item &it, const sub_interval &v)
{
    q.i = it.i;
    q.j = it.j;
    q.step = it.b;
    q.flags = v.flags;
    q.lb_rf = v.lb_rf;
    q.rf_int = v.rf_int;
    q.di = v.di;
    q.dj = v.dj;
    q.seg_i = v.gsi;
    q.seg_j = v.gsj;
}

// One item by one warp (OP1 <= 32); shift[k * OP1 + i] = C(i + k, k).  Returns
// whether the item goes to root finding, lane k's f then being coefficient k
// of its squared-distance polynomial.  The pairwise sums run over OP1 terms in
// every lane: a lane with fewer has -0.0 in the others' places, and x + -0.0
// is x, so the tree is the reference's.
template <int OP1>
__device__ __forceinline__ bool narrow_by_warp(const dev_pj &pj, const double *__restrict__ shift,
                                               const double *nodes, const np_item &it, const sub_interval &v,
                                               double thresh2, unsigned long long &n_pruned, double &f,
                                               dev_status *st)
{
    constexpr int n = OP1 - 1;
    constexpr unsigned ALL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31;
    const bool in = lane < OP1;
    const double node = in ? nodes[lane] : 0.0;
    const double x = node * v.rf_int;
    double vi = 0;
    f = 0;
#pragma unroll 1
    for (int r = 0; r < 6; ++r) {
        const int c = r >> 1, o = r & 1; // coordinate, object
        const double delta = o ? v.dj : v.di;
        double tr = in ? __ldg(coef_row<OP1>(pj, o ? v.gsj : v.gsi, c) + lane) : 0.0;
        if (delta != 0) {
            double ap[OP1], t[OP1];
            powers<OP1>(delta, ap);
#pragma unroll
            for (int k = 0; k < OP1; ++k) {
                const double ck = __shfl_down_sync(ALL, tr, k);
                t[k] = lane + k <= n ? (ck * __ldg(shift + k * OP1 + lane)) * ap[k] : -0.0;
            }
            tr = pw<OP1>::reduce(t, add_op{});
        }
        double h = __shfl_sync(ALL, tr, n);
#pragma unroll
        for (int k = n - 1; k >= 0; --k) h = __shfl_sync(ALL, tr, k) + h * x;
        if (o == 0) {
            vi = h;
        } else {
            const double d = vi - h;
            f = (c == 0) ? d * d : f + d * d;
        }
    }
    // Bjorck-Pereyra on the ascending nodes.
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        const double lo = __shfl_up_sync(ALL, f, 1), a_lo = __shfl_up_sync(ALL, x, k + 1);
        if (in && int(lane) > k) f = (f - lo) / (x - a_lo);
    }
#pragma unroll 1
    for (int k = n - 1; k >= 0; --k) {
        const double hi = __shfl_down_sync(ALL, f, 1), ck = __shfl_sync(ALL, x, k);
        if (int(lane) >= k && int(lane) < n) f = f - ck * hi;
    }
    // Cargo-Shisha: lane 0 meets b_k at step k.
    double dp[OP1], t = f;
    powers<OP1>(v.rf_int, dp);
#pragma unroll
    for (int k = 0; k < OP1; ++k)
        if (int(lane) == k) t = (t * dp[k]) / c_binom[n][k];
    double emin = t, emax = t;
#pragma unroll 1
    for (int k = 1; k < OP1; ++k) {
        t = t + __shfl_down_sync(ALL, t, 1);
        emin = hy_min_op{}(emin, t);
        emax = hy_max_op{}(emax, t);
    }
    emin = __shfl_sync(ALL, emin, 0);
    emax = __shfl_sync(ALL, emax, 0);
    if (!isfinite(emin) || !isfinite(emax)) {
        if (lane == 0) set_error(st, ERR_NP_NONFINITE, it.i, it.j, 0, 0);
        return false;
    }
    if (emin < thresh2) return true;
    n_pruned += lane == 0;
    return false;
}

template <int OP1>
__global__ void __launch_bounds__(NARROW_T) k_narrow(dev_pj pj, cheb_nodes cheb, const double *__restrict__ shift,
                                                     const double2 *__restrict__ cd_bounds,
                                                     uint32_t s_first, const np_item *__restrict__ items,
                                                     const unsigned long long *item_count, uint64_t item_cap,
                                                     double thresh2, root_item *__restrict__ rq, uint64_t rq_cap,
                                                     unsigned long long *rq_count, unsigned long long *counters,
                                                     dev_status *st)
{
    __shared__ double vs[OP1][NARROW_T], fs[OP1][NARROW_T], nodes[OP1];
    const unsigned tid = threadIdx.x;
    if (tid < OP1) nodes[tid] = cheb.v[tid];
    __syncthreads();
    const uint64_t n_items = min(*item_count, (unsigned long long)item_cap);
    const uint64_t stride = uint64_t(gridDim.x) * NARROW_T;
    unsigned long long n_pruned = 0;
    if constexpr (OP1 <= 32) {
        if (n_items <= WARP_ITEMS) {
            const unsigned lane = tid & 31;
            const uint64_t nwarps = stride / 32;
            for (uint64_t w = (blockIdx.x * uint64_t(NARROW_T) + tid) / 32; w < n_items; w += nwarps) {
                const np_item it = items[w];
                sub_interval v;
                if (!item_interval(pj, cd_bounds, s_first, it, v)) {
                    if (lane == 0) set_error(st, ERR_NP_INTERVAL, it.i, it.j, 0, 0);
                    continue;
                }
                double f;
                if (!narrow_by_warp<OP1>(pj, shift, nodes, it, v, thresh2, n_pruned, f, st)) continue;
                unsigned long long slot = 0;
                if (lane == 0) slot = atomicAdd(rq_count, 1ull);
                slot = __shfl_sync(0xffffffffu, slot, 0);
                if (slot < rq_cap) {
                    if (lane == 0) fill_root_item(rq[slot], it, v);
                    if (lane < OP1) rq[slot].ptd2[lane] = f;
                }
            }
            warp_add(counters + 1, n_pruned);
            return;
        }
    }
    for (uint64_t base = blockIdx.x * uint64_t(NARROW_T); base < n_items; base += stride) {
        const uint64_t q_idx = base + tid;
        const bool active = q_idx < n_items;
        bool push = false;
        np_item it{};
        sub_interval v{};
        if (active) {
            it = items[q_idx];
            if (!item_interval(pj, cd_bounds, s_first, it, v)) {
                set_error(st, ERR_NP_INTERVAL, it.i, it.j, 0, 0);
            } else {
                const double rf_int = v.rf_int;
#pragma unroll 1
                for (int r = 0; r < 6; ++r) {
                    const int c = r >> 1, o = r & 1; // coordinate, object
                    const double delta = o ? v.dj : v.di;
                    double cf[OP1], tr[OP1];
                    load_row<OP1>(coef_row<OP1>(pj, o ? v.gsj : v.gsi, c), cf);
                    if (delta != 0) translate<OP1>(cf, delta, tr);
                    else
#pragma unroll
                        for (int k = 0; k < OP1; ++k) tr[k] = cf[k];
#pragma unroll 4
                    for (int m = 0; m < OP1; ++m) {
                        const double h = horner<OP1>(tr, nodes[m] * rf_int);
                        if (o == 0) {
                            vs[m][tid] = h;
                        } else {
                            const double d = vs[m][tid] - h;
                            fs[m][tid] = (c == 0) ? d * d : fs[m][tid] + d * d;
                        }
                    }
                }
                // Bjorck-Pereyra on the ascending nodes.
#pragma unroll 1
                for (int k = 0; k < OP1 - 1; ++k) {
                    double hi = fs[OP1 - 1][tid];
#pragma unroll 4
                    for (int jj = OP1 - 1; jj > k; --jj) {
                        const double lo = fs[jj - 1][tid];
                        fs[jj][tid] = (hi - lo) / (nodes[jj] * rf_int - nodes[jj - k - 1] * rf_int);
                        hi = lo;
                    }
                }
#pragma unroll 1
                for (int k = OP1 - 2; k >= 0; --k) {
                    const double ck = nodes[k] * rf_int;
                    double lo = fs[k][tid];
#pragma unroll 4
                    for (int jj = k; jj < OP1 - 1; ++jj) {
                        const double hi = fs[jj + 1][tid];
                        fs[jj][tid] = lo - ck * hi;
                        lo = hi;
                    }
                }
                double e[OP1];
#pragma unroll
                for (int k = 0; k < OP1; ++k) e[k] = fs[k][tid];
                double emin, emax;
                cs_from_translated<OP1>(e, rf_int, emin, emax);
                if (!isfinite(emin) || !isfinite(emax)) {
                    set_error(st, ERR_NP_NONFINITE, it.i, it.j, 0, 0);
                } else if (emin < thresh2) {
                    push = true;
                } else {
                    ++n_pruned;
                }
            }
        }
        const unsigned long long slot = warp_append(rq_count, push);
        if (push && slot < rq_cap) {
            root_item &q = rq[slot];
            fill_root_item(q, it, v);
#pragma unroll 4
            for (int k = 0; k < OP1; ++k) q.ptd2[k] = fs[k][tid];
        }
    }
    warp_add(counters + 1, n_pruned);
}

// ---------------------------------------------------------------- filter
//
// In front of k_narrow, in both forms.  Of the items of a catalogue day 85 %
// have an enclosure that clears the threshold and 15 % go to root finding,
// where all but 1 % turn out to have one minimum, above the threshold.  The
// reference formulation takes 8,921 FP64 operations and 190 divisions for an
// item, and root finding as much again; which of the two outcomes it will
// have can be proven from an FMA-native evaluation of 2,700 operations:
//
// * both objects' segment polynomials are shifted to the sub-interval's
//   midpoint (synthetic division) and subtracted, and the difference is
//   scaled to [-1, 1], where the nodes are symmetric: its even and odd parts
//   give the values at a node and its mirror together.  The squared distances
//   are interpolated in the normalised time s = t / rf_int on the fixed nodes
//   c_m by Bjorck-Pereyra with precomputed reciprocals 1 / (c_j - c_{j-k-1}),
//   and their Bernstein coefficients b_i over [0, 1] come from the difference
//   table of Cargo-Shisha;
// * both formulations interpolate the same polynomial's values on the same
//   nodes, and M bounds how far their Bernstein coefficients can differ by
//   rounding, u = 2^-53 (filter_margins, in filter_margin.cuh):
//   - an object's coordinate at a node: the reference formulation (powers,
//     binomial sums, Horner) is within sum (3k + 8) u |c_k| e^k of its exact
//     value, this one (shift, scaling, even and odd Horner) within sum (4k + 5)
//     u |c_k| e^k, e = delta + rf_int, and 7k + 14 <= 39.2 1.08^k (no base is
//     closer over coefficients that fall off, k about 3, and ones that do not).
//     With P_c the sum of |c_k| (1.08 e)^k over both objects' coordinate c and
//     P^2 = sum P_c^2, the squared distance at node m differs by at most 78.4 u P
//     sqrt(f_m) + 1537 u^2 P^2 + 10 u f_m, and a Bernstein coefficient by
//     node_w[m] times that.  Their sum over the nodes is bounded with
//     F = sum node_w[m] f_m (Cauchy-Schwarz); the weights, together 1.3 times the
//     largest Bernstein coefficient of the Chebyshev polynomial, are largest in
//     the middle, where an encounter is close;
//   - each divided difference has a relative rounding of 4 u here, 3 u there and
//     u (c_j + c_i) / (c_j - c_i) for the nodes c rf_int there; each step from
//     Newton form to monomials four roundings of what it adds up.  All of them
//     are at most linear in the magnitudes of the Newton coefficients; newton[l]
//     is what the l-th one's can do to a Bernstein coefficient;
//   - scaling by 1 / C(n, i) and the difference table: (3n + 5) u sum |f_k|, f_k
//     the monomials' coefficients on [0, 1]; Ms = (6n + 24) u sum |f_k|, part of
//     M, also covers the derivative in root finding: its coefficients (n (n + 12)
//     u sum |f_k|), values (n (3n + 2)) and slope (3 n^3).
//   On segments of a catalogue the first term is nearly all of M, where the
//   coefficients do not fall off the other two are.  A margin measured on the
//   former, 32 u A_n (P sqrt(max f) + max f), lost conjunctions of the latter at
//   orders from 20 on;
// * min b >= threshold^2 + M: the reference prunes the item (counter 1);
// * b_1 - b_0 < -2M - Ms, b_n - b_{n-1} > 2M + Ms, every second difference >
//   4M + 2Ms and min b < threshold^2 - M: the reference keeps the item.  The
//   Bernstein coefficients of its derivative ascend from negative to positive,
//   by steps and with ends that exceed their roundings, so it finds exactly one
//   root, a minimum.  The polynomial is convex with p'' / 2 >= kappa =
//   n (n - 1) / 2 (min second difference - 4M), so p is at least
//   p(s) - p'(s)^2 / (4 kappa) for any s; after a Newton step from the secant of
//   p' that bound is the minimum itself for all purposes.  If it is at least
//   threshold^2 + 2M (with n Ms more for p'), the minimum is discarded
//   (counters 2, 5 and 6) and no trajectory boundary in the item can be below
//   the threshold either;
// * everything else (also values outside the range in which neither
//   formulation can overflow: see filter_range) goes to k_narrow.
//
// So the records and all counters are those of the reference formulation.
//
// Bound by the FP64 pipe, if the coefficients arrive: 960 bytes an item, in
// rows of 160 (order 18).  Loaded by each thread for itself, a 16-byte load of
// a warp touched 32 lines and the load pipe was the bound (31 % of the FP64
// rate).  Here a warp copies its items' rows of one coordinate and object to
// shared memory together (cp.async, consecutive lanes on consecutive bytes of
// a row), reads them back at an odd stride of 16-byte units (conflict-free),
// and has the next rows in flight while it computes.  One object's rows at a
// time, the sums of squares in shared memory between the coordinates and all
// constants as kernel parameters (operands of the instructions instead of
// loads) leave room for 16 warps an SM at order 18 (124 registers; 12 warps
// are 4 % slower, 18 with spills 14 %).  6.38 M items of the 20,000-object day:
// 1.8 ms (2.6 with Horner at every node and both objects' rows, 168
// registers and 12 warps; 0.04 of it are the margin's sums).  With the merge walk and root finding, the plain
// form's narrow phase took 10.4 ms with the reference formulation for every
// item and takes 2.2; 60,000 objects x 48 steps at 20 km, mixed, 11.9 and 4.2.
static_assert(FILTER_MAX_OP1 == MAX_OP1, "tables for every order");
// Reciprocal node differences, row k: 1 / (c_j - c_{j-k-1}), j = k + 1 .. n.
template <int OP1>
struct filter_consts {
    filter_tables t;
    double inv_dd[OP1 * (OP1 - 1) / 2];
};
template <int OP1>
static filter_consts<OP1> make_filter_consts()
{
    filter_consts<OP1> f{};
    const cheb_nodes c = make_cheb_nodes(OP1);
    f.t = make_filter_tables(c.v, OP1);
    int at = 0;
    for (int k = 0; k < OP1 - 1; ++k)
        for (int j = k + 1; j < OP1; ++j) f.inv_dd[at++] = 1.0 / (c.v[j] - c.v[j - k - 1]);
    return f;
}
__host__ __device__ constexpr int filter_row(int op1, int k) { return k * (op1 - 1) - k * (k - 1) / 2; } // start of row k

// One warp a CTA: the work is per warp.
template <int OP1>
struct filter_shape {
    static constexpr int UNITS = row_ld(OP1) / 2; // 16-byte units of a row
    static constexpr int STRIDE = UNITS | 1;      // odd: conflict-free 16-byte reads
    static constexpr int GROUPS = 32 / UNITS;     // rows copied per instruction
    static constexpr int CTAS = OP1 <= 20 ? 16 : 8;
};

template <int OP1>
__global__ void __launch_bounds__(32, filter_shape<OP1>::CTAS)
    k_narrow_filter(dev_pj pj, const filter_consts<OP1> K, const double2 *__restrict__ cd_bounds,
                    uint32_t s_first, const np_item *__restrict__ items, const unsigned long long *item_count,
                    uint64_t item_cap, double thresh2, np_item *__restrict__ surv, uint64_t surv_cap,
                    unsigned long long *surv_count, unsigned long long *counters)
{
    using F = filter_shape<OP1>;
    constexpr int n = OP1 - 1;
    __shared__ __align__(16) double2 rows[32 * F::STRIDE];
    __shared__ double fs[OP1][32];
    __shared__ const double2 *base[2][32];
    const unsigned lane = threadIdx.x;
    const uint64_t n_items = min(*item_count, (unsigned long long)item_cap);
    unsigned n_pruned = 0, n_single = 0;
    // The rows of coordinate c and object o of the warp's 32 items, GROUPS
    // rows at a time.
    const unsigned part = lane % F::UNITS, grp = lane / F::UNITS;
    const unsigned dst0 = unsigned(__cvta_generic_to_shared(rows + grp * F::STRIDE + part));
    auto fetch = [&](int o, int c) {
#pragma unroll
        for (int k = 0; k < (32 + F::GROUPS - 1) / F::GROUPS; ++k) {
            const unsigned r = grp + unsigned(k * F::GROUPS);
            if (grp < F::GROUPS && r < 32) {
                const double2 *src = base[o][r] + c * F::UNITS + part;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 dst0 + unsigned(k * F::GROUPS * F::STRIDE * 16)),
                             "l"(src)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // The fetched row into registers, when it has arrived; afterwards the next
    // rows may land.
    auto row_in = [&](double(&c)[OP1]) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        const double2 *r = rows + lane * F::STRIDE;
#pragma unroll
        for (int k = 0; k < OP1 / 2; ++k) {
            const double2 v = r[k];
            c[2 * k] = v.x;
            c[2 * k + 1] = v.y;
        }
        if (OP1 & 1) c[OP1 - 1] = r[OP1 / 2].x;
        __syncwarp();
    };
    // Shift to the origin a; returns sum |c_k| (1.08 e)^k first.
    auto shifted = [](double(&c)[OP1], double a, double e) {
        e *= 1.08;
        double p = fabs(c[n]);
#pragma unroll
        for (int k = n - 1; k >= 0; --k) p = fma(p, e, fabs(c[k]));
#pragma unroll
        for (int i = 0; i < n; ++i)
#pragma unroll
            for (int k = n - 1; k >= i; --k) c[k] = fma(a, c[k + 1], c[k]);
        return p;
    };
    for (uint64_t b0 = blockIdx.x * uint64_t(32); b0 < n_items; b0 += uint64_t(gridDim.x) * 32) {
        const uint64_t q_idx = b0 + lane;
        const bool active = q_idx < n_items;
        np_item it{};
        double rf_int = 0, di = 0, dj = 0;
        uint64_t gsi = 0, gsj = 0;
        bool usable = false;
        if (active) {
            it = items[q_idx];
            const double2 cbe = cd_bounds[s_first + it.b];
            const double cb = cbe.x, ce = cbe.y;
            const double *ti = pj.time + pj.time_off[it.i];
            const double *tj = pj.time + pj.time_off[it.j];
            const double si = ti[it.it_i - 1], sj = tj[it.it_j - 1];
            const double lb_i = dmax_ref(cb, si), ub_i = dmin_ref(ce, ti[it.it_i]);
            const double lb_j = dmax_ref(cb, sj), ub_j = dmin_ref(ce, tj[it.it_j]);
            const double lb_rf = dmax_ref(lb_i, lb_j);
            const double ub_rf = dmin_ref(ub_i, ub_j);
            di = lb_rf - si;
            dj = lb_rf - sj;
            rf_int = ub_rf - lb_rf;
            usable = di >= 0 && dj >= 0 && rf_int >= K.t.rf_lo && rf_int <= K.t.rf_hi;
            gsi = pj.seg_off[it.i] + it.it_i - 1;
            gsj = pj.seg_off[it.j] + it.it_j - 1;
        }
        // Rows of lanes without an item are segment 0's: copied, not used.
        base[0][lane] = reinterpret_cast<const double2 *>(coef_row<OP1>(pj, gsi, 0));
        base[1][lane] = reinterpret_cast<const double2 *>(coef_row<OP1>(pj, gsj, 0));
        __syncwarp();
        fetch(0, 0);
        double P2 = 0;
        const double h = 0.5 * rf_int;
#pragma unroll 1
        for (int c = 0; c < 3; ++c) {
            double g[OP1], t[OP1];
            row_in(g);
            fetch(1, c);
            double pc = shifted(g, di + h, di + rf_int);
            row_in(t);
            if (c < 2) fetch(0, c + 1);
            pc += shifted(t, dj + h, dj + rf_int);
            P2 = fma(pc, pc, P2);
            double hp = h;
            g[0] = g[0] - t[0];
#pragma unroll
            for (int k = 1; k < OP1; ++k) {
                g[k] = (g[k] - t[k]) * hp;
                hp *= h;
            }
            // Node n - m and its mirror m: even part +- x times odd part.
            auto add = [&](int m, double d) { fs[m][lane] = (c == 0) ? d * d : fma(d, d, fs[m][lane]); };
            constexpr int EV = n & ~1, OD = (n - 1) | 1;
#pragma unroll
            for (int m = 0; m < OP1 / 2; ++m) {
                double even = g[EV], odd = g[OD];
#pragma unroll
                for (int k = EV - 2; k >= 0; k -= 2) even = fma(even, K.t.y[m], g[k]);
#pragma unroll
                for (int k = OD - 2; k >= 1; k -= 2) odd = fma(odd, K.t.y[m], g[k]);
                add(n - m, fma(K.t.x[m], odd, even));
                add(m, fma(-K.t.x[m], odd, even));
            }
            if (OP1 & 1) add(n / 2, g[0]);
        }
        double f[OP1], F_s = 0;
#pragma unroll
        for (int m = 0; m < OP1; ++m) {
            f[m] = fs[m][lane];
            F_s = fma(K.t.node_w[m], f[m], F_s);
        }
        // Bjorck-Pereyra on the normalised nodes.
#pragma unroll
        for (int k = 0; k < n; ++k)
#pragma unroll
            for (int jj = n; jj > k; --jj) f[jj] = (f[jj] - f[jj - 1]) * K.inv_dd[filter_row(OP1, k) + jj - k - 1];
        double M = 1e-250;
#pragma unroll
        for (int k = 0; k < OP1; ++k) M = fma(K.t.newton[k], fabs(f[k]), M);
#pragma unroll
        for (int k = n - 1; k >= 0; --k)
#pragma unroll
            for (int jj = k; jj < n; ++jj) f[jj] = fma(-K.t.node[k], f[jj + 1], f[jj]);
        double Ms = 0;
#pragma unroll
        for (int k = 0; k < OP1; ++k) Ms += fabs(f[k]);
        Ms *= K.t.mono;
        // Bernstein coefficients over s in [0, 1], each one's first and
        // second differences as it appears.
        double e[OP1];
#pragma unroll
        for (int k = 0; k < OP1; ++k) e[k] = f[k] * K.t.inv_binom[k];
        double emin = e[0], b1 = e[0], d_first = 0, d_prev = 0, dd_min = INFINITY;
#pragma unroll
        for (int k = 1; k < OP1; ++k) {
#pragma unroll
            for (int jj = 0; jj + k < OP1; ++jj) e[jj] = e[jj] + e[jj + 1];
            emin = e[0] < emin ? e[0] : emin;
            const double d = e[0] - b1;
            if (k == 1) {
                d_first = d;
            } else {
                const double dd = d - d_prev;
                dd_min = dd < dd_min ? dd : dd_min;
            }
            d_prev = d;
            b1 = e[0];
        }
        auto root_up = [](double x) { return double(__fsqrt_ru(__double2float_ru(x))); };
        M += Ms + fma(K.t.value * root_up(F_s), root_up(P2), fma(K.t.square, F_s, K.t.norm * P2));
        // F is NaN or too large for non-finite values (the comparisons above
        // would drop a NaN); every node_w is above 1.
        usable = usable && F_s <= 1e30 && P2 <= 1e30;
        const bool pruned = usable && emin >= thresh2 + M;
        bool single = false;
        if (usable && !pruned && emin < thresh2 - M && d_first < -2 * M - Ms && d_prev > 2 * M + Ms
            && dd_min > 4 * M + 2 * Ms) {
            const double kappa = 0.5 * (double(n) * (n - 1)) * (dd_min - 4 * M);
            double s = d_first / (d_first - d_prev);
            double p = 0, p1 = 0;
#pragma unroll 1
            for (int r = 0; r < 2; ++r) {
                double p2 = 0;
                p = f[n], p1 = 0;
#pragma unroll
                for (int k = n - 1; k >= 0; --k) {
                    p2 = fma(p2, s, p1);
                    p1 = fma(p1, s, p);
                    p = fma(p, s, f[k]);
                }
                if (r == 0) s = fmin(fmax(s - p1 / (2 * p2), 0.0), 1.0);
            }
            p1 = fabs(p1) + n * Ms;
            single = p - p1 * p1 / (4 * kappa) >= thresh2 + 2 * M;
        }
        n_pruned += pruned;
        n_single += single;
        const bool push = active && !pruned && !single;
        const unsigned long long slot = warp_append(surv_count, push);
        if (push && slot < surv_cap) surv[slot] = it;
    }
    n_pruned = __reduce_add_sync(0xffffffffu, n_pruned);
    n_single = __reduce_add_sync(0xffffffffu, n_single);
    if (lane == 0) {
        if (n_pruned) atomicAdd(counters + 1, (unsigned long long)n_pruned);
        if (n_single)
            for (int k : {2, 5, 6, 7}) atomicAdd(counters + k, (unsigned long long)n_single);
    }
}

// Screen ahead of the filter (mixed form): a rigorous lower bound on the
// distance over the item's sub-interval from linear models of both objects.
// For each object, on the portion of its segment inside the step, Taylor's
// theorem gives x(tm + s) = x(tm) + x'(tm) s + R(s) with |R(s)| <= |A| s^2 / 2,
// A_c = sum_k k (k - 1) |c_k| t_max^(k-2) bounding |x_c''| (t_max the portion
// end in the segment's own time).  The relative linear model over the item
// is D0 + Dv s, |s| <= h (half the sub-interval), so
//   min |dr(t)| >= min_{|s| <= h} |D0 + Dv s| - (|A_i| si^2 + |A_j| sj^2) / 2,
// si, sj the largest distance of the item from each model point; the first
// term is the closest approach of a straight line, in closed form.  Items
// whose bound clears the threshold (relative slack 1e-6) cannot hold a
// conjunction: they are dropped and counted as pruned by the distance
// check; the rest go on to k_narrow_filter, compacted so its warps stay full.
//
// The models come from the mixed AABB pass (32 bytes each, FP32: position,
// velocity at the portion midpoint, |A| rounded up) for the first and second
// segments of each object in the step; their FP32 rounding is added to the
// margin.  Items on a later segment (objects with segments shorter than half
// a step) build the models here from the coefficients, at the item midpoint.
// The distance screen of one item (above): false when the item cannot hold
// a conjunction (then *pruned is set).
template <int OP1>
__device__ __forceinline__ bool screen_keeps(const dev_pj &pj, const double2 *__restrict__ cd_bounds,
                                             uint32_t s_first, const np_item &it, double thresh,
                                             const float4 *__restrict__ scr, bool &pruned)
{
    constexpr int n = OP1 - 1;
    const uint64_t N = pj.n_objs;
    bool push = false;
    const double2 cbe = cd_bounds[s_first + it.b];
    const double cb = cbe.x, ce = cbe.y;
    const double *ti = pj.time + pj.time_off[it.i];
    const double *tj = pj.time + pj.time_off[it.j];
    const double si = ti[it.it_i - 1], sj = tj[it.it_j - 1];
    const double ti_e = ti[it.it_i], tj_e = tj[it.it_j];
    const double lb_i = dmax_ref(cb, si), ub_i = dmin_ref(ce, ti_e);
    const double lb_j = dmax_ref(cb, sj), ub_j = dmin_ref(ce, tj_e);
    const double lb_rf = dmax_ref(lb_i, lb_j), ub_rf = dmin_ref(ub_i, ub_j);
    const double di = lb_rf - si, dj = lb_rf - sj, rf_int = ub_rf - lb_rf;
    push = true;
    if (isfinite(di) && isfinite(dj) && isfinite(rf_int) && di >= 0 && dj >= 0 && rf_int >= 0) {
        const double h = rf_int / 2;
        // Slot of each object's model: 0 for the step's first
        // overlapping segment, 1 for the second, none after that.
        int slot_i = -1, slot_j = -1;
        if (scr) {
            if (it.it_i == 1 || si <= cb) slot_i = 0;
            else if (it.it_i == 2 || ti[it.it_i - 2] <= cb) slot_i = 1;
            if (it.it_j == 1 || sj <= cb) slot_j = 0;
            else if (it.it_j == 2 || tj[it.it_j - 2] <= cb) slot_j = 1;
        }
        double P[2][3], V[2][3], A[2], off[2], emod = 0;
        if (slot_i >= 0 && slot_j >= 0) {
            const float4 *m[2] = {scr + (uint64_t(it.b) * N + it.i) * 4 + 2 * slot_i,
                                  scr + (uint64_t(it.b) * N + it.j) * 4 + 2 * slot_j};
            const double tm[2] = {((lb_i - si) + (ub_i - si)) / 2, ((lb_j - sj) + (ub_j - sj)) / 2};
            const double dd[2] = {di, dj};
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const float4 a = m[o][0], b = m[o][1];
                P[o][0] = a.x, P[o][1] = a.y, P[o][2] = a.z;
                V[o][0] = a.w, V[o][1] = b.x, V[o][2] = b.y;
                A[o] = b.z;
                off[o] = dd[o] + h - tm[o]; // item centre from the model point
                // FP32 storage: |fl(x) - x| <= 2^-24 |x| for each value.
                emod += 1.1920928955078125e-07
                        * (sqrt(P[o][0] * P[o][0] + P[o][1] * P[o][1] + P[o][2] * P[o][2])
                           + sqrt(V[o][0] * V[o][0] + V[o][1] * V[o][1] + V[o][2] * V[o][2])
                                 * (fabs(off[o]) + h));
            }
        } else {
            // Models at the item midpoint from the coefficients.
            const double tmi = di + h, tmj = dj + h, tei = di + rf_int, tej = dj + rf_int;
            const double *ci_base = coef_row<OP1>(pj, pj.seg_off[it.i] + it.it_i - 1, 0);
            const double *cj_base = coef_row<OP1>(pj, pj.seg_off[it.j] + it.it_j - 1, 0);
            double ai2 = 0, aj2 = 0;
#pragma unroll 1
            for (int c = 0; c < 3; ++c) {
                double ci[OP1], cj[OP1];
                load_row<OP1>(ci_base + c * row_ld(OP1), ci);
                load_row<OP1>(cj_base + c * row_ld(OP1), cj);
                double pi = ci[n], pj_ = cj[n], vi = 0, vj = 0;
                double ai = double(n) * (n - 1) * fabs(ci[n]), aj = double(n) * (n - 1) * fabs(cj[n]);
#pragma unroll
                for (int k = n - 1; k >= 0; --k) {
                    vi = fma(vi, tmi, pi);
                    vj = fma(vj, tmj, pj_);
                    pi = fma(pi, tmi, ci[k]);
                    pj_ = fma(pj_, tmj, cj[k]);
                    if (k >= 2) {
                        ai = fma(ai, tei, double(k) * (k - 1) * fabs(ci[k]));
                        aj = fma(aj, tej, double(k) * (k - 1) * fabs(cj[k]));
                    }
                }
                P[0][c] = pi, P[1][c] = pj_, V[0][c] = vi, V[1][c] = vj;
                ai2 = fma(ai, ai, ai2);
                aj2 = fma(aj, aj, aj2);
            }
            A[0] = sqrt(ai2) * (1.0 + 1e-12);
            A[1] = sqrt(aj2) * (1.0 + 1e-12);
            off[0] = off[1] = 0;
        }
        double d0[3], dv[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            d0[c] = fma(V[0][c], off[0], P[0][c]) - fma(V[1][c], off[1], P[1][c]);
            dv[c] = V[0][c] - V[1][c];
        }
        const double vv = dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2];
        const double rv = d0[0] * dv[0] + d0[1] * dv[1] + d0[2] * dv[2];
        double sst = vv > 0 ? -rv / vv : 0;
        sst = fmin(fmax(sst, -h), h);
        const double e0 = fma(dv[0], sst, d0[0]), e1 = fma(dv[1], sst, d0[1]), e2 = fma(dv[2], sst, d0[2]);
        const double dlin = sqrt(e0 * e0 + e1 * e1 + e2 * e2);
        const double s_i = fabs(off[0]) + h, s_j = fabs(off[1]) + h;
        const double R = 0.5 * (A[0] * s_i * s_i + A[1] * s_j * s_j);
        const double slack =
            1e-6 * (thresh + sqrt(d0[0] * d0[0] + d0[1] * d0[1] + d0[2] * d0[2]) + sqrt(vv) * h + R) + emod;
        if (isfinite(dlin) && isfinite(R) && isfinite(slack) && dlin - R > thresh + slack) {
            push = false;
            pruned = true;
        }
    }
    return push;
}

// The mixed form's merge walk (k_items) with the distance screen inside: each item of the
// merge walk is screened as it is found and only the items the screen keeps
// are appended (to the filter's queue), so the day's 6.4 M items are
// never written out and read back.  Counters: every item (counter 0, and
// *item_count), the pruned ones (counter 1).
template <int OP1>
__global__ void __launch_bounds__(128, 6) k_items_screen(const dev_pj pj, const double2 *__restrict__ cd_bounds,
                                                         uint32_t s_first, uint32_t nb, const uint2 *__restrict__ pairs,
                                                         const uint64_t *__restrict__ step_off,
                                                         const uint2 *__restrict__ srange, double thresh,
                                                         const float4 *__restrict__ scr, np_item *__restrict__ cand,
                                                         uint64_t cand_cap, unsigned long long *cand_count,
                                                         unsigned long long *item_count,
                                                         unsigned long long *counters, dev_status *st)
{
    const uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    const uint64_t n_pairs = step_off[nb];
    bool active = p < n_pairs;
    uint32_t b = 0, i = 0, j = 0, it_i = 0, it_j = 0, ei = 0, ej = 0;
    const double *ti = nullptr, *tj = nullptr;
    double cb = 0, ce = 0;
    if (active) {
        uint32_t lo = 0, hi = nb;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (step_off[mid] <= p) lo = mid;
            else hi = mid;
        }
        b = lo;
        const double2 cbe = cd_bounds[s_first + b];
        cb = cbe.x;
        ce = cbe.y;
        const uint2 pr = pairs[p];
        i = pr.x;
        j = pr.y;
        ti = pj.time + pj.time_off[i];
        tj = pj.time + pj.time_off[j];
        const uint2 ri = srange[uint64_t(b) * pj.n_objs + i], rj = srange[uint64_t(b) * pj.n_objs + j];
        it_i = ri.x, ei = ri.y;
        it_j = rj.x, ej = rj.y;
    }
    unsigned n_items = 0, n_pruned = 0; // a thread has fewer than 2^32 items
    uint32_t budget = (ei - it_i) + (ej - it_j);
    // Warp-synchronous loop as in k_items (bounded the same way).
    for (;;) {
        bool live = active && it_i != ei && it_j != ej;
        if (live && budget == 0) {
            set_error(st, ERR_NP_INTERVAL, i, j, 0.0, 0.0);
            live = false;
            active = false;
        }
        if (!__any_sync(0xffffffffu, live)) break;
        bool emit = false;
        double ti_e = 0, tj_e = 0;
        if (live) {
            const double si = ti[it_i - 1], sj = tj[it_j - 1];
            ti_e = ti[it_i];
            tj_e = tj[it_j];
            const double lb_i = dmax_ref(cb, si), ub_i = dmin_ref(ce, ti_e);
            const double lb_j = dmax_ref(cb, sj), ub_j = dmin_ref(ce, tj_e);
            emit = ub_i > lb_j && lb_i < ub_j;
        }
        bool keep = false;
        const np_item it{i, j, b, it_i, it_j, 0};
        if (emit) {
            ++n_items;
            bool pruned = false;
            keep = screen_keeps<OP1>(pj, cd_bounds, s_first, it, thresh, scr, pruned);
            n_pruned += pruned;
        }
        const unsigned long long slot = warp_append(cand_count, keep);
        if (keep && slot < cand_cap) cand[slot] = it;
        if (live) {
            it_i += (ti_e <= tj_e);
            it_j += (tj_e <= ti_e);
            --budget;
        }
    }
    block_add2(counters + 0, item_count, n_items, counters + 1, n_pruned);
}

template <int OP1>
static void items_screen_t(const dev_pj &pj, const double2 *cdb, uint32_t s_first, uint32_t nb, const uint2 *pairs,
                           const uint64_t *step_off, const uint2 *srange, uint64_t n_pairs, double thresh,
                           const float4 *scr, np_item *cand, uint64_t cand_cap, unsigned long long *cand_count,
                           unsigned long long *item_count, unsigned long long *counters, dev_status *st,
                           cudaStream_t stream)
{
    const unsigned bs = 128;
    const unsigned g = unsigned((n_pairs + bs - 1) / bs);
    if (g == 0) return;
    k_items_screen<OP1><<<g, bs, 0, stream>>>(pj, cdb, s_first, nb, pairs, step_off, srange, thresh, scr, cand,
                                               cand_cap, cand_count, item_count, counters, st);
}

void launch_items_screen(const dev_pj &pj, const double2 *cdb, uint32_t s_first, uint32_t nb, const uint2 *pairs,
                         const uint64_t *step_off, const uint2 *srange, uint64_t n_pairs, double thresh,
                         const float4 *scr, np_item *cand, uint64_t cand_cap, unsigned long long *cand_count,
                         unsigned long long *item_count, unsigned long long *counters, dev_status *st,
                         cudaStream_t stream)
{
    switch (pj.op1) {
#define X(K)                                                                                                         \
    case K:                                                                                                            \
        items_screen_t<K>(pj, cdb, s_first, nb, pairs, step_off, srange, n_pairs, thresh, scr, cand, cand_cap,        \
                          cand_count, item_count, counters, st, stream);                                               \
        break;
        MZB_FOR_EACH_OP1(X)
#undef X
    default:
        break;
    }
}

// -------------------------------------------------------------- k_roots

constexpr int WL_CAP = 251; // the reference throws once its list exceeds 250

__device__ __forceinline__ int sgn(double v) { return (0. < v) - (v < 0.); }

__device__ __forceinline__ bool tol_ok(double a, double b)
{
    return fabs(a - b) <= (4 * 2.220446049250313e-16) * fmin(fabs(a), fabs(b));
}

__device__ double secant_step(double a, double b, double fa, double fb)
{
    const double e5 = 5 * 2.220446049250313e-16;
    const double c = a - (fa / (fb - fa)) * (b - a);
    if (c <= a + fabs(a) * e5 || c >= b - fabs(b) * e5) return (a + b) / 2;
    return c;
}

__device__ double guarded_div(double num, double den, double fallback)
{
    if (fabs(den) < 1 && fabs(den * 1.7976931348623157e308) <= fabs(num)) return fallback;
    return num / den;
}

__device__ double newton_quadratic(double a, double b, double d, double fa, double fb, double fd, int k)
{
    const double big = 1.7976931348623157e308;
    const double f_ab = guarded_div(fb - fa, b - a, big);
    double f_abd = guarded_div(fd - fb, d - b, big);
    f_abd = guarded_div(f_abd - f_ab, d - a, 0);
    if (f_abd == 0) return secant_step(a, b, fa, fb);
    double c = (sgn(f_abd) * sgn(fa) > 0) ? a : b;
    for (int i = 0; i < k; ++i)
        c -= guarded_div(fa + (f_ab + f_abd * (c - b)) * (c - a), f_ab + f_abd * (2 * c - a - b), 1 + c - a);
    if (c <= a || c >= b) c = secant_step(a, b, fa, fb);
    return c;
}

__device__ double inverse_cubic(double a, double b, double d, double e, double fa, double fb, double fd, double fe)
{
    const double q11 = (d - e) * fd / (fe - fd);
    const double q21 = (b - d) * fb / (fd - fb);
    const double q31 = (a - b) * fa / (fb - fa);
    const double d21 = (b - d) * fd / (fd - fb);
    const double d31 = (a - b) * fb / (fb - fa);
    const double q22 = (d21 - q11) * fb / (fe - fb);
    const double q32 = (d31 - q21) * fa / (fd - fa);
    const double d32 = (d31 - q21) * fd / (fd - fa);
    const double q33 = (d32 - q22) * fa / (fe - fa);
    double c = q31 + q32 + q33 + a;
    if (c <= a || c >= b) c = newton_quadratic(a, b, d, fa, fb, fd, 3);
    return c;
}

__device__ bool near_equal_values(double fa, double fb, double fd, double fe)
{
    const double m = 2.2250738585072014e-308 * 32;
    return fabs(fa - fb) < m || fabs(fa - fd) < m || fabs(fa - fe) < m || fabs(fb - fd) < m || fabs(fb - fe) < m
           || fabs(fd - fe) < m;
}

constexpr int MAX_ROOTS = 2 * MAX_OP1;

// ---- Compile-time-order building blocks of the minimum search.

// Taylor shift by 1 (heyoka poly_translate_1): out_I = sum_{k >= I} C(k, I) in_k,
// pairwise summed in k order.
template <int OP1, int I>
__device__ __forceinline__ double shift1_coef(const double (&in)[OP1])
{
    constexpr int M = OP1 - I;
    double t[M];
#pragma unroll
    for (int k = 0; k < M; ++k) t[k] = c_binom[I + k][I] * in[I + k];
    return pw<M>::reduce(t, add_op{});
}
template <int OP1, int... I>
__device__ __forceinline__ void shift1_impl(const double (&in)[OP1], double (&out)[OP1],
                                            std::integer_sequence<int, I...>)
{
    ((out[I] = shift1_coef<OP1, I>(in)), ...);
}
template <int OP1>
__device__ __forceinline__ void shift1(const double (&in)[OP1], double (&out)[OP1])
{
    shift1_impl<OP1>(in, out, std::make_integer_sequence<int, OP1>{});
}

// Descartes sign changes of the coefficients, zeros skipped.
template <int OP1>
__device__ __forceinline__ int sign_changes_t(const double (&c)[OP1])
{
    int cnt = 0, prev = 0;
#pragma unroll
    for (int k = 0; k < OP1; ++k) {
        const int s = sgn(c[k]);
        cnt += (s != 0 && prev != 0 && s != prev);
        prev = (s != 0) ? s : prev;
    }
    return cnt;
}

// First derivative of a (poly_utils.cpp poly_eval_1).
template <int OP1>
__device__ __forceinline__ double poly_eval_1_t(const double (&a)[OP1], double x)
{
    constexpr int n = OP1 - 1;
    double r = a[n] * n;
#pragma unroll
    for (int i = 1; i < n; ++i) r = a[n - i] * (n - i) + r * x;
    return r;
}

// Fast exclusion: interval Horner over [0, h]; true = no root there.
template <int OP1>
__device__ __forceinline__ bool fex_excludes_t(const double (&p)[OP1], double h)
{
    constexpr int n = OP1 - 1;
    double lo = p[n], hi = p[n];
#pragma unroll
    for (int o = 1; o <= n; ++o) {
        const double a = lo * h, b = hi * h;
        const double plo = fmin(0., fmin(a, b)), phi = fmax(0., fmax(a, b));
        lo = p[n - o] + plo;
        hi = p[n - o] + phi;
    }
    return lo > 0 || hi < 0;
}

// ---- TOMS 748 (Alefeld, Potra, Shi 1995, Algorithm 4.2) on st.f, which
// evaluates the polynomial and counts its calls in st.evals.
template <int OP1>
struct toms_t {
    const double (&p)[OP1];
    int evals;
    __device__ double f(double x)
    {
        ++evals;
        return horner<OP1>(p, x);
    }
};

// Shrink [a, b] around c (paper: BRACKT), keeping c off the endpoints.
template <typename ST>
__device__ void bracket_at_t(ST &st, double &a, double &b, double c, double &fa, double &fb, double &d, double &fd)
{
    const double t = 2 * 2.220446049250313e-16;
    if ((b - a) < 2 * t * a) c = a + (b - a) / 2;
    else if (c <= a + fabs(a) * t) c = a + fabs(a) * t;
    else if (c >= b - fabs(b) * t) c = b - fabs(b) * t;
    const double fc = st.f(c);
    if (fc == 0) {
        a = c;
        fa = 0;
        d = 0;
        fd = 0;
        return;
    }
    if (sgn(fa) * sgn(fc) < 0) {
        d = b;
        fd = fb;
        b = c;
        fb = fc;
    } else {
        d = a;
        fd = fa;
        a = c;
        fa = fc;
    }
}

// Returns the flag (0 ok, 33 = EDOM for a non-bracketing interval, -1 for an
// exhausted budget of 100 evaluations) and the root in *root.
template <typename ST>
__device__ int toms748_t(ST &st, double lo, double hi, double *root)
{
    constexpr int budget = 100;
    double a = lo, b = hi;
    double fa = st.f(a), fb = st.f(b);
    if (!(a < b)) return 33;
    if (tol_ok(a, b) || fa == 0 || fb == 0) {
        if (fa == 0) b = a;
        else if (fb == 0) a = b;
        *root = a / 2 + b / 2;
        return 0;
    }
    if (sgn(fa) * sgn(fb) > 0) return 33;
    double d = 0, fd = 0, e = 1e5, fe = 1e5;
#define MZB_DONE() (st.evals >= budget || fa == 0 || tol_ok(a, b))
    bracket_at_t(st, a, b, secant_step(a, b, fa, fb), fa, fb, d, fd);
    if (!MZB_DONE()) {
        const double c = newton_quadratic(a, b, d, fa, fb, fd, 2);
        e = d;
        fe = fd;
        bracket_at_t(st, a, b, c, fa, fb, d, fd);
    }
    while (!MZB_DONE()) {
        const double a0 = a, b0 = b;
        double c = near_equal_values(fa, fb, fd, fe) ? newton_quadratic(a, b, d, fa, fb, fd, 2)
                                                     : inverse_cubic(a, b, d, e, fa, fb, fd, fe);
        e = d;
        fe = fd;
        bracket_at_t(st, a, b, c, fa, fb, d, fd);
        if (MZB_DONE()) break;
        c = near_equal_values(fa, fb, fd, fe) ? newton_quadratic(a, b, d, fa, fb, fd, 3)
                                              : inverse_cubic(a, b, d, e, fa, fb, fd, fe);
        bracket_at_t(st, a, b, c, fa, fb, d, fd);
        if (MZB_DONE()) break;
        double u, fu;
        if (fabs(fa) < fabs(fb)) u = a, fu = fa;
        else u = b, fu = fb;
        c = u - 2 * (fu / (fb - fa)) * (b - a);
        if (fabs(c - u) > (b - a) / 2) c = a + (b - a) / 2;
        e = d;
        fe = fd;
        bracket_at_t(st, a, b, c, fa, fb, d, fd);
        if (MZB_DONE()) break;
        if ((b - a) < 0.5 * (b0 - a0)) continue;
        e = d;
        fe = fd;
        bracket_at_t(st, a, b, a + (b - a) / 2, fa, fb, d, fd);
    }
#undef MZB_DONE
    if (fa == 0) b = a;
    else if (fb == 0) a = b;
    *root = a / 2 + b / 2;
    if (st.evals >= budget && !(fa == 0 || tol_ok(a, b))) return -1;
    return 0;
}

// State vectors at tm for one object's segment translated by delta
// (add_conjunction, narrow.cpp:542-575).
template <int OP1>
__device__ void states_at_t(const dev_pj &pj, uint64_t gseg, double delta, double tm, double *r, double *v)
{
#pragma unroll 1
    for (int var = 0; var < 6; ++var) {
        double c[OP1], t[OP1];
        load_row<OP1>(coef_row<OP1>(pj, gseg, var), c);
        double x;
        if (delta != 0) {
            translate<OP1>(c, delta, t);
            x = horner<OP1>(t, tm);
        } else {
            x = horner<OP1>(c, tm);
        }
        if (var < 3) r[var] = x;
        else v[var - 3] = x;
    }
}

// ---- One item by one warp (OP1 <= 32), for launches with few items.
//
// One thread takes 45 to 70 us for an item however few there are: a chain of
// Taylor shifts, evaluations and, for a conjunction, twelve translated
// polynomials one after the other.  Here lane I computes coefficient I of a
// shift, lanes 0 to 11 one state variable each, and all lanes run the scalar
// part (fast exclusion, TOMS 748) on coefficients in shared memory; every
// value comes from the same operations in the same order.  52 items 46 -> 23
// us, 2,700 items 83 -> 46, 5,000 items 89 -> 68; at order 25 2,200 items 133 ->
// 58 us, 6,400 items 136 -> 141.  Beyond two items a resident warp (4,736 of
// them) the thread per item is as fast and keeps all lanes busy (11,000 items:
// 79 against 95 us).
constexpr uint64_t ROOTS_WARP_ITEMS = 4096;
constexpr int ROOTS_T = 128;

template <int OP1>
struct roots_smem {
    double pt[OP1], d[OP1], sp[OP1]; // dist^2, its derivative, the derivative on [0, 1]
    double roots[MAX_ROOTS], isol[OP1 + 1][2];
};

__device__ __noinline__ double horner_smem(const double *p, int n, double x)
{
    double r = p[n];
#pragma unroll 4
    for (int k = n - 1; k >= 0; --k) r = p[k] + r * x;
    return r;
}
struct toms_smem {
    const double *p;
    int n, evals;
    __device__ double f(double x)
    {
        ++evals;
        return horner_smem(p, n, x);
    }
};

// Taylor shift by 1 of the polynomial whose coefficient I lane I holds (see
// narrow_by_warp for the table and the sums).
template <int OP1>
__device__ __noinline__ double shift1_by_warp(const double *__restrict__ shift, double c)
{
    constexpr int n = OP1 - 1;
    const unsigned lane = threadIdx.x & 31;
    double t[OP1];
#pragma unroll
    for (int k = 0; k < OP1; ++k) {
        const double ck = __shfl_down_sync(0xffffffffu, c, k);
        t[k] = lane + k <= n ? __ldg(shift + k * OP1 + lane) * ck : -0.0;
    }
    return pw<OP1>::reduce(t, add_op{});
}

// counts: root findings, fast exclusions, without a root, minima, discarded.
template <int OP1>
__device__ __forceinline__ void roots_by_warp(const dev_pj &pj, const double *__restrict__ shift, const root_item &q,
                                              double thresh2, double *__restrict__ wl, roots_smem<OP1> &S,
                                              conj_out *__restrict__ cq, uint64_t cq_cap,
                                              unsigned long long *cq_count, unsigned (&counts)[5], dev_status *st)
{
    constexpr int n = OP1 - 1;
    constexpr int ENT = OP1 + 2;
    constexpr unsigned ALL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31;
    const bool in = lane < OP1;
    const double rf_int = q.rf_int;
    const double pt = in ? q.ptd2[lane] : 0.0;
    const double d2 = __shfl_down_sync(ALL, pt, 1);
    const double d = lane < unsigned(n) ? (lane + 1u) * d2 : 0.0;
    double fct = 1; // rf_int^lane, by repeated multiplication
#pragma unroll 1
    for (int k = 0; k < n; ++k)
        if (int(lane) > k) fct *= rf_int;
    __syncwarp();
    if (in) {
        S.pt[lane] = pt;
        S.d[lane] = d;
        S.sp[lane] = fct * d;
    }
    __syncwarp();
    int nroots = 0;
    bool failed = false;
    auto error = [&](int code, double x, double y) {
        if (lane == 0) set_error(st, code, q.i, q.j, x, y);
        failed = true;
    };
    auto add_root = [&](double root) {
        if (!isfinite(root)) {
            error(ERR_ROOT_NONFINITE, root, 0);
            return;
        }
        double der = S.d[n] * n;
#pragma unroll 1
        for (int i = 1; i < n; ++i) der = S.d[n - i] * (n - i) + der * root;
        if (!isfinite(der)) {
            error(ERR_ROOT_DER, root, der);
            return;
        }
        if (sgn(der) == 1) {
            if (nroots < MAX_ROOTS) {
                if (lane == 0) S.roots[nroots] = root;
                ++nroots;
            } else {
                error(ERR_ISOLATION, MAX_ROOTS, 0);
            }
        }
    };
    // Fast exclusion: interval Horner over [0, rf_int].
    bool fex;
    {
        double lo = S.d[n], hi = lo;
#pragma unroll 1
        for (int o = 1; o <= n; ++o) {
            const double a = lo * rf_int, b = hi * rf_int;
            const double plo = fmin(0., fmin(a, b)), phi = fmax(0., fmax(a, b));
            lo = S.d[n - o] + plo;
            hi = S.d[n - o] + phi;
        }
        fex = lo > 0 || hi < 0;
    }
    if (!fex) {
        if (lane == 0) wl[0] = 0, wl[1] = 1;
        if (in) wl[2 + lane] = fct * d;
        int wsz = 1, nisol = 0;
        do {
            --wsz;
            __syncwarp();
            const double *ent = wl + uint64_t(wsz) * ENT;
            const double lb = ent[0], ub = ent[1];
            const double cur = in ? ent[2 + lane] : 0.0;
            const bool tail_finite = __all_sync(ALL, lane == 0 || !in || isfinite(cur));
            if (__shfl_sync(ALL, cur, 0) == 0 && tail_finite) add_root(lb * rf_int);
            const double r2 = shift1_by_warp<OP1>(shift, __shfl_sync(ALL, cur, (n - lane) & 31));
            // Descartes sign changes, zeros skipped.
            const int sg = in ? sgn(r2) : 0;
            const unsigned pos = __ballot_sync(ALL, sg > 0), nz = __ballot_sync(ALL, sg != 0);
            const unsigned before = nz & lanemask_lt();
            const bool change = sg != 0 && before && ((pos >> lane) & 1u) != ((pos >> (31 - __clz(before))) & 1u);
            const int nsc = __popc(__ballot_sync(ALL, change));
            if (nsc == 1) {
                if (nisol < OP1 + 1 && lane == 0) S.isol[nisol][0] = lb, S.isol[nisol][1] = ub;
                ++nisol;
            } else if (nsc > 1) {
                if (wsz + 2 > WL_CAP) {
                    error(ERR_ISOLATION, wsz + 2, nisol);
                    break;
                }
                const double L = in ? double(1ull << (n - lane)) * cur : 0.0;
                const double R = shift1_by_warp<OP1>(shift, L);
                const double mid = lb / 2 + ub / 2;
                double *El = wl + uint64_t(wsz) * ENT, *Er = El + ENT;
                __syncwarp(); // every lane has read the entry that El replaces
                if (lane == 0) El[0] = lb, El[1] = mid, Er[0] = mid, Er[1] = ub;
                if (in) El[2 + lane] = L, Er[2 + lane] = R;
                wsz += 2;
            }
            if (wsz > 250 || nisol > n) {
                error(ERR_ISOLATION, wsz, nisol);
                break;
            }
        } while (wsz > 0 && !failed);
        __syncwarp();
        for (int r = 0; r < nisol && !failed; ++r) {
            const double lb = S.isol[r][0];
            double ub = S.isol[r][1];
            if (isfinite(lb) && isfinite(ub) && ub > lb) ub = nextafter(ub, lb);
            double root = 0;
            toms_smem ev{S.sp, n, 0};
            const int flag = toms748_t(ev, lb, ub, &root);
            if (flag == -1) error(ERR_TOMS_ITER, 0, 0);
            else if (flag != 0) error(ERR_TOMS_ERRNO, flag, 0);
            else add_root(root * rf_int);
        }
    }
    if (failed) return;
    __syncwarp();
    ++counts[0];
    counts[1] += fex;
    counts[2] += nroots == 0;
    counts[3] += nroots;
    // The minima below the threshold, then the boundary minima: entry nroots
    // is the end of the data, nroots + 1 their start.
#pragma unroll 1
    for (int r = 0; r < nroots + 2; ++r) {
        double tm = 0.0;
        if (r < nroots) {
            tm = S.roots[r];
        } else if (r == nroots) {
            if (!(q.flags & 1u)) continue;
            tm = nextafter(rf_int, -1.);
            const double dv = horner_smem(S.d, n, tm);
            if (!isfinite(dv)) error(ERR_UB_DER, dv, 0);
            if (!(dv < 0)) continue;
        } else {
            if (!(q.flags & 2u)) continue;
            const double dv = horner_smem(S.d, n, 0.);
            if (!isfinite(dv)) error(ERR_LB_DER, dv, 0);
            if (!(dv > 0)) continue;
        }
        const double m2 = horner_smem(S.pt, n, tm);
        if (!isfinite(m2)) {
            error(r < nroots ? ERR_CONJ_D2 : r == nroots ? ERR_UB_D2 : ERR_LB_D2, m2, 0);
            continue;
        }
        if (!(m2 < thresh2)) {
            counts[4] += r < nroots;
            continue;
        }
        // Lane o * 6 + v: variable v of object o at tm (states_at_t).
        double x = 0;
        if (lane < 12) {
            const unsigned o = lane / 6, v = lane % 6;
            const double delta = o ? q.dj : q.di;
            double c[OP1], t[OP1];
            load_row<OP1>(coef_row<OP1>(pj, o ? q.seg_j : q.seg_i, int(v)), c);
            if (delta != 0) translate<OP1>(c, delta, t);
            else
#pragma unroll
                for (int k = 0; k < OP1; ++k) t[k] = c[k];
            x = horner<OP1>(t, tm);
        }
        const double y = __shfl_down_sync(ALL, x, 6); // the other object's
        const double df = x - y, sq = df * df;
        const double s1 = __shfl_sync(ALL, sq, 1), s2 = __shfl_sync(ALL, sq, 2);
        unsigned long long slot = 0;
        if (lane == 0) slot = atomicAdd(cq_count, 1ull);
        slot = __shfl_sync(ALL, slot, 0);
        if (slot < cq_cap) {
            double *rec = reinterpret_cast<double *>(&cq[slot].c);
            if (lane < 12) rec[3 + lane] = x; // ri, vi, rj, vj
            if (lane == 0) {
                cq[slot].c.i = q.i;
                cq[slot].c.j = q.j;
                cq[slot].c.tca = q.lb_rf + tm;
                cq[slot].c.dca = sqrt(sq + s1 + s2);
                cq[slot].step = q.step;
            }
        }
    }
}

// wl_cap: working-list entries available per thread.  With wl_cap < 251 an
// item whose list would outgrow it is deferred to `retry` untouched and is
// run again with the full 251-entry list by a second, smaller launch.  The
// item count is read on the device (persistent grid).
template <int OP1>
__global__ void __launch_bounds__(ROOTS_T) k_roots(dev_pj pj, const double *__restrict__ shift,
                                               const root_item *__restrict__ rq,
                                               const unsigned long long *rq_count, uint64_t rq_cap,
                                               const uint32_t *__restrict__ item_list,
                                               const unsigned long long *item_list_count, double thresh2,
                                               double *__restrict__ wl_scratch, int wl_cap,
                                               uint32_t *__restrict__ retry, unsigned long long *retry_count,
                                               conj_out *__restrict__ cq, uint64_t cq_cap,
                                               unsigned long long *cq_count, unsigned long long *counters,
                                               dev_status *st)
{
    constexpr int n = OP1 - 1;
    constexpr int ENT = OP1 + 2; // (lb, ub, q[0..n])
    const uint64_t tid = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    const uint64_t nthreads = uint64_t(gridDim.x) * blockDim.x;
    const uint64_t n_items = item_list ? *item_list_count : min(*rq_count, (unsigned long long)rq_cap);
    if constexpr (OP1 <= 32) {
        // Few items: a warp each, with its lanes' working lists as one (the
        // full list fits: 32 x ROOTS_WL_SMALL entries), so none is deferred.
        static_assert(32 * ROOTS_WL_SMALL >= WL_CAP, "a warp's share holds the full working list");
        if (n_items <= ROOTS_WARP_ITEMS && !item_list) {
            __shared__ roots_smem<OP1> S[ROOTS_T / 32];
            unsigned counts[5] = {0, 0, 0, 0, 0};
            double *wwl = wl_scratch + (tid & ~uint64_t(31)) * uint64_t(wl_cap) * ENT;
            for (uint64_t w = tid / 32; w < n_items; w += nthreads / 32)
                roots_by_warp<OP1>(pj, shift, rq[w], thresh2, wwl, S[threadIdx.x >> 5], cq, cq_cap, cq_count, counts,
                                   st);
            if ((threadIdx.x & 31) == 0)
                for (int k = 0; k < 5; ++k)
                    if (counts[k]) atomicAdd(counters + 2 + k, (unsigned long long)counts[k]);
            return;
        }
    }
    double *wl = wl_scratch + tid * uint64_t(wl_cap) * ENT;
    unsigned long long n_roots = 0, n_fex = 0, n_noroot = 0, n_minima = 0, n_disc = 0;
    for (uint64_t it = tid; it < n_items; it += nthreads) {
        const uint32_t item = item_list ? item_list[it] : uint32_t(it);
        const root_item &q = rq[item];
        const double rf_int = q.rf_int;
        double d2p[OP1];
#pragma unroll
        for (int k = 0; k < n; ++k) d2p[k] = (k + 1u) * q.ptd2[k + 1];
        d2p[n] = 0;
        double roots[MAX_ROOTS];
        int nroots = 0;
        bool failed = false, deferred = false;
        auto add_root = [&](double root) {
            if (!isfinite(root)) {
                set_error(st, ERR_ROOT_NONFINITE, q.i, q.j, root, 0);
                failed = true;
                return;
            }
            const double der = poly_eval_1_t<OP1>(d2p, root);
            if (!isfinite(der)) {
                set_error(st, ERR_ROOT_DER, q.i, q.j, root, der);
                failed = true;
                return;
            }
            if (sgn(der) == 1) {
                if (nroots < MAX_ROOTS) roots[nroots++] = root;
                else {
                    set_error(st, ERR_ISOLATION, q.i, q.j, MAX_ROOTS, 0);
                    failed = true;
                }
            }
        };
        const bool fex = fex_excludes_t<OP1>(d2p, rf_int);
        if (!fex) {
            // VCA isolation with a LIFO working list of (lb, ub, q[0..n]).
            {
                double fct = 1;
                wl[0] = 0;
                wl[1] = 1;
#pragma unroll
                for (int k = 0; k < OP1; ++k) {
                    wl[2 + k] = fct * d2p[k];
                    fct *= rf_int;
                }
            }
            int wsz = 1;
            double isol_lb[OP1 + 1], isol_ub[OP1 + 1];
            int nisol = 0;
            do {
                --wsz;
                const double *ent = wl + uint64_t(wsz) * ENT;
                const double lb = ent[0], ub = ent[1];
                double cur[OP1], r1[OP1], r2[OP1];
#pragma unroll
                for (int k = 0; k < OP1; ++k) cur[k] = ent[2 + k];
                bool tail_finite = true;
#pragma unroll
                for (int k = 1; k < OP1; ++k) tail_finite = tail_finite && isfinite(cur[k]);
                if (cur[0] == 0 && tail_finite) add_root(lb * rf_int);
#pragma unroll
                for (int k = 0; k < OP1; ++k) r1[k] = cur[n - k];
                shift1<OP1>(r1, r2);
                const int nsc = sign_changes_t<OP1>(r2);
                if (nsc == 1) {
                    if (nisol < OP1 + 1) {
                        isol_lb[nisol] = lb;
                        isol_ub[nisol] = ub;
                    }
                    ++nisol;
                } else if (nsc > 1) {
                    if (wsz + 2 > wl_cap) {
                        if (wl_cap < WL_CAP) {
                            const unsigned long long r = atomicAdd(retry_count, 1ull);
                            retry[r] = item;
                            deferred = true;
                        } else {
                            set_error(st, ERR_ISOLATION, q.i, q.j, wsz + 2, nisol);
                            failed = true;
                        }
                        break;
                    }
                    double L[OP1], R[OP1];
                    double fct = 1;
#pragma unroll
                    for (int k = 0; k < OP1; ++k) {
                        L[n - k] = fct * cur[n - k];
                        fct *= 2;
                    }
                    shift1<OP1>(L, R);
                    const double mid = lb / 2 + ub / 2;
                    double *El = wl + uint64_t(wsz) * ENT;
                    double *Er = El + ENT;
                    El[0] = lb;
                    El[1] = mid;
                    Er[0] = mid;
                    Er[1] = ub;
#pragma unroll
                    for (int k = 0; k < OP1; ++k) {
                        El[2 + k] = L[k];
                        Er[2 + k] = R[k];
                    }
                    wsz += 2;
                }
                if (wsz > 250 || nisol > n) {
                    set_error(st, ERR_ISOLATION, q.i, q.j, wsz, nisol);
                    failed = true;
                    break;
                }
            } while (wsz > 0 && !failed);
            if (deferred) continue;
            if (!failed && nisol > 0) {
                double sp[OP1];
                double fct = 1;
#pragma unroll
                for (int k = 0; k < OP1; ++k) {
                    sp[k] = fct * d2p[k];
                    fct *= rf_int;
                }
                for (int r = 0; r < nisol && !failed; ++r) {
                    double lb = isol_lb[r], ub = isol_ub[r];
                    if (isfinite(lb) && isfinite(ub) && ub > lb) ub = nextafter(ub, lb);
                    double root = 0;
                    toms_t<OP1> ev{sp, 0};
                    const int flag = toms748_t(ev, lb, ub, &root);
                    if (flag == -1) {
                        set_error(st, ERR_TOMS_ITER, q.i, q.j, 0, 0);
                        failed = true;
                    } else if (flag != 0) {
                        set_error(st, ERR_TOMS_ERRNO, q.i, q.j, flag, 0);
                        failed = true;
                    } else {
                        add_root(root * rf_int);
                    }
                }
            }
        }
        if (failed) continue;
        ++n_roots;
        n_fex += fex;
        n_noroot += (nroots == 0);
        n_minima += nroots;

        double ptd2[OP1];
#pragma unroll
        for (int k = 0; k < OP1; ++k) ptd2[k] = q.ptd2[k];
        auto emit = [&](double tm) {
            conj_out o;
            o.c.i = q.i;
            o.c.j = q.j;
            states_at_t<OP1>(pj, q.seg_i, q.di, tm, o.c.ri, o.c.vi);
            states_at_t<OP1>(pj, q.seg_j, q.dj, tm, o.c.rj, o.c.vj);
            const double dx = o.c.ri[0] - o.c.rj[0], dy = o.c.ri[1] - o.c.rj[1], dz = o.c.ri[2] - o.c.rj[2];
            o.c.dca = sqrt((dx * dx) + (dy * dy) + (dz * dz));
            o.c.tca = q.lb_rf + tm;
            o.step = q.step;
            const unsigned long long slot = atomicAdd(cq_count, 1ull);
            if (slot < cq_cap) cq[slot] = o;
        };
        for (int r = 0; r < nroots; ++r) {
            const double tm = roots[r];
            const double d2 = horner<OP1>(ptd2, tm);
            if (!isfinite(d2)) {
                set_error(st, ERR_CONJ_D2, q.i, q.j, d2, 0);
                continue;
            }
            if (d2 < thresh2) emit(tm);
            else ++n_disc;
        }
        if (q.flags & 1u) {
            const double tm = nextafter(rf_int, -1.);
            const double dv = horner<OP1>(d2p, tm);
            if (!isfinite(dv)) set_error(st, ERR_UB_DER, q.i, q.j, dv, 0);
            else if (dv < 0) {
                const double d2 = horner<OP1>(ptd2, tm);
                if (!isfinite(d2)) set_error(st, ERR_UB_D2, q.i, q.j, d2, 0);
                else if (d2 < thresh2) emit(tm);
            }
        }
        if (q.flags & 2u) {
            const double dv = horner<OP1>(d2p, 0.);
            if (!isfinite(dv)) set_error(st, ERR_LB_DER, q.i, q.j, dv, 0);
            else if (dv > 0) {
                const double d2 = horner<OP1>(ptd2, 0.);
                if (!isfinite(d2)) set_error(st, ERR_LB_D2, q.i, q.j, d2, 0);
                else if (d2 < thresh2) emit(0.);
            }
        }
    }
    warp_add(counters + 2, n_roots);
    warp_add(counters + 3, n_fex);
    warp_add(counters + 4, n_noroot);
    warp_add(counters + 5, n_minima);
    warp_add(counters + 6, n_disc);
}

// ------------------------------------------------------------- conj order

__device__ __forceinline__ bool conj_less(const conj_rec &a, const conj_rec &b)
{
    if (a.tca != b.tca) return a.tca < b.tca;
    if (a.i != b.i) return a.i < b.i;
    if (a.j != b.j) return a.j < b.j;
    if (a.dca != b.dca) return a.dca < b.dca;
    const double *pa[4] = {a.ri, a.vi, a.rj, a.vj}, *pb[4] = {b.ri, b.vi, b.rj, b.vj};
    for (int v = 0; v < 4; ++v)
        for (int k = 0; k < 3; ++k)
            if (pa[v][k] != pb[v][k]) return pa[v][k] < pb[v][k];
    return false;
}

// The batch's conjunctions ordered by (step, tca, record)
// (detect_conjunctions_narrow_phase.cpp:751-757: by tca within a step, ties by
// the record's three-way comparison).
//
// Up to CONJ_SMALL of them: one CTA sorts them all (k_conj_small).  More: they
// are grouped by step as (tca key, queue index) pairs, every step's group is
// cut into chunks of CONJ_CHUNK that one CTA each sorts in shared memory, and
// every conjunction's place is its place in its chunk plus, by binary search,
// the numbers of smaller ones in the step's other chunks; the records move
// once, to their places.  Counting and grouping take one global atomic per
// CTA and step.  With one CTA a step, a counter hit by every record and the
// runs of equal TCAs sorted by one thread each, the 507,000 conjunctions of
// 60,000 objects x 48 steps at 20 km took 2.8 ms; 0.24 ms now.  A handful of
// them takes one launch instead of five (22 -> 10 us).
constexpr uint32_t CONJ_SMALL = 512;
constexpr uint32_t CONJ_CHUNK = 2048;
constexpr uint32_t CONJ_HIST = 8192; // steps counted in shared memory

// Order-preserving integer image of a double (the TCAs are finite).
__device__ __forceinline__ uint64_t tca_key(double x)
{
    const uint64_t b = uint64_t(__double_as_longlong(x));
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// The pair of a record as the second key: (i, j) follow tca in its order.
__device__ __forceinline__ uint64_t pair_key(const conj_rec &r) { return (uint64_t(r.i) << 32) | r.j; }

constexpr int CONJ_T = 512;

// Sorts n entries (n at most the arrays' power-of-two size) of shared memory
// by (step, tca key, pair), and each run of equal entries by the whole record.
// Many conjunctions share a TCA exactly (every close pair at the start of the
// data has one there), so the pair is a key and not left to the runs.  step
// may be null (one step).  Whole CTA of CONJ_T threads.
__device__ __forceinline__ void conj_sort_smem(uint64_t *key, uint64_t *pair, uint32_t *idx, uint32_t *step,
                                               uint32_t n, const conj_out *__restrict__ cq)
{
    uint32_t P = 1;
    while (P < n) P <<= 1;
    for (uint32_t k = n + threadIdx.x; k < P; k += CONJ_T) {
        key[k] = pair[k] = ~0ull;
        idx[k] = 0xffffffffu;
        if (step) step[k] = 0xffffffffu;
    }
    __syncthreads();
    for (uint32_t size = 2; size <= P; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t t = threadIdx.x; t < P / 2; t += CONJ_T) {
                const uint32_t i = 2 * t - (t & (stride - 1)), j = i + stride;
                const bool asc = (i & size) == 0;
                const uint64_t ki = key[i], kj = key[j];
                const uint32_t si = step ? step[i] : 0, sj = step ? step[j] : 0;
                const uint64_t pi = pair[i], pj = pair[j];
                const uint32_t ii = idx[i], ij = idx[j];
                const bool gt = si != sj ? si > sj : ki != kj ? ki > kj : pi != pj ? pi > pj : ii > ij;
                if (gt == asc) {
                    key[i] = kj;
                    key[j] = ki;
                    pair[i] = pj;
                    pair[j] = pi;
                    idx[i] = ij;
                    idx[j] = ii;
                    if (step) {
                        step[i] = sj;
                        step[j] = si;
                    }
                }
            }
            __syncthreads();
        }
    // One pair twice at one TCA: insertion sort by the whole record.
    auto same = [&](uint32_t a, uint32_t b) {
        return key[a] == key[b] && pair[a] == pair[b] && (!step || step[a] == step[b]);
    };
    for (uint32_t k = threadIdx.x; k < n; k += CONJ_T) {
        if ((k == 0 || !same(k - 1, k)) && k + 1 < n && same(k + 1, k)) {
            uint32_t e = k + 1;
            while (e < n && same(e, k)) ++e;
            for (uint32_t a = k + 1; a < e; ++a)
                for (uint32_t c = a; c > k && conj_less(cq[idx[c]].c, cq[idx[c - 1]].c); --c) {
                    const uint32_t t2 = idx[c];
                    idx[c] = idx[c - 1];
                    idx[c - 1] = t2;
                }
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(CONJ_T) k_conj_small(const conj_out *__restrict__ cq, uint32_t n,
                                                       conj_rec *__restrict__ out)
{
    __shared__ uint64_t key[CONJ_SMALL], pair[CONJ_SMALL];
    __shared__ uint32_t idx[CONJ_SMALL], step[CONJ_SMALL];
    for (uint32_t k = threadIdx.x; k < n; k += CONJ_T) {
        key[k] = tca_key(cq[k].c.tca);
        pair[k] = pair_key(cq[k].c);
        idx[k] = k;
        step[k] = cq[k].step;
    }
    conj_sort_smem(key, pair, idx, step, n, cq);
    for (uint32_t k = threadIdx.x; k < n; k += CONJ_T) out[k] = cq[idx[k]].c;
}

// Conjunctions per step: one global atomic per CTA and step it meets.
__global__ void __launch_bounds__(1024) k_conj_count(const conj_out *__restrict__ cq, uint64_t n, uint32_t nb,
                                                     uint32_t *__restrict__ cnt)
{
    __shared__ uint32_t hist[CONJ_HIST];
    for (uint32_t s = threadIdx.x; s < min(nb, CONJ_HIST); s += blockDim.x) hist[s] = 0;
    __syncthreads();
    for (uint64_t g = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; g < n; g += uint64_t(gridDim.x) * blockDim.x) {
        const uint32_t s = cq[g].step;
        if (s < CONJ_HIST) atomicAdd(&hist[s], 1u);
        else atomicAdd(cnt + s, 1u);
    }
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < min(nb, CONJ_HIST); s += blockDim.x)
        if (hist[s]) atomicAdd(cnt + s, hist[s]);
}

// One block: exclusive scans of the per-step counts and chunk numbers (also
// resets cursors).
__global__ void k_conj_offsets(const uint32_t *cnt, uint32_t nb, uint32_t *off, uint32_t *choff, uint32_t *cursor)
{
    __shared__ uint32_t sm[33];
    uint32_t carry = 0, ccarry = 0;
    for (uint32_t base = 0; base < nb; base += blockDim.x) {
        const uint32_t k = base + threadIdx.x;
        const uint32_t v = k < nb ? cnt[k] : 0;
        uint32_t tot, ctot;
        const uint32_t ex = block_excl_scan(v, sm, &tot);
        const uint32_t cex = block_excl_scan((v + CONJ_CHUNK - 1) / CONJ_CHUNK, sm, &ctot);
        if (k < nb) {
            off[k] = carry + ex;
            choff[k] = ccarry + cex;
            cursor[k] = 0;
        }
        carry += tot;
        ccarry += ctot;
    }
    if (threadIdx.x == 0) {
        off[nb] = carry;
        choff[nb] = ccarry;
    }
}

__global__ void __launch_bounds__(1024) k_conj_group(const conj_out *__restrict__ cq, uint64_t n, uint32_t nb,
                                                     const uint32_t *__restrict__ off, uint32_t *__restrict__ cursor,
                                                     uint64_t *__restrict__ gkey, uint32_t *__restrict__ gidx)
{
    __shared__ uint32_t hist[CONJ_HIST];
    for (uint32_t s = threadIdx.x; s < min(nb, CONJ_HIST); s += blockDim.x) hist[s] = 0;
    __syncthreads();
    const uint64_t g = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    const uint32_t s = g < n ? cq[g].step : 0;
    uint32_t r = 0;
    if (g < n) r = s < CONJ_HIST ? atomicAdd(&hist[s], 1u) : atomicAdd(cursor + s, 1u);
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < min(nb, CONJ_HIST); q += blockDim.x)
        if (hist[q]) hist[q] = atomicAdd(cursor + q, hist[q]);
    __syncthreads();
    if (g < n) {
        const uint32_t at = off[s] + r + (s < CONJ_HIST ? hist[s] : 0);
        gkey[at] = tca_key(cq[g].c.tca);
        gidx[at] = uint32_t(g);
    }
}

// The chunk of CTA c: its step, and its range in the grouped arrays.
__device__ __forceinline__ uint32_t conj_chunk(const uint32_t *off, const uint32_t *choff, uint32_t nb, uint32_t c,
                                               uint32_t &b, uint32_t &e)
{
    uint32_t lo = 0, hi = nb; // last step with choff <= c
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (choff[mid] <= c) lo = mid;
        else hi = mid;
    }
    b = off[lo] + (c - choff[lo]) * CONJ_CHUNK;
    e = min(off[lo + 1], b + CONJ_CHUNK);
    return lo;
}

__global__ void __launch_bounds__(CONJ_T) k_conj_chunks(const conj_out *__restrict__ cq, uint32_t nb,
                                                        const uint32_t *__restrict__ off,
                                                        const uint32_t *__restrict__ choff,
                                                        uint64_t *__restrict__ gkey, uint32_t *__restrict__ gidx)
{
    __shared__ uint64_t key[CONJ_CHUNK], pair[CONJ_CHUNK];
    __shared__ uint32_t idx[CONJ_CHUNK];
    if (blockIdx.x >= choff[nb]) return;
    uint32_t b, e;
    conj_chunk(off, choff, nb, blockIdx.x, b, e);
    for (uint32_t k = threadIdx.x; k < e - b; k += CONJ_T) {
        key[k] = gkey[b + k];
        idx[k] = gidx[b + k];
        pair[k] = pair_key(cq[idx[k]].c);
    }
    conj_sort_smem(key, pair, idx, nullptr, e - b, cq);
    for (uint32_t k = threadIdx.x; k < e - b; k += CONJ_T) {
        gkey[b + k] = key[k];
        gidx[b + k] = idx[k];
    }
}

__global__ void __launch_bounds__(CONJ_T) k_conj_merge(const conj_out *__restrict__ cq, uint32_t nb,
                                                       const uint32_t *__restrict__ off,
                                                       const uint32_t *__restrict__ choff,
                                                       const uint64_t *__restrict__ gkey,
                                                       const uint32_t *__restrict__ gidx, conj_rec *__restrict__ out)
{
    if (blockIdx.x >= choff[nb]) return;
    uint32_t b, e;
    const uint32_t s = conj_chunk(off, choff, nb, blockIdx.x, b, e);
    for (uint32_t k = b + threadIdx.x; k < e; k += CONJ_T) {
        const uint64_t key = gkey[k];
        const conj_rec me = cq[gidx[k]].c;
        const uint64_t pair = pair_key(me);
        uint32_t place = k - b;
        for (uint32_t c0 = off[s]; c0 < off[s + 1]; c0 += CONJ_CHUNK) {
            if (c0 == b) continue;
            const uint32_t c1 = min(off[s + 1], c0 + CONJ_CHUNK);
            uint32_t lo = c0, hi = c1; // first (key, pair) >= mine
            while (lo < hi) {
                const uint32_t mid = (lo + hi) / 2;
                const uint64_t o = gkey[mid];
                if (o < key || (o == key && pair_key(cq[gidx[mid]].c) < pair)) lo = mid + 1;
                else hi = mid;
            }
            // The same pair at the same TCA: by the record; of equal records
            // the earlier chunk's come first.
            while (lo < c1 && gkey[lo] == key) {
                const conj_rec &o = cq[gidx[lo]].c;
                if (pair_key(o) != pair || !(conj_less(o, me) || (c0 < b && !conj_less(me, o)))) break;
                ++lo;
            }
            place += lo - c0;
        }
        out[off[s] + place] = me;
    }
}

// ------------------------------------------------------------- launchers

void launch_items(const dev_pj &pj, const double2 *cdb, uint32_t s_first, uint32_t nb, const uint2 *pairs,
                  const uint64_t *step_off, const uint2 *srange, uint64_t n_pairs, np_item *items, uint64_t cap,
                  unsigned long long *item_count, unsigned long long *counters, dev_status *st, cudaStream_t stream)
{
    const unsigned bs = 128;
    const unsigned g = unsigned((n_pairs + bs - 1) / bs);
    if (g == 0) return;
    k_items<<<g, bs, 0, stream>>>(pj, cdb, s_first, nb, pairs, step_off, srange, items, cap, item_count, counters,
                                  st);
}

template <int OP1>
static void narrow_t(const dev_pj &pj, const double *shift, const double2 *cdb, uint32_t s_first, const np_item *items,
                     const unsigned long long *item_count, uint64_t item_cap, double thresh2, root_item *rq,
                     uint64_t rq_cap, unsigned long long *rq_count, unsigned long long *counters, dev_status *st,
                     unsigned grid, cudaStream_t stream)
{
    k_narrow<OP1><<<grid, NARROW_T, 0, stream>>>(pj, make_cheb_nodes(OP1), shift, cdb, s_first, items,
                                                  item_count, item_cap, thresh2, rq, rq_cap, rq_count, counters, st);
}

// shift[k * op1 + i] = C(i + k, k), device memory.
void launch_narrow(const dev_pj &pj, const double *shift, const double2 *cdb, uint32_t s_first, const np_item *items,
                   const unsigned long long *item_count, uint64_t item_cap, double thresh2, root_item *rq,
                   uint64_t rq_cap, unsigned long long *rq_count, unsigned long long *counters, dev_status *st,
                   unsigned grid, cudaStream_t stream)
{
    switch (pj.op1) {
#define X(K)                                                                                                         \
    case K:                                                                                                            \
        narrow_t<K>(pj, shift, cdb, s_first, items, item_count, item_cap, thresh2, rq, rq_cap, rq_count, counters, st, grid, \
                    stream);                                                                                           \
        break;
        MZB_FOR_EACH_OP1(X)
#undef X
    default:
        break;
    }
}

template <int OP1>
static void filter_t(const dev_pj &pj, const double2 *cdb, uint32_t s_first, const np_item *items,
                     const unsigned long long *item_count, uint64_t item_cap, double thresh2, np_item *surv,
                     uint64_t surv_cap, unsigned long long *surv_count, unsigned long long *counters,
                     cudaStream_t stream)
{
    using F = filter_shape<OP1>;
    static const filter_consts<OP1> consts = make_filter_consts<OP1>();
    k_narrow_filter<OP1><<<148 * F::CTAS, 32, 0, stream>>>(pj, consts, cdb, s_first, items, item_count, item_cap,
                                                             thresh2, surv, surv_cap, surv_count, counters);
}

void launch_narrow_filter(const dev_pj &pj, const double2 *cdb, uint32_t s_first, const np_item *items,
                          const unsigned long long *item_count, uint64_t item_cap, double thresh2, np_item *surv,
                          uint64_t surv_cap, unsigned long long *surv_count, unsigned long long *counters,
                          cudaStream_t stream)
{
    switch (pj.op1) {
#define X(K)                                                                                                         \
    case K:                                                                                                            \
        filter_t<K>(pj, cdb, s_first, items, item_count, item_cap, thresh2, surv, surv_cap, surv_count,     \
                    counters, stream);                                                                                 \
        break;
        MZB_FOR_EACH_OP1(X)
#undef X
    default:
        break;
    }
}

template <int OP1>
static void roots_t(const dev_pj &pj, const double *shift, const root_item *rq, const unsigned long long *rq_count, uint64_t rq_cap,
                    const uint32_t *item_list, const unsigned long long *item_list_count, double thresh2,
                    double *wl_scratch, int wl_cap, unsigned grid, uint32_t *retry, unsigned long long *retry_count,
                    conj_out *cq, uint64_t cq_cap, unsigned long long *cq_count, unsigned long long *counters,
                    dev_status *st, cudaStream_t stream)
{
    k_roots<OP1><<<grid, ROOTS_T, 0, stream>>>(pj, shift, rq, rq_count, rq_cap, item_list, item_list_count, thresh2, wl_scratch,
                                            wl_cap, retry, retry_count, cq, cq_cap, cq_count, counters, st);
}

// shift as for launch_narrow.
void launch_roots(const dev_pj &pj, const double *shift, const root_item *rq, const unsigned long long *rq_count, uint64_t rq_cap,
                  const uint32_t *item_list, const unsigned long long *item_list_count, double thresh2,
                  double *wl_scratch, int wl_cap, unsigned grid, uint32_t *retry, unsigned long long *retry_count,
                  conj_out *cq, uint64_t cq_cap, unsigned long long *cq_count, unsigned long long *counters,
                  dev_status *st, cudaStream_t stream)
{
    switch (pj.op1) {
#define X(K)                                                                                                         \
    case K:                                                                                                            \
        roots_t<K>(pj, shift, rq, rq_count, rq_cap, item_list, item_list_count, thresh2, wl_scratch, wl_cap, grid, retry,    \
                   retry_count, cq, cq_cap, cq_count, counters, st, stream);                                          \
        break;
        MZB_FOR_EACH_OP1(X)
#undef X
    default:
        break;
    }
}

// cnt, off, choff, cursor: nb + 1 words; gkey, gidx: n entries (used when
// there are more than CONJ_SMALL conjunctions).  Returns the launches.
int launch_conj_sort(const conj_out *cq, uint64_t n, uint32_t nb, uint32_t *cnt, uint32_t *off, uint32_t *choff,
                     uint32_t *cursor, uint64_t *gkey, uint32_t *gidx, conj_rec *out, cudaStream_t stream)
{
    if (n == 0) return 0;
    if (n <= CONJ_SMALL) {
        k_conj_small<<<1, CONJ_T, 0, stream>>>(cq, uint32_t(n), out);
        return 1;
    }
    cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * nb, stream);
    const unsigned g = unsigned((n + 1023) / 1024);
    k_conj_count<<<std::min(g, 148u * 2), 1024, 0, stream>>>(cq, n, nb, cnt);
    k_conj_offsets<<<1, 1024, 0, stream>>>(cnt, nb, off, choff, cursor);
    k_conj_group<<<g, 1024, 0, stream>>>(cq, n, nb, off, cursor, gkey, gidx);
    const unsigned chunks = unsigned(n / CONJ_CHUNK) + unsigned(std::min<uint64_t>(n, nb));
    k_conj_chunks<<<chunks, CONJ_T, 0, stream>>>(cq, nb, off, choff, gkey, gidx);
    k_conj_merge<<<chunks, CONJ_T, 0, stream>>>(cq, nb, off, choff, gkey, gidx, out);
    return 5;
}

cudaError_t init_narrow_consts() { return upload_binom_table(); }

} // namespace mzb
