// SGP4 polyjectory production on the GPU (mizuba's make_sgp4_polyjectory,
// mizuba/make_sgp4_polyjectory.cpp:478-913 and :1461-1603).
//
// For every satellite the reference walks its element sets in epoch order,
// each over the span up to the next set's epoch.  Within a span it takes
// steps of Keplerian motion from the SGP4 state at each step's start
// (sgp4pj.cuh), interpolates the SGP4 state (x, y, z, vx, vy, vz, r) at the
// order + 1 Chebyshev nodes of the step with Bjorck-Pereyra, estimates the
// position error at the midpoints between nodes against SGP4 itself, and
// bisects the step while the error is 1e-7 km or more (steps under 5 s are
// accepted as they are; more than 20 polynomials in one step is an error).
//
// Near-Earth and deep-space element sets alike (sgp4.cuh).  The steps of a span
// do not depend on its polynomials, so the work is laid out by what is
// independent: one thread per span finds its steps (k_sgp4_steps); then every
// step of every span is interpolated and checked at once, one thread per node
// and midpoint, packed without idle lanes (k_sgp4_interp); the few steps that
// need bisection or end in an error go through the reference's procedure one
// warp per step (k_sgp4_bisect), which also yields its exact status.  A pass
// over each span's steps numbers its polynomials up to the first failure, and
// a gather lays them out as the polyjectory's trajectory and time arrays.
#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <type_traits>
#include <vector>

#include "block.cuh"
#include "common.cuh"
#include "kernels.cuh"
#include "sgp4pj.cuh"

namespace mzb
{
namespace sgp4pj
{

constexpr int WARPS = 4;
constexpr int STACK = 40;
constexpr int MAX_POLYS = 20;                  // make_sgp4_polyjectory.cpp:495-502
constexpr double MIN_STEP = 5.0 / 86400.0;     // days, make_sgp4_polyjectory.cpp:487
constexpr double ERR_THRESH = 1e-7;            // km, make_sgp4_polyjectory.cpp:490
constexpr uint32_t NOT_KEPT = 0xffffffffu;

// One step of a span: [b, e) in days from the polyjectory epoch, [bs, es) the
// same instants from the element set's epoch; the k-th of its job.
struct step_rec {
    double b, e, bs, es;
    uint32_t job, k;
};

// One accepted polynomial: number `seq` of step `step`, over [t0, t1).
struct seg_rec {
    uint32_t step, seq;
    double t0, t1;
};

struct nodes_t {
    double c[OP1]; // Chebyshev nodes of [-1, 1], ascending
};

struct warp_smem {
    double val[OP1][7];
    double cf[OP1][7];
    double stk[STACK][4];
    double acc_t0[MAX_POLYS + 2], acc_t1[MAX_POLYS + 2];
    unsigned long long acc_slot[MAX_POLYS + 2];
};

// SGP4 state at t [min]: x, y, z, vx, vy, vz and the radius.
__device__ __forceinline__ int state7(const sgp4::sat &s, double t, double o[7])
{
    double r[3], v[3];
    const int e = sgp4::propagate(s, t, r, v);
    o[0] = r[0];
    o[1] = r[1];
    o[2] = r[2];
    o[3] = v[0];
    o[4] = v[1];
    o[5] = v[2];
    o[6] = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    return e;
}

// The lowest lane's non-zero code (the reference checks the nodes in order).
__device__ __forceinline__ int first_code(int code)
{
    const unsigned m = __ballot_sync(0xffffffffu, code != 0);
    return m ? __shfl_sync(0xffffffffu, code, __ffs(m) - 1) : 0;
}

// Interpolation of one step [b, e) (days from the polyjectory epoch; bs, es
// the same instants in days from the element set's epoch) with bisection
// (make_sgp4_polyjectory.cpp:478-700).  Warp-collective.  Returns 0 and the
// accepted polynomials (pool slots and time spans in S.acc_*), or a status.
__device__ int interpolate_step(const sgp4::sat &sat, const nodes_t &nd, double b0, double e0, double bs0,
                                double es0, warp_smem &S, int &n_acc, double *__restrict__ pool, uint64_t cap,
                                unsigned long long *pool_count, int *overflow)
{
    const unsigned lane = threadIdx.x & 31;
    int sp = 0;
    if (lane == 0) {
        S.stk[0][0] = b0;
        S.stk[0][1] = e0;
        S.stk[0][2] = bs0;
        S.stk[0][3] = es0;
    }
    sp = 1;
    n_acc = 0;
    __syncwarp();
    while (sp > 0) {
        if (n_acc > MAX_POLYS) return ST_INTERPOLATION;
        --sp;
        const double b = S.stk[sp][0], e = S.stk[sp][1], bs = S.stk[sp][2], es = S.stk[sp][3];
        __syncwarp();
        const double dur = e - b, dur_s = es - bs;
        if (!isfinite(dur) || !isfinite(dur_s)) return ST_NONFINITE;
        // SGP4 at the nodes (minutes from the element set's epoch).
        double st[7];
        int code = 0;
        if (lane < OP1) {
            const double tp = (nd.c[lane] + 1) / 2 * (dur_s * 1440.) + bs * 1440.;
            code = state7(sat, tp, st);
            if (code == 0)
                for (int v = 0; v < 7; ++v) S.val[lane][v] = st[v];
        }
        code = first_code(code);
        if (code) return code;
        __syncwarp();
        // Bjorck-Pereyra on the nodes of [0, dur], one variable per lane
        // (vm_interp, mizuba/detail/poly_utils.cpp:467-535).
        if (lane < 7) {
            double f[OP1], al[OP1];
#pragma unroll
            for (int j = 0; j < OP1; ++j) {
                f[j] = S.val[j][lane];
                al[j] = (nd.c[j] + 1) / 2 * dur;
            }
#pragma unroll
            for (int k = 0; k < ORDER; ++k)
#pragma unroll
                for (int j = ORDER; j > k; --j) f[j] = (f[j] - f[j - 1]) / (al[j] - al[j - k - 1]);
#pragma unroll
            for (int k = ORDER - 1; k >= 0; --k)
#pragma unroll
                for (int j = k; j < ORDER; ++j) f[j] = f[j] - al[k] * f[j + 1];
#pragma unroll
            for (int j = 0; j < OP1; ++j) S.cf[j][lane] = f[j];
        }
        __syncwarp();
        bool accept = dur < MIN_STEP;
        if (!accept) {
            // Position error halfway between the nodes
            // (eval_interp_error2, make_sgp4_polyjectory.cpp:325-410).
            double err2 = 0;
            code = 0;
            int nonfinite = 0;
            if (lane < OP1) {
                const double a_cur = (nd.c[lane] + 1) / 2 * dur;
                const double a_prev = lane == 0 ? 0. : (nd.c[lane - 1] + 1) / 2 * dur;
                const double ev = a_prev / 2 + a_cur / 2;
                double xyz[3];
                for (int v = 0; v < 3; ++v) {
                    double r = S.cf[ORDER][v];
                    for (int o = 1; o <= ORDER; ++o) r = S.cf[ORDER - o][v] + r * ev;
                    xyz[v] = r;
                }
                const double s_cur = (nd.c[lane] + 1) / 2 * (dur_s * 1440.) + bs * 1440.;
                const double s_prev = lane == 0 ? bs * 1440. : (nd.c[lane - 1] + 1) / 2 * (dur_s * 1440.) + bs * 1440.;
                code = state7(sat, s_prev / 2 + s_cur / 2, st);
                const double dx = xyz[0] - st[0], dy = xyz[1] - st[1], dz = xyz[2] - st[2];
                err2 = dx * dx + dy * dy + dz * dz;
                nonfinite = !isfinite(err2);
            }
            code = first_code(code);
            if (code) return code;
            if (__any_sync(0xffffffffu, nonfinite)) return ST_NONFINITE;
            for (int o = 16; o > 0; o >>= 1) err2 = fmax(err2, __shfl_xor_sync(0xffffffffu, err2, o));
            accept = err2 < ERR_THRESH * ERR_THRESH;
        }
        if (accept) {
            unsigned long long slot = 0;
            if (lane == 0) slot = atomicAdd(pool_count, 1ull);
            slot = __shfl_sync(0xffffffffu, slot, 0);
            if (slot < cap) {
                double *dst = pool + slot * uint64_t(OP1 * 7);
                for (int k = lane; k < OP1 * 7; k += 32) dst[k] = S.cf[k / 7][k % 7];
            } else if (lane == 0) {
                *overflow = 1;
            }
            if (lane == 0) {
                S.acc_slot[n_acc] = slot;
                S.acc_t0[n_acc] = b;
                S.acc_t1[n_acc] = e;
            }
            ++n_acc;
        } else {
            if (sp + 2 > STACK) return ST_INTERPOLATION;
            const double mid = b + dur / 2, mid_s = bs + dur_s / 2;
            if (lane == 0) {
                S.stk[sp][0] = b;
                S.stk[sp][1] = mid;
                S.stk[sp][2] = bs;
                S.stk[sp][3] = mid_s;
                S.stk[sp + 1][0] = mid;
                S.stk[sp + 1][1] = e;
                S.stk[sp + 1][2] = mid_s;
                S.stk[sp + 1][3] = es;
            }
            sp += 2;
        }
        __syncwarp();
    }
    return 0;
}

// Set-up of every element set, once (its coefficients are read by all of its
// propagations); init[j] is the set-up's error code.
__global__ void __launch_bounds__(64) k_sgp4_setup(const job *__restrict__ jobs, uint32_t n, sgp4::sat *sats,
                                                   int *__restrict__ init)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const job J = jobs[j];
    init[j] = sgp4::setup(J.n0, J.e0, J.i0, J.node0, J.omega0, J.m0, J.bstar, J.epoch1950, sats[j]);
}

__global__ void __launch_bounds__(64) k_sgp4_setup_gpes(const gpe_host *__restrict__ gpes, uint64_t n,
                                                        sgp4::sat *sats, int *__restrict__ init)
{
    const uint64_t j = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    if (j >= n) return;
    const gpe_host g = gpes[j];
    const double epoch1950 = dfl_sub(dfl_norm(g.epoch_jd1, g.epoch_jd2), dfl{2433281.5, 0.0}).hi;
    init[j] = sgp4::setup(g.n0, g.e0, g.i0, g.node0, g.omega0, g.m0, g.bstar, epoch1950, sats[j]);
}

// The steps of every span, one thread per span in the sequence `order` (the
// jobs by decreasing expected work, so that the lanes of a warp take about as
// many steps).  A serial chain of one propagation and one Taylor step size
// per step: bound by its latency, and short against the interpolation
// (1.2 of 4.1 ms of kernels for 6,000 element sets over 6 hours; 2.7 ms with
// the step size's Taylor coefficients in local memory instead of registers).  n_steps[j] steps are appended to `out` in any order, end[j]
// is the status that ended them (0: the span's end).
__global__ void __launch_bounds__(32) k_sgp4_steps(const job *__restrict__ jobs, uint32_t n_jobs,
                                                   const uint32_t *__restrict__ order, const sgp4::sat *sats,
                                                   const int *__restrict__ init, dfl pj_epoch, double reentry,
                                                   double exit_r, uint64_t max_steps, step_rec *__restrict__ out,
                                                   uint64_t cap, unsigned long long *count,
                                                   uint32_t *__restrict__ n_steps, int *__restrict__ end)
{
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_jobs) return;
    const uint32_t jb = order[q];
    const job J = jobs[jb];
    const sgp4::sat &sat = sats[jb];
    int st = init[jb];
    uint32_t k = 0;
    dfl cur = J.begin_tai;
    // Every step but the last is at least 1 s long, so max_steps bounds the
    // loop; reaching it reports the small-step status.
    for (uint64_t it = 0; st == 0; ++it) {
        if (it >= max_steps) {
            st = ST_SMALL_STEP;
            break;
        }
        const double step_begin = dfl_sub(cur, pj_epoch).hi;
        const dfl sb_s = dfl_sub(cur, J.epoch_tai);
        double r[3], v[3];
        const int e = sgp4::propagate(sat, sb_s.hi * 1440., r, v);
        if (e) {
            st = e;
            break;
        }
        const double r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
        if (r2 < reentry * reentry) {
            st = ST_REENTRY;
            break;
        }
        if (r2 >= exit_r * exit_r) {
            st = ST_EXIT;
            break;
        }
        const double hmax = dfl_sub(J.end_tai, cur).hi * 86400.;
        double h = kepler_step(r, v);
        bool last = false;
        if (!isfinite(h)) {
            st = ST_NONFINITE;
            break;
        }
        if (h >= hmax) {
            h = hmax;
            last = true;
        } else if (h < 1.) {
            st = ST_SMALL_STEP;
            break;
        }
        const unsigned long long slot = atomicAdd(count, 1ull);
        if (slot < cap)
            out[slot] = step_rec{step_begin, step_begin + h / 86400., sb_s.hi, dfl_add(sb_s, h / 86400.).hi, jb, k};
        ++k;
        if (last) break;
        cur = dfl_add(cur, h / 86400.);
    }
    n_steps[jb] = k;
    end[jb] = st;
}

// First step of every job when the steps stand job by job in the sequence
// `order` (one block).
__global__ void __launch_bounds__(1024) k_sgp4_bases(const uint32_t *__restrict__ order, uint32_t n_jobs,
                                                     const uint32_t *__restrict__ n_steps, uint32_t *__restrict__ base)
{
    __shared__ uint32_t sm[33];
    uint32_t carry = 0;
    for (uint32_t q0 = 0; q0 < n_jobs; q0 += blockDim.x) {
        const uint32_t q = q0 + threadIdx.x;
        const uint32_t jb = q < n_jobs ? order[q] : 0;
        uint32_t tot;
        const uint32_t ex = block_excl_scan(q < n_jobs ? n_steps[jb] : 0, sm, &tot);
        if (q < n_jobs) base[jb] = carry + ex;
        carry += tot;
    }
}

__global__ void __launch_bounds__(256) k_sgp4_place(const step_rec *__restrict__ in, uint64_t n,
                                                    const uint32_t *__restrict__ base, step_rec *__restrict__ out)
{
    const uint64_t g = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    if (g >= n) return;
    const step_rec r = in[g];
    out[base[r.job] + r.k] = r;
}

// Interpolation and error check of INTERP_STEPS steps by one CTA
// (make_sgp4_polyjectory.cpp:478-700 without the bisection): thread (s, m)
// propagates step s to node m, thread (s, v) interpolates variable v of step
// s, thread (s, m) compares the interpolant with SGP4 halfway to node m.
// An accepted step's polynomial goes to the pool slot of its own number; the
// others are listed for k_sgp4_bisect.
//
// Bound by the latency of the propagator (FP64 and the transcendental
// functions around it), so residency counts more than registers: 3.3 ms at two
// CTAs an SM (154 registers), 1.8 at four, 1.7 at five (72), for 6,000
// element sets over 6 hours.  With 8 steps a CTA 152 of 160 lanes propagate; a
// warp per step had 19 of 32, computed the step size in all of them and
// interpolated with 7 (23.7 ms, step sizes included; the day of every third of
// the 26,389 sets of a catalogue 155 -> 35 ms).
constexpr int INTERP_STEPS = 8;
constexpr int INTERP_T = 160;
static_assert(INTERP_STEPS * OP1 <= INTERP_T, "one thread per node");

__global__ void __launch_bounds__(INTERP_T, 5) k_sgp4_interp(const step_rec *__restrict__ steps, uint64_t n_steps,
                                                          const sgp4::sat *sats, nodes_t nd,
                                                          double *__restrict__ pool, seg_rec *__restrict__ recs,
                                                          uint32_t *__restrict__ n_polys,
                                                          uint32_t *__restrict__ redo, unsigned long long *n_redo)
{
    __shared__ double f[INTERP_STEPS][OP1][7]; // node values, then coefficients
    __shared__ double al[INTERP_STEPS][OP1], cn[OP1];
    __shared__ step_rec sr[INTERP_STEPS];
    __shared__ int bad[INTERP_STEPS];
    const unsigned tid = threadIdx.x;
    const uint64_t first = blockIdx.x * uint64_t(INTERP_STEPS);
    const unsigned n = unsigned(n_steps - first < INTERP_STEPS ? n_steps - first : INTERP_STEPS);
    if (tid < OP1) cn[tid] = nd.c[tid];
    if (tid < n) {
        const step_rec r = steps[first + tid];
        sr[tid] = r;
        bad[tid] = !isfinite(r.e - r.b) || !isfinite(r.es - r.bs);
    }
    __syncthreads();
    const unsigned s = tid / OP1, m = tid % OP1;
    const bool mine = s < n && !bad[s < n ? s : 0];
    double b = 0, bs = 0, dur = 0, dur_s = 0;
    const sgp4::sat *sat = sats;
    if (mine) {
        b = sr[s].b;
        bs = sr[s].bs;
        dur = sr[s].e - b;
        dur_s = sr[s].es - bs;
        sat = sats + sr[s].job;
        al[s][m] = (cn[m] + 1) / 2 * dur;
        double st[7];
        if (state7(*sat, (cn[m] + 1) / 2 * (dur_s * 1440.) + bs * 1440., st)) bad[s] = 1;
        for (int v = 0; v < 7; ++v) f[s][m][v] = st[v];
    }
    __syncthreads();
    // Bjorck-Pereyra on the nodes of [0, dur], one variable per thread
    // (vm_interp, mizuba/detail/poly_utils.cpp:467-535).
    if (tid < n * 7) {
        const unsigned u = tid / 7, v = tid % 7;
        if (!bad[u]) {
#pragma unroll 1
            for (int k = 0; k < ORDER; ++k) {
                double hi = f[u][ORDER][v];
#pragma unroll 6
                for (int j = ORDER; j > k; --j) {
                    const double lo = f[u][j - 1][v];
                    f[u][j][v] = (hi - lo) / (al[u][j] - al[u][j - k - 1]);
                    hi = lo;
                }
            }
#pragma unroll 1
            for (int k = ORDER - 1; k >= 0; --k) {
                const double ck = al[u][k];
                double lo = f[u][k][v];
#pragma unroll 6
                for (int j = k; j < ORDER; ++j) {
                    const double hi = f[u][j + 1][v];
                    f[u][j][v] = lo - ck * hi;
                    lo = hi;
                }
            }
        }
    }
    __syncthreads();
    // Position error halfway between the nodes (eval_interp_error2,
    // make_sgp4_polyjectory.cpp:325-410).
    if (mine && !bad[s] && !(dur < MIN_STEP)) {
        const double a_cur = (cn[m] + 1) / 2 * dur;
        const double a_prev = m == 0 ? 0. : (cn[m - 1] + 1) / 2 * dur;
        const double ev = a_prev / 2 + a_cur / 2;
        double xyz[3];
        for (int v = 0; v < 3; ++v) {
            double r = f[s][ORDER][v];
            for (int o = 1; o <= ORDER; ++o) r = f[s][ORDER - o][v] + r * ev;
            xyz[v] = r;
        }
        const double s_cur = (cn[m] + 1) / 2 * (dur_s * 1440.) + bs * 1440.;
        const double s_prev = m == 0 ? bs * 1440. : (cn[m - 1] + 1) / 2 * (dur_s * 1440.) + bs * 1440.;
        double st[7];
        const int code = state7(*sat, s_prev / 2 + s_cur / 2, st);
        const double dx = xyz[0] - st[0], dy = xyz[1] - st[1], dz = xyz[2] - st[2];
        const double err2 = dx * dx + dy * dy + dz * dz;
        if (code || !isfinite(err2) || !(err2 < ERR_THRESH * ERR_THRESH)) bad[s] = 1;
    }
    __syncthreads();
    for (unsigned e = tid; e < n * (OP1 * 7); e += INTERP_T)
        if (!bad[e / (OP1 * 7)]) pool[first * (OP1 * 7) + e] = (&f[0][0][0])[e];
    if (tid < n) {
        const uint32_t idx = uint32_t(first + tid);
        recs[idx] = seg_rec{bad[tid] ? NOT_KEPT : idx, 0, sr[tid].b, sr[tid].e};
        n_polys[idx] = bad[tid] ? 0 : 1;
        if (bad[tid]) redo[atomicAdd(n_redo, 1ull)] = idx;
    }
}

// The steps that k_sgp4_interp left, one warp per step: interpolation with
// bisection as the reference does it, polynomials appended to the pool from
// slot n_steps on.
__global__ void __launch_bounds__(32 * WARPS, 4) k_sgp4_bisect(const step_rec *__restrict__ steps,
                                                            const sgp4::sat *sats, nodes_t nd,
                                                            const uint32_t *__restrict__ redo,
                                                            const unsigned long long *n_redo,
                                                            double *__restrict__ pool, seg_rec *__restrict__ recs,
                                                            uint64_t cap, unsigned long long *pool_count,
                                                            int *overflow, uint32_t *__restrict__ n_polys,
                                                            int *__restrict__ status)
{
    __shared__ warp_smem smem[WARPS];
    const unsigned w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    warp_smem &S = smem[w];
    const uint64_t n = *n_redo;
    for (uint64_t k = blockIdx.x * uint64_t(WARPS) + w; k < n; k += uint64_t(gridDim.x) * WARPS) {
        const uint32_t idx = redo[k];
        const step_rec r = steps[idx];
        int n_acc = 0;
        const int st = interpolate_step(sats[r.job], nd, r.b, r.e, r.bs, r.es, S, n_acc, pool, cap, pool_count,
                                        overflow);
        // The step's polynomials in time order.
        if (lane == 0) {
            for (int a = 1; a < n_acc; ++a)
                for (int c = a; c > 0 && S.acc_t0[c] < S.acc_t0[c - 1]; --c) {
                    const double t0 = S.acc_t0[c], t1 = S.acc_t1[c];
                    const unsigned long long sl = S.acc_slot[c];
                    S.acc_t0[c] = S.acc_t0[c - 1];
                    S.acc_t1[c] = S.acc_t1[c - 1];
                    S.acc_slot[c] = S.acc_slot[c - 1];
                    S.acc_t0[c - 1] = t0;
                    S.acc_t1[c - 1] = t1;
                    S.acc_slot[c - 1] = sl;
                }
            for (int a = 0; a < n_acc; ++a)
                if (S.acc_slot[a] < cap)
                    recs[S.acc_slot[a]] = seg_rec{idx, uint32_t(a), S.acc_t0[a], S.acc_t1[a]};
            n_polys[idx] = uint32_t(n_acc);
            status[idx] = st;
        }
        __syncwarp();
    }
}

// Numbers each span's polynomials up to its first failing step: step_seq[s]
// is the number of step s's first polynomial, NOT_KEPT from the failure on.
__global__ void __launch_bounds__(64) k_sgp4_number(uint32_t n_jobs, const uint32_t *__restrict__ base,
                                                    const uint32_t *__restrict__ n_steps,
                                                    const uint32_t *__restrict__ n_polys,
                                                    const int *__restrict__ status, const int *__restrict__ end,
                                                    uint32_t *__restrict__ step_seq, int *__restrict__ job_status,
                                                    uint32_t *__restrict__ job_committed)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_jobs) return;
    const uint32_t b = base[j], e = b + n_steps[j];
    uint32_t committed = 0;
    int st = 0;
    for (uint32_t s = b; s < e; ++s) {
        if (st == 0) st = status[s];
        step_seq[s] = st ? NOT_KEPT : committed;
        if (st == 0) committed += n_polys[s];
    }
    job_status[j] = st ? st : end[j];
    job_committed[j] = committed;
}

// Lays the pool out as the polyjectory, one warp per polynomial: segment
// dest = seg_base[job] + number, its coefficients (mizuba layout [order + 1][7]) and its end time; the
// first segment of each satellite also writes the start time.
__global__ void k_sgp4_gather(const double *__restrict__ pool, const seg_rec *__restrict__ recs, uint64_t n_slots,
                              const step_rec *__restrict__ steps, const uint32_t *__restrict__ step_seq,
                              const uint64_t *__restrict__ seg_base, const uint32_t *__restrict__ keep,
                              const uint32_t *__restrict__ job_sat, const uint64_t *__restrict__ sat_seg_off,
                              const uint64_t *__restrict__ sat_time_off, double *__restrict__ traj,
                              double *__restrict__ time, unsigned long long *bad_seg)
{
    constexpr unsigned per = OP1 * 7;
    const unsigned lane = threadIdx.x & 31;
    for (uint64_t slot = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5; slot < n_slots;
         slot += (uint64_t(gridDim.x) * blockDim.x) >> 5) {
        const seg_rec rc = recs[slot];
        if (rc.step == NOT_KEPT) continue;
        const uint32_t s0 = step_seq[rc.step], jb = steps[rc.step].job;
        if (s0 == NOT_KEPT || s0 + rc.seq >= keep[jb]) continue;
        const uint64_t dest = seg_base[jb] + s0 + rc.seq;
        // The polyjectory constructor's finiteness check (polyjectory.cpp:
        // 558-569), on the coefficients as they are laid out.
        bool finite = true;
        for (unsigned k = lane; k < per; k += 32) {
            const double v = pool[slot * per + k];
            finite = finite && isfinite(v);
            traj[dest * per + k] = v;
        }
        if (!finite) atomicMin(bad_seg, (unsigned long long)dest);
        if (lane == 0) {
            const uint32_t sat = job_sat[jb];
            const uint64_t local = dest - sat_seg_off[sat];
            time[sat_time_off[sat] + local + 1] = rc.t1;
            if (local == 0) time[sat_time_off[sat]] = rc.t0;
        }
    }
}

// Every element set at every time, one thread per propagation; consecutive
// threads take consecutive times of one set and so read its coefficients
// together.
__global__ void __launch_bounds__(128) k_sgp4_propagate(const sgp4::sat *sats, const int *__restrict__ init,
                                                        uint64_t n, const double *__restrict__ tsince, uint64_t n_t,
                                                        double *__restrict__ out, int *__restrict__ err)
{
    const uint64_t g = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    if (g >= n * n_t) return;
    const uint64_t i = g / n_t, t = g % n_t;
    int e = init[i];
    double *o = out + g * 6;
    bool state = false;
    if (e == 0) {
        double r[3], v[3];
        e = sgp4::propagate(sats[i], tsince[t], r, v);
        // Decay (6) has a state; the other errors come before there is one.
        state = e == 0 || e == 6;
        if (state)
            for (int k = 0; k < 3; ++k) {
                o[k] = r[k];
                o[3 + k] = v[k];
            }
    }
    if (!state)
        for (int k = 0; k < 6; ++k) o[k] = NAN;
    err[g] = e;
}

} // namespace sgp4pj

// ------------------------------------------------------------ host driver

namespace
{

[[noreturn]] void sgp4_cuda_fail(cudaError_t e, const char *what)
{
    throw std::runtime_error(std::string("CUDA error in ") + what + ": " + cudaGetErrorString(e));
}
#define SK(x)                                                                                                        \
    do {                                                                                                               \
        const cudaError_t e_ = (x);                                                                                    \
        if (e_ != cudaSuccess) sgp4_cuda_fail(e_, #x);                                                                 \
    } while (0)

// A device's pool for this file's buffers and the produced coefficients, apart
// from the default one, whose blocks stay with the process: up to KEEP bytes
// stay between calls (production of 3,000 element sets over a day takes half of
// that), more goes back to the device at the next synchronisation, and
// mzb_scratch_release gives back all that is not in use.  Blocks of LARGE bytes
// or more (whole catalogues over days) are the device's own allocations instead,
// which cost 1.2 ms for 4 GB and go back when freed: from the pool, past KEEP,
// every synchronisation of a call unmapped what its next buffers mapped again (7
// ms a gigabyte; one day of 26,389 element sets 57 -> 350 ms).
constexpr uint64_t KEEP = uint64_t(2) << 30;
constexpr size_t LARGE = size_t(512) << 20;

cudaMemPool_t g_pools[64];
std::once_flag g_pool_flags[64];
cudaMemPool_t device_pool()
{
    int dev = 0;
    SK(cudaGetDevice(&dev));
    std::call_once(g_pool_flags[dev & 63], [dev]() {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool;
        SK(cudaMemPoolCreate(&pool, &props));
        uint64_t keep = KEEP;
        SK(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        g_pools[dev & 63] = pool;
    });
    return g_pools[dev & 63];
}

void *device_alloc(size_t bytes)
{
    void *p = nullptr;
    if (bytes >= LARGE) SK(cudaMalloc(&p, bytes));
    else if (bytes) SK(cudaMallocFromPoolAsync(&p, bytes, device_pool(), 0));
    return p;
}
void device_free(void *p, size_t bytes)
{
    if (bytes >= LARGE) cudaFree(p);
    else if (p) cudaFreeAsync(p, 0);
}

// A device buffer, on the legacy default stream (all of this file's work is on
// it).
template <typename T>
struct devbuf {
    T *p = nullptr;
    size_t n = 0;
    devbuf() = default;
    explicit devbuf(size_t count) { alloc(count); }
    devbuf(const devbuf &) = delete;
    devbuf &operator=(const devbuf &) = delete;
    ~devbuf() { release(); }
    void release()
    {
        device_free(p, n * sizeof(T));
        p = nullptr;
        n = 0;
    }
    void alloc(size_t count)
    {
        release();
        p = static_cast<T *>(device_alloc(count * sizeof(T)));
        n = count;
    }
};

std::string fmt_g(double x)
{
    char buf[64];
    std::snprintf(buf, sizeof(buf), "%.17g", x);
    return buf;
}

// TAI - UTC in seconds from 1972 on (IERS Bulletin C): the Julian date of
// 0h UTC on which each value takes effect.
struct leap {
    double jd;
    double dat;
};
const leap LEAPS[] = {
    {2441317.5, 10}, {2441499.5, 11}, {2441683.5, 12}, {2442048.5, 13}, {2442413.5, 14}, {2442778.5, 15},
    {2443144.5, 16}, {2443509.5, 17}, {2443874.5, 18}, {2444239.5, 19}, {2444786.5, 20}, {2445151.5, 21},
    {2445516.5, 22}, {2446247.5, 23}, {2447161.5, 24}, {2447892.5, 25}, {2448257.5, 26}, {2448804.5, 27},
    {2449169.5, 28}, {2449534.5, 29}, {2450083.5, 30}, {2450630.5, 31}, {2451179.5, 32}, {2453736.5, 33},
    {2454832.5, 34}, {2456109.5, 35}, {2457204.5, 36}, {2457754.5, 37},
};

double dat_at(double jd0)
{
    double d = LEAPS[0].dat;
    for (const leap &l : LEAPS)
        if (jd0 >= l.jd) d = l.dat;
    return d;
}

} // namespace

namespace sgp4pj
{

// UTC -> TAI for a double-length Julian date, from 1972 on, the way the IAU
// SOFA library's utctai does it: the instant's UTC day starts at jd0 (0h),
// TAI - UTC at 0h (dat0) applies to the whole day, and on a day that ends
// with a leap second the day's fraction is stretched over 86400 + 1 SI
// seconds.
dfl utc_to_tai(dfl utc)
{
    if (utc.hi < LEAPS[0].jd) throw std::invalid_argument("UTC dates before 1972 are not supported by make_sgp4_polyjectory()");
    const double jd0 = std::floor(utc.hi - 0.5) + 0.5;
    dfl frac = dfl_sub(utc, dfl{jd0, 0.0});
    if (frac.hi < 0) frac = dfl_add(frac, 1.0);
    const double dat0 = dat_at(jd0), dat24 = dat_at(jd0 + 1.0);
    const double dleap = dat24 - dat0;
    const double scale = (86400.0 + dleap) / 86400.0;
    const double f = (frac.hi + frac.lo) * scale;
    return dfl_add(dfl_add(dfl{jd0, 0.0}, f), dat0 / 86400.0);
}

void gpe_check(const gpe_host *g, uint64_t n, double jd_begin, double jd_end, double reentry, double exit_r)
{
    if (!std::isfinite(jd_begin) || !std::isfinite(jd_end) || !(jd_begin < jd_end))
        throw std::invalid_argument("Invalid Julian date interval [" + fmt_g(jd_begin) + ", " + fmt_g(jd_end)
                                    + ") supplied to make_sgp4_polyjectory(): the begin/end dates must be finite and "
                                      "the end date must be strictly after the begin date");
    if (std::isnan(reentry) || std::isnan(exit_r))
        throw std::invalid_argument("The reentry/exit radiuses in make_sgp4_polyjectory() cannot be NaN");
    if (!(reentry < exit_r))
        throw std::invalid_argument("The reentry radius (" + fmt_g(reentry) + ") must be less than the exit radius ("
                                    + fmt_g(exit_r) + ") in make_sgp4_polyjectory()");
    if (n == 0) throw std::invalid_argument("make_sgp4_polyjectory() requires a non-empty array of GPEs in input");
    // make_sgp4_polyjectory.cpp:123-148: every field finite, in field order.
    static const char *names[] = {"epoch_jd1", "epoch_jd2", "n0", "e0", "i0", "node0", "omega0", "m0", "bstar"};
    for (uint64_t i = 0; i < n; ++i) {
        const double f[] = {g[i].epoch_jd1, g[i].epoch_jd2, g[i].n0,     g[i].e0,   g[i].i0,
                            g[i].node0,     g[i].omega0,    g[i].m0,     g[i].bstar};
        for (int k = 0; k < 9; ++k)
            if (!std::isfinite(f[k]))
                throw std::invalid_argument(std::string("Invalid GPE detected by make_sgp4_polyjectory(): the '")
                                            + names[k] + "' of the GPE at index " + std::to_string(i)
                                            + " is not finite");
    }
    // make_sgp4_polyjectory.cpp:150-185: sorted by NORAD ID, then epoch,
    // and no two sets of one satellite with the same epoch.
    for (uint64_t i = 0; i + 1 < n; ++i) {
        const gpe_host &a = g[i], &b = g[i + 1];
        bool unsorted = b.norad_id < a.norad_id;
        if (b.norad_id == a.norad_id) {
            const dfl ea = dfl_norm(a.epoch_jd1, a.epoch_jd2), eb = dfl_norm(b.epoch_jd1, b.epoch_jd2);
            unsorted = dfl_lt(eb, ea);
            if (!unsorted && !dfl_lt(ea, eb))
                throw std::invalid_argument("Two GPEs with identical NORAD ID " + std::to_string(a.norad_id)
                                            + " and epoch (" + fmt_g(b.epoch_jd1) + ", " + fmt_g(b.epoch_jd2)
                                            + ") were identified by make_sgp4_polyjectory() - this is not allowed");
        }
        if (unsorted)
            throw std::invalid_argument("The set of GPEs passed to make_sgp4_polyjectory() is not sorted correctly: "
                                        "it must be ordered first by NORAD ID and then by epoch");
    }
}

sgp4_pj_out *make_sgp4_pj(const gpe_host *g, uint64_t n, double jd_begin, double jd_end, double reentry,
                          double exit_r)
{
    gpe_check(g, n, jd_begin, jd_end, reentry, exit_r);
    auto out = std::make_unique<sgp4_pj_out>();
    const dfl jb{jd_begin, 0.0}, je{jd_end, 0.0};
    out->epoch = utc_to_tai(jb);
    // Satellites (runs of equal NORAD IDs) and their spans
    // (make_sgp4_polyjectory.cpp:1261-1330).
    std::vector<job> jobs;
    std::vector<uint32_t> sat_first_job;
    uint32_t n_sats = 0;
    for (uint64_t i0 = 0; i0 < n;) {
        uint64_t i1 = i0 + 1;
        while (i1 < n && g[i1].norad_id == g[i0].norad_id) ++i1;
        // The last set with epoch <= jd_begin (or the first set).
        uint64_t it = i0;
        while (it + 1 < i1 && dfl_le(dfl_norm(g[it + 1].epoch_jd1, g[it + 1].epoch_jd2), jb)) ++it;
        sat_first_job.push_back(uint32_t(jobs.size()));
        dfl ibeg = jb;
        for (uint32_t k = 0;; ++k) {
            bool last = false;
            dfl iend;
            if (it + 1 == i1) {
                iend = je;
                last = true;
            } else {
                const dfl ne = dfl_norm(g[it + 1].epoch_jd1, g[it + 1].epoch_jd2);
                if (!dfl_lt(ne, je)) {
                    iend = je;
                    last = true;
                } else {
                    iend = ne;
                }
            }
            const gpe_host &e = g[it];
            job J{};
            J.n0 = e.n0;
            J.e0 = e.e0;
            J.i0 = e.i0;
            J.node0 = e.node0;
            J.omega0 = e.omega0;
            J.m0 = e.m0;
            J.bstar = e.bstar;
            J.epoch1950 = dfl_sub(dfl_norm(e.epoch_jd1, e.epoch_jd2), dfl{2433281.5, 0.0}).hi;
            J.epoch_tai = utc_to_tai(dfl_norm(e.epoch_jd1, e.epoch_jd2));
            J.begin_tai = utc_to_tai(ibeg);
            J.end_tai = utc_to_tai(iend);
            J.sat = n_sats;
            J.k = k;
            jobs.push_back(J);
            if (last) break;
            ibeg = dfl_norm(g[it + 1].epoch_jd1, g[it + 1].epoch_jd2);
            ++it;
        }
        ++n_sats;
        i0 = i1;
    }
    sat_first_job.push_back(uint32_t(jobs.size()));
    const uint32_t n_jobs = uint32_t(jobs.size());

    nodes_t nd{};
    for (int i = 0; i < OP1; ++i)
        nd.c[OP1 - 1 - i] = std::cos((2. * i + 1) / (2. * OP1) * 3.14159265358979323846);

    devbuf<job> d_jobs(n_jobs);
    SK(cudaMemcpy(d_jobs.p, jobs.data(), n_jobs * sizeof(job), cudaMemcpyHostToDevice));
    // Execution order: decreasing mean motion x span length (the number of
    // Keplerian steps a span takes grows with both).
    std::vector<uint32_t> order(n_jobs);
    for (uint32_t j = 0; j < n_jobs; ++j) order[j] = j;
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
        const double wa = jobs[a].n0 * dfl_sub(jobs[a].end_tai, jobs[a].begin_tai).hi;
        const double wb = jobs[b].n0 * dfl_sub(jobs[b].end_tai, jobs[b].begin_tai).hi;
        return wa > wb;
    });
    devbuf<uint32_t> d_order(n_jobs);
    SK(cudaMemcpy(d_order.p, order.data(), n_jobs * sizeof(uint32_t), cudaMemcpyHostToDevice));
    devbuf<sgp4::sat> d_sats(n_jobs);
    devbuf<int> d_init(n_jobs), d_end(n_jobs), d_status(n_jobs), d_overflow(1);
    devbuf<uint32_t> d_nsteps(n_jobs), d_base(n_jobs), d_committed(n_jobs);
    devbuf<unsigned long long> d_count(1), d_nredo(1);
    const double span_s = (jd_end - jd_begin) * 86400.0;
    const uint64_t max_steps = uint64_t(span_s) + 16;
    // Room for about 150 steps a day per span for low orbits, grown and run
    // again when it is not enough.
    uint64_t cap = uint64_t(n_jobs) * 64 + uint64_t(std::ceil(std::max(1.0, jd_end - jd_begin)) * 160.0) * n_sats;
    devbuf<step_rec> found, steps;
    devbuf<double> pool;
    devbuf<seg_rec> recs;
    devbuf<uint32_t> n_polys, redo, step_seq;
    devbuf<int> step_status;
    unsigned long long n_steps = 0, count = 0;
    int dev = 0, n_sm = 148;
    SK(cudaGetDevice(&dev));
    SK(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    struct ev_pair {
        cudaEvent_t a = nullptr, b = nullptr;
        ev_pair()
        {
            SK(cudaEventCreate(&a));
            SK(cudaEventCreate(&b));
        }
        ~ev_pair()
        {
            cudaEventDestroy(a);
            cudaEventDestroy(b);
        }
        float ms() const
        {
            float t = 0;
            cudaEventElapsedTime(&t, a, b);
            return t;
        }
    } ev_k, ev_g;
    SK(cudaEventRecord(ev_k.a));
    k_sgp4_setup<<<(n_jobs + 63) / 64, 64>>>(d_jobs.p, n_jobs, d_sats.p, d_init.p);
    ++out->n_launches;
    for (;;) {
        found.alloc(cap);
        SK(cudaMemsetAsync(d_count.p, 0, sizeof(unsigned long long)));
        k_sgp4_steps<<<(n_jobs + 31) / 32, 32>>>(d_jobs.p, n_jobs, d_order.p, d_sats.p, d_init.p, out->epoch,
                                                 reentry, exit_r, max_steps, found.p, cap, d_count.p, d_nsteps.p,
                                                 d_end.p);
        ++out->n_launches;
        SK(cudaGetLastError());
        SK(cudaMemcpy(&n_steps, d_count.p, sizeof(n_steps), cudaMemcpyDeviceToHost));
        if (n_steps <= cap) break;
        cap = n_steps;
    }
    if (n_steps >= NOT_KEPT) throw std::runtime_error("too many interpolation steps in make_sgp4_polyjectory()");
    steps.alloc(n_steps);
    n_polys.alloc(n_steps);
    redo.alloc(n_steps);
    step_seq.alloc(n_steps);
    step_status.alloc(n_steps);
    k_sgp4_bases<<<1, 1024>>>(d_order.p, n_jobs, d_nsteps.p, d_base.p);
    if (n_steps) k_sgp4_place<<<unsigned((n_steps + 255) / 256), 256>>>(found.p, n_steps, d_base.p, steps.p);
    out->n_launches += 2;
    found.release();
    // Pool: a slot per step, and room for the polynomials of bisected ones
    // behind them.
    cap = n_steps + n_steps / 8 + 4096;
    for (; n_steps;) {
        pool.alloc(cap * OP1 * 7);
        recs.alloc(cap);
        SK(cudaMemcpyAsync(d_count.p, &n_steps, sizeof(n_steps), cudaMemcpyHostToDevice, 0));
        SK(cudaMemsetAsync(d_overflow.p, 0, sizeof(int)));
        SK(cudaMemsetAsync(d_nredo.p, 0, sizeof(unsigned long long)));
        SK(cudaMemsetAsync(step_status.p, 0, n_steps * sizeof(int)));
        k_sgp4_interp<<<unsigned((n_steps + INTERP_STEPS - 1) / INTERP_STEPS), INTERP_T>>>(
            steps.p, n_steps, d_sats.p, nd, pool.p, recs.p, n_polys.p, redo.p, d_nredo.p);
        // Every polynomial of a step, the ones of a step that fails in the
        // end included, takes a slot.
        k_sgp4_bisect<<<n_sm * 4, 32 * WARPS>>>(steps.p, d_sats.p, nd, redo.p, d_nredo.p, pool.p, recs.p, cap,
                                                 d_count.p, d_overflow.p, n_polys.p, step_status.p);
        out->n_launches += 2;
        SK(cudaGetLastError());
        SK(cudaMemcpy(&count, d_count.p, sizeof(count), cudaMemcpyDeviceToHost));
        if (count <= cap) break;
        cap = count + count / 8 + 1024;
    }
    k_sgp4_number<<<(n_jobs + 63) / 64, 64>>>(n_jobs, d_base.p, d_nsteps.p, n_polys.p, step_status.p, d_end.p,
                                              step_seq.p, d_status.p, d_committed.p);
    ++out->n_launches;
    SK(cudaEventRecord(ev_k.b));
    SK(cudaGetLastError());
    std::vector<int> status(n_jobs);
    std::vector<uint32_t> committed(n_jobs);
    SK(cudaMemcpy(status.data(), d_status.p, n_jobs * sizeof(int), cudaMemcpyDeviceToHost));
    out->kernel_ms = ev_k.ms();
    SK(cudaMemcpy(committed.data(), d_committed.p, n_jobs * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    // Per satellite: its spans in order up to the first that failed (the
    // failing span keeps the steps completed before the error).
    std::vector<uint64_t> seg_base(n_jobs, 0), sat_seg_off(n_sats), sat_time_off(n_sats);
    std::vector<uint32_t> keep(n_jobs, 0), job_sat(n_jobs);
    out->status.assign(n_sats, 0);
    out->traj_off.resize(2 * size_t(n_sats));
    out->time_off.resize(n_sats);
    uint64_t seg_cursor = 0, time_cursor = 0;
    for (uint32_t s = 0; s < n_sats; ++s) {
        sat_seg_off[s] = seg_cursor;
        sat_time_off[s] = time_cursor;
        uint64_t nseg = 0;
        for (uint32_t j = sat_first_job[s]; j < sat_first_job[s + 1]; ++j) {
            job_sat[j] = s;
            seg_base[j] = seg_cursor + nseg;
            keep[j] = committed[j];
            nseg += committed[j];
            if (status[j] != 0) {
                out->status[s] = status[j];
                for (uint32_t q = j + 1; q < sat_first_job[s + 1]; ++q) job_sat[q] = s;
                break;
            }
        }
        out->traj_off[2 * s] = seg_cursor * OP1 * 7;
        out->traj_off[2 * s + 1] = nseg;
        out->time_off[s] = time_cursor;
        seg_cursor += nseg;
        time_cursor += nseg ? nseg + 1 : 0;
    }
    devbuf<uint64_t> d_seg_base(n_jobs), d_sat_seg_off(n_sats), d_sat_time_off(n_sats);
    devbuf<uint32_t> d_keep(n_jobs), d_job_sat(n_jobs);
    SK(cudaMemcpy(d_seg_base.p, seg_base.data(), n_jobs * 8, cudaMemcpyHostToDevice));
    SK(cudaMemcpy(d_keep.p, keep.data(), n_jobs * 4, cudaMemcpyHostToDevice));
    SK(cudaMemcpy(d_job_sat.p, job_sat.data(), n_jobs * 4, cudaMemcpyHostToDevice));
    SK(cudaMemcpy(d_sat_seg_off.p, sat_seg_off.data(), n_sats * 8, cudaMemcpyHostToDevice));
    SK(cudaMemcpy(d_sat_time_off.p, sat_time_off.data(), n_sats * 8, cudaMemcpyHostToDevice));
    out->n_traj = seg_cursor * OP1 * 7;
    out->dev = dev;
    out->d_traj = static_cast<double *>(device_alloc(out->n_traj * sizeof(double)));
    devbuf<double> d_time(time_cursor);
    devbuf<unsigned long long> d_bad(1);
    SK(cudaMemset(d_bad.p, 0xff, sizeof(unsigned long long)));
    if (seg_cursor) {
        SK(cudaEventRecord(ev_g.a));
        k_sgp4_gather<<<n_sm * 8, 256>>>(pool.p, recs.p, count, steps.p, step_seq.p, d_seg_base.p, d_keep.p,
                                          d_job_sat.p, d_sat_seg_off.p, d_sat_time_off.p, out->d_traj, d_time.p,
                                          d_bad.p);
        SK(cudaEventRecord(ev_g.b));
        ++out->n_launches;
        SK(cudaGetLastError());
    }
    out->time.resize(time_cursor);
    unsigned long long bad = ~0ull;
    if (seg_cursor) {
        SK(cudaMemcpy(out->time.data(), d_time.p, out->time.size() * 8, cudaMemcpyDeviceToHost));
        SK(cudaMemcpy(&bad, d_bad.p, sizeof(bad), cudaMemcpyDeviceToHost));
        out->gather_ms = ev_g.ms();
    }
    if (bad != ~0ull) {
        uint32_t s = 0;
        while (s + 1 < n_sats && sat_seg_off[s + 1] <= bad) ++s;
        throw std::invalid_argument("A non-finite value was found in the trajectory at index " + std::to_string(s));
    }
    for (uint32_t s = 0; s < n_sats; ++s)
        if (out->traj_off[2 * s + 1]) {
            const double te = out->time[out->time_off[s] + out->traj_off[2 * s + 1]];
            out->maxT = std::max(out->maxT, te);
        }
    return out.release();
}

void free_sgp4_pj(sgp4_pj_out *p) { delete p; }

sgp4_pj_out::~sgp4_pj_out()
{
    if (!d_traj) return;
    int cur = 0;
    cudaGetDevice(&cur);
    cudaSetDevice(dev);
    device_free(d_traj, n_traj * sizeof(double));
    cudaSetDevice(cur);
}

void release_scratch()
{
    const cudaMemPool_t pool = device_pool();
    SK(cudaStreamSynchronize(0)); // the frees queued so far
    SK(cudaMemPoolTrimTo(pool, 0));
}

uint64_t scratch_bytes()
{
    uint64_t b = 0;
    SK(cudaMemPoolGetAttribute(device_pool(), cudaMemPoolAttrReservedMemCurrent, &b));
    return b;
}

void sgp4_propagate(const gpe_host *g, uint64_t n, const double *tsince, uint64_t n_t, double *out, int32_t *err)
{
    if (n == 0 || n_t == 0) return;
    std::vector<double> keep_t;
    const double *ht = tsince;
    {
        cudaPointerAttributes pa{};
        if (cudaPointerGetAttributes(&pa, tsince) == cudaSuccess && pa.type == cudaMemoryTypeDevice) {
            keep_t.resize(n_t);
            SK(cudaMemcpy(keep_t.data(), tsince, n_t * 8, cudaMemcpyDeviceToHost));
            ht = keep_t.data();
        }
        cudaGetLastError();
    }
    for (uint64_t k = 0; k < n_t; ++k)
        if (!std::isfinite(ht[k]))
            throw std::invalid_argument("A non-finite propagation time was passed to mzb_sgp4_propagate()");
    // Arrays in this device's memory are read and written in place if they are
    // aligned as the kernels' loads and stores need; others go through buffers.
    int dev = 0;
    SK(cudaGetDevice(&dev));
    auto here = [dev](const auto *p) {
        if (reinterpret_cast<uintptr_t>(p) % alignof(std::remove_pointer_t<decltype(p)>) != 0) return false;
        cudaPointerAttributes pa{};
        const bool ok = cudaPointerGetAttributes(&pa, p) == cudaSuccess;
        if (!ok) cudaGetLastError();
        return ok && pa.type == cudaMemoryTypeDevice && pa.device == dev;
    };
    const bool g_here = here(g), t_here = here(tsince), out_here = here(out), err_here = here(err);
    devbuf<gpe_host> d_g(g_here ? 0 : n);
    devbuf<char> d_set(n * (sizeof(sgp4::sat) + sizeof(int))); // set-ups, then their error codes
    sgp4::sat *const sats = reinterpret_cast<sgp4::sat *>(d_set.p);
    int *const init = reinterpret_cast<int *>(sats + n);
    devbuf<double> d_t(t_here ? 0 : n_t), d_out(out_here ? 0 : n * n_t * 6);
    devbuf<int> d_err(err_here ? 0 : n * n_t);
    double *po = out_here ? out : d_out.p;
    int *pe = err_here ? err : d_err.p;
    if (!g_here) SK(cudaMemcpyAsync(d_g.p, g, n * sizeof(gpe_host), cudaMemcpyDefault, 0));
    if (!t_here) SK(cudaMemcpyAsync(d_t.p, tsince, n_t * 8, cudaMemcpyDefault, 0));
    k_sgp4_setup_gpes<<<unsigned((n + 63) / 64), 64>>>(g_here ? g : d_g.p, n, sats, init);
    k_sgp4_propagate<<<unsigned((n * n_t + 127) / 128), 128>>>(sats, init, n, t_here ? tsince : d_t.p, n_t, po, pe);
    SK(cudaGetLastError());
    if (!out_here) SK(cudaMemcpy(out, po, n * n_t * 6 * 8, cudaMemcpyDefault));
    if (!err_here) SK(cudaMemcpy(err, pe, n * n_t * 4, cudaMemcpyDefault));
    SK(cudaStreamSynchronize(0));
}

} // namespace sgp4pj
} // namespace mzb
