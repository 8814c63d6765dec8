/*
 * siminf_kernels.cuh -- the GB300 kernels of the ssm/mssm solver, as
 * templates over the device model, and their launchers.  siminf_kernels.cu
 * instantiates them for the models the library ships; a model compiled
 * from generated C code (siminf_gb300/devmodel.py) instantiates them in a
 * library of its own, with the same launcher table.
 *
 * The phases of a (replicate, node) pair g and their kernels:
 *   k_init       rate initialisation, a thread a node
 *                                          src/solvers/SimInf_solver_ssm.c:96-117
 *   k_ssa_e1     direct-method SSA up to the next unit of time, a thread or,
 *                for heavy nodes, a group of 8, 16 or 32 lanes a node
 *                                          src/solvers/SimInf_solver_ssm.c:144-235
 *                followed by the node's E1 events of the day
 *                                          src/solvers/SimInf_solver.c:658-822
 *   k_quick      the nodes whose day has no transition, ahead of k_ssa_e1
 *   k_e2_wave    one conflict-free wavefront of external transfers
 *                                          src/solvers/SimInf_solver.c:824-902
 *   k_e2_tail    a day's last wavefronts, in order, by one cluster
 *   k_pts_store  post time step, rate refresh, U/V store
 *                                          src/solvers/SimInf_solver_ssm.c:262-334
 *   k_horizon    all days of one node in one thread, for schedules without
 *                external transfers (nodes never interact)
 *
 * Node state lives in registers for the whole day (u as int[NC], rates as
 * double[NT]); S and the G column masks sit in shared memory so the
 * transition index can stay dynamic without spilling the register arrays.
 * Random draws come from the node's Philox stream (siminf_stream.h), and
 * the waiting-time logarithm is the integer fixed-point si_neglog_u32 (a
 * 32-bit-input -log(u) with two table reductions): on GB300 the FP64 pipe
 * retires one warp instruction per 64 cycles per SM sub-partition, while the
 * integer pipes are ~40x faster, so the SSA chain keeps only the FP64
 * operations the reference's arithmetic requires.
 *
 * Compiled with -fmad=false: every double operation rounds as in the
 * reference's C, which is what makes trajectories bit-identical.
 */
#ifndef SIMINF_KERNELS_CUH
#define SIMINF_KERNELS_CUH

#include <cfloat>
#include <climits>
#include <cstdint>
#include <cuda_runtime.h>

#include "siminf_stream.h"
#include "siminf_models.cuh"
#include "siminf_plan.h"
#include "siminf_launch.h"

namespace siminf {

enum { ERR_NEGATIVE_STATE = -1, ERR_UNDEFINED_EVENT = -3, ERR_SAMPLE_SELECT = -8,
       ERR_INVALID_RATE = -11, ERR_EVENTS_N = -15, ERR_EVENT_SHIFT = -16,
       ERR_SHIFT_OUT_OF_BOUNDS = -17, ERR_INVALID_PROPORTION = -18, ERR_TIMEOUT = -33 };


enum { EV_EXIT = 0, EV_ENTER = 1, EV_INTERNAL = 2, EV_EXTERNAL = 3 };

/* Out of line: errors are rare, and every kernel calls this. */
static __device__ __noinline__ void record_error(const DevState &s, int code, int phase,
                                                int day, long long g, int tr, int evi,
                                                double time, double rate)
{
    const int slot = atomicAdd(s.err_count, 1);
    atomicMin(s.err_day, day);
    if (phase <= PHASE_E1)
        atomicMin(s.err_day_pre_e2, day);
    if (slot < MAX_ERR) {
        ErrRec e;
        e.code = code;
        e.phase = phase;
        e.day = day;
        e.rep = (int) (g / s.Nn);
        e.node = (int) (g % s.Nn);
        e.transition = tr;
        e.event_index = evi;
        e.pad = 0;
        e.time = time;
        e.rate = rate;
        s.err[slot] = e;
    }
}

/* Replicate and node of g, without the ~150 instructions of a 64-bit
 * division where 32 bits or none will do. */
__device__ __forceinline__ int rep_of(const DevState &s, long long g)
{
    if (s.Nrep == 1)
        return 0;
    return s.Ntot <= 0xFFFFFFFFll ? (int) ((unsigned) g / (unsigned) s.Nn) : (int) (g / s.Nn);
}

__device__ __forceinline__ int node_of(const DevState &s, long long g)
{
    return (int) (g - (long long) rep_of(s, g) * s.Nn);
}

__device__ __forceinline__ const double *gdata_of(const DevState &s, long long g)
{
    if (s.job_of)
        return s.gdata + (size_t) s.job_of[g] * s.gdata_stride;
    if (s.gdata_stride == 0)
        return s.gdata;
    return s.gdata + (size_t) rep_of(s, g) * s.gdata_stride;
}

/* Key of node g's stream: (seed, replicate * Nn + node) for one model, the
 * job's own seed and local node index in a batch. */
__device__ __forceinline__ void stream_key(const DevState &s, long long g, uint64_t &seed,
                                           uint64_t &sid)
{
    if (s.job_of) {
        const int j = s.job_of[g];
        seed = s.job_seed[j];
        sid = (uint64_t) (g - s.job_node0[j]);
    } else {
        seed = s.pf_seeds ? s.pf_seeds[*s.pf_interval] : s.seed;
        sid = (uint64_t) g;
    }
}

/* Node g's model has run all its days (batches only). */
__device__ __forceinline__ bool job_over(const DevState &s, long long g, int day)
{
    return s.job_of && day >= s.job_ndays[s.job_of[g]];
}

__device__ __forceinline__ int load_flag(const int *p)
{
    return *(volatile const int *) p;
}

/* Sum the per-thread transition counts of a warp into the global counter. */
__device__ __forceinline__ void add_fired(const DevState &s, unsigned long long n)
{
    for (int o = 16; o > 0; o >>= 1)
        n += __shfl_down_sync(0xFFFFFFFFu, n, o);
    if ((threadIdx.x & 31) == 0 && n)
        atomicAdd(s.fired, n);
}

/* ------------------------------------------------------------------ */
/* Direct-method SSA of one node up to `next`                           */
/* (src/solvers/SimInf_solver_ssm.c:144-235), arranged for latency: the */
/* heaviest node of a day sets the day's critical path, and one node's  */
/* transitions form a chain of dependent operations, so everything that */
/* does not depend on the running sum leaves the chain:                 */
/*  - the two draws of the next transition (Philox block, -log(u) by    */
/*    si_neglog_u32, the selection uniform) are computed while the      */
/*    current transition updates the state, from the draw index alone;  */
/*  - the prefix sums of the rates, used by the inversion, are formed   */
/*    once per rate update, so choosing the transition is NT-1          */
/*    independent comparisons instead of a dependent add/compare chain; */
/*  - divisions, comparisons and int->double conversions run on the     */
/*    integer pipes (si_div, si_dge_num, si_i2d): same bits, and a      */
/*    rate's division by a population count reuses its prepared         */
/*    reciprocal (si_div_cached).                                       */
/* Draw i of the node's stream is word i & 3 of Philox block i >> 2; a  */
/* transition uses draws c (waiting time) and c + 1 (selection), so the */
/* next transition's pair lies in block (c + 3) >> 2, except the first  */
/* draw when (c + 2) & 3 == 3, which lies in the block this transition  */
/* fetched.                                                             */
/* ------------------------------------------------------------------ */
template <class M>
__device__ __forceinline__ void prefix_sums(const double (&rate)[M::NT], double (&cum)[M::NT])
{
    cum[0] = rate[0];
#pragma unroll
    for (int k = 1; k < M::NT; k++)
        cum[k] = cum[k - 1] + rate[k];
}

/* The transition the inversion picks (ssm.c:165-169): the first k with
 * !(rnd > rate[0] + ... + rate[k]), else NT - 1.  The prefix sums are
 * formed from the rates at each selection -- they depend on the rates
 * alone, so they run beside the rate sum's update -- instead of being
 * carried from step to step in registers. */
template <class M>
__device__ __forceinline__ int select_transition(const double (&rate)[M::NT], double rnd)
{
    double cum[M::NT];
    prefix_sums<M>(rate, cum);
    /* rnd > 0 and the sums are not NaN and not below zero: their bits
     * compare as integers, which leaves the FP64 pipe to the chain */
    int tr = M::NT - 1;
#pragma unroll
    for (int k = M::NT - 2; k >= 0; k--)
        if (!((int64_t) si_double_bits(rnd) > (int64_t) si_double_bits(cum[k])))
            tr = k;
    return tr;
}

__device__ __forceinline__ uint32_t word_of(uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3,
                                            uint32_t i)
{
    const uint32_t lo = (i & 1) ? b1 : b0, hi = (i & 1) ? b3 : b2;
    return (i & 2) ? hi : lo;
}

/* x <= 0.0 for the double with bits b (false for NaN), on the integer pipes. */
__device__ __forceinline__ bool le_zero(uint64_t b)
{
    return (int64_t) b <= 0 && !si_isnan_bits(b);
}

/* The double x's value as a float, truncated (normal range; from the bits). */
__device__ __forceinline__ float trunc_to_float(double x)
{
    const uint64_t b = si_double_bits(x);
    const int e = (int) ((b >> 52) & 0x7FF) - 1023 + 127;
    if (e <= 0)
        return 0.0f;
    if (e >= 255)
        return __int_as_float(0x7F800000);
    return __int_as_float((e << 23) | (int) ((b >> 29) & 0x7FFFFF));
}

/* Philox block `blk` of the stream held in r (key and stream id only). */
__device__ __forceinline__ void philox_block(const si_rng &r, uint64_t blk, uint32_t &b0,
                                             uint32_t &b1, uint32_t &b2, uint32_t &b3)
{
    b0 = (uint32_t) blk;
    b1 = (uint32_t) (blk >> 32);
    b2 = r.s0;
    b3 = r.s1;
    si_philox4x32_10(&b0, &b1, &b2, &b3, r.k0, r.k1);
}

/* The SSA state of one node during its day, held by one thread. */
template <class M>
struct SsaLane {
    int u[M::NC];
    double rate[M::NT];
    double sum, t, L, U, tau;
    uint64_t c;                       /* draw index of the next waiting time */
    uint32_t q0, q1, q2, q3;          /* Philox block (c + 1) >> 2 */
    unsigned fired;
    int err, err_tr;
    double err_t, err_rate;
    si_recip dc;
};

/* Start the day of a node whose u, rate, sum and t are loaded and whose
 * next draw is `c`; key holds the stream's key.  Returns true when nothing
 * fires today (rate sum <= 0, or not finite after a recorded invalid rate,
 * which would never reach `next`). */
template <class M>
__device__ __forceinline__ bool ssa_begin(SsaLane<M> &ln, const si_rng &key, uint64_t c,
                                          double next, const si_nl_tables *nl)
{
    ln.fired = 0;
    ln.c = c;
    if (!si_finite_pos(ln.sum)) {
        /* sum <= 0: nothing fires (ssm.c:148-151) */
        if (!le_zero(si_double_bits(ln.sum)) && !ln.err) {
            ln.err = ERR_INVALID_RATE;
            ln.err_tr = -1;
            ln.err_t = ln.t;
            ln.err_rate = ln.sum;
        }
        ln.t = next;
        return true;
    }
    /* the pair of the first transition */
    uint32_t p0, p1, p2, p3;
    philox_block(key, c >> 2, p0, p1, p2, p3);
    philox_block(key, (c + 1) >> 2, ln.q0, ln.q1, ln.q2, ln.q3);
    ln.L = si_neglog_u32_in(word_of(p0, p1, p2, p3, (uint32_t) c & 3u), nl);
    ln.U = si_u32_to_uniform_pos(word_of(ln.q0, ln.q1, ln.q2, ln.q3, (uint32_t) (c + 1) & 3u));
    if (!M::RATES_TIME_INVARIANT)
        ln.tau = si_div(ln.L, ln.sum);  /* ssa_step_ahead divides at each step */
    return false;
}

/* One step of the direct method for models whose rates do not read t:
 * the same operations as ssa_step_in_order, arranged so that the waiting
 * time's division (~550 cycles) does not hold up the next transition.
 * The transition the step would fire is selected and applied to copies of
 * the state while the division runs -- its rates need no time -- and the
 * copies replace the state only once the waiting time shows that it fires
 * before the day ends.  Returns true when the node's day is over.  It is
 * the exact path behind ssa_step_spec, taken only for that step's rare
 * cases, so it stays out of line: inlined, it doubled the code of the SSA
 * loop that every warp keeps in its instruction cache (3% of the headline
 * run's time). */
template <class M>
__device__ __noinline__ bool ssa_step_ahead(SsaLane<M> &ln, const si_rng &key, double next,
                                               const double *v, const double *ld,
                                               const double *gd, const int *sS,
                                               const uint32_t *sG, unsigned max_fired)
{
    constexpr int NC = M::NC, NT = M::NT;
    const double tau = si_div(ln.L, ln.sum);
    const double rnd = ln.U * ln.sum;

    int tr = select_transition<M>(ln.rate, rnd);
    double rtr = ln.rate[0];
#pragma unroll
    for (int k = 1; k < NT; k++)
        if (tr == k)
            rtr = ln.rate[k];
    bool nil = false;
    if (si_is_zero(rtr)) {
        /* Back-scan to the first non-zero rate (ssm.c:171-189). */
#pragma unroll
        for (int k = NT - 1; k >= 1; k--)
            if (tr == k && si_is_zero(ln.rate[k]))
                tr = k - 1;
        double r2 = ln.rate[0];
#pragma unroll
        for (int k = 1; k < NT; k++)
            if (tr == k)
                r2 = ln.rate[k];
        nil = si_is_zero(r2);
    }

    /* The state after that transition, in copies. */
    int u2[NC];
    int neg = 0;
#pragma unroll
    for (int cc = 0; cc < NC; cc++) {
        const int d = sS[tr * NC + cc];
        u2[cc] = ln.u[cc] + d;
        neg |= (d != 0) & (u2[cc] < 0);
    }
    double rate2[NT];
    double delta = 0.0;
    const uint32_t gm = sG[tr];
    int bad = -1;
    double bad_rate = 0.0;
#pragma unroll
    for (int k = 0; k < NT; k++) {
        rate2[k] = ln.rate[k];
        if (gm & (1u << k)) {
            const double nr = M::rate(k, u2, v, ld, gd, ln.t, ln.dc);
            rate2[k] = nr;
            delta += nr - ln.rate[k];
            if (si_bad_rate(nr)) {
                bad = k;
                bad_rate = nr;
            }
        }
    }
    const double sum2 = ln.sum + delta;

    /* Draws of the transition after it. */
    const uint64_t c2 = ln.c + 2;
    uint32_t n0, n1, n2, n3;
    philox_block(key, (c2 + 1) >> 2, n0, n1, n2, n3);
    const uint32_t ci = (uint32_t) c2 & 3u;
    const uint32_t wl = (ci == 3u) ? ln.q3 : word_of(n0, n1, n2, n3, ci);
    const uint32_t wu = word_of(n0, n1, n2, n3, (ci + 1u) & 3u);

    /* The waiting time decides: the day ends first, or the transition fires. */
    const double tn = tau + ln.t;
    if (tn >= next) {
        ln.t = next;
        ln.c += 1;                            /* the waiting time's draw was used */
        return true;
    }
    ln.t = tn;
    ln.c = c2;
    if (nil) {
        ln.sum = 0.0;
        return true;
    }
    if (++ln.fired > max_fired) {
        ln.err = ERR_TIMEOUT;
        ln.err_tr = tr;
        ln.err_t = ln.t;
        ln.t = next;
        return true;
    }
#pragma unroll
    for (int cc = 0; cc < NC; cc++)
        ln.u[cc] = u2[cc];
#pragma unroll
    for (int k = 0; k < NT; k++)
        ln.rate[k] = rate2[k];
    ln.sum = sum2;
    ln.q0 = n0;
    ln.q1 = n1;
    ln.q2 = n2;
    ln.q3 = n3;
    ln.L = si_neglog_u32(wl);
    ln.U = si_u32_to_uniform_pos(wu);
    if (neg) {
        ln.err = ERR_NEGATIVE_STATE;
        ln.err_tr = tr;
        ln.err_t = ln.t;
        ln.err_rate = 0.0;
    }
    if (bad >= 0) {
        ln.err = ERR_INVALID_RATE;
        ln.err_tr = bad;
        ln.err_t = ln.t;
        ln.err_rate = bad_rate;
    }
    if (!si_finite_pos(ln.sum)) {
        if (!le_zero(si_double_bits(ln.sum)) && !ln.err) {
            ln.err = ERR_INVALID_RATE;
            ln.err_tr = -1;
            ln.err_t = ln.t;
            ln.err_rate = ln.sum;
        }
        ln.t = next;
        return true;
    }
    return false;
}

/* The step of ssa_step_ahead as one block of straight-line code, for
 * the common case: no zero rate selected, no negative state, no invalid
 * or non-positive rate sum, no division off the integer path, a prepared
 * divisor that every rate's division finds in the cache, a waiting time
 * on the table path of -log(u), and the transition count within
 * max_fired.  Every rate is evaluated (and kept where its G bit is set),
 * so that no branch splits the block.  L and U are the step's -log(u) and
 * selection uniform; with NEXT, the step also computes the next step's
 * pair into ln.L and ln.U (the way ssa_step_ahead does), without it the
 * caller supplies every step's pair.  Returns SSA_FIRED or SSA_DAY_OVER
 * with the state updated exactly as ssa_step_ahead updates it, or
 * SSA_REDO with the state untouched when any of those conditions fails;
 * the caller then runs ssa_step_ahead on the same state and draws. */
enum { SSA_FIRED = 0, SSA_DAY_OVER = 1, SSA_REDO = 2 };

template <class M, bool NEXT>
__device__ __forceinline__ int ssa_step_spec(SsaLane<M> &ln, const si_rng &key, double L,
                                             double U, double next, const double *v,
                                             const double *ld, const double *gd, const int *sS,
                                             const uint32_t *sG, unsigned max_fired,
                                             const si_nl_tables *nl)
{
    constexpr int NC = M::NC, NT = M::NT;
    int tau_special = 0;
    const double tau = si_div_spec(L, ln.sum, &tau_special);
    const double rnd = U * ln.sum;

    int tr = select_transition<M>(ln.rate, rnd);
    double rtr = ln.rate[0];
#pragma unroll
    for (int k = 1; k < NT; k++)
        if (tr == k)
            rtr = ln.rate[k];
    int redo = si_is_zero(rtr);             /* the back-scan of ssm.c:171-189 */

    /* The state after that transition. */
    int u2[NC];
#pragma unroll
    for (int cc = 0; cc < NC; cc++) {
        const int d = sS[tr * NC + cc];
        u2[cc] = ln.u[cc] + d;
        redo |= (d != 0) & (u2[cc] < 0);
    }
    /* Every rate at that state; those flagged in column tr of G replace
     * the old ones and enter the delta in row order. */
    const uint32_t gm = sG[tr];
    si_recip_spec dcs;
    dcs.c = &ln.dc;
    dcs.flag = 0;
    double rate2[NT];
    double delta = 0.0;
#pragma unroll
    for (int k = 0; k < NT; k++) {
        const int f0 = dcs.flag;            /* a rate that is not kept flags nothing */
        const double nr = M::rate(k, u2, v, ld, gd, ln.t, dcs);
        const bool g = (gm >> k) & 1u;
        dcs.flag = g ? dcs.flag : f0;
        rate2[k] = g ? nr : ln.rate[k];
        /* (0.0 + x is x, but for a zero's sign, which a sum drops) */
        const double dk = k == 0 ? nr - ln.rate[k] : delta + (nr - ln.rate[k]);
        delta = g ? dk : delta;
        redo |= g & si_bad_rate(nr);
    }
    const double sum2 = ln.sum + delta;
    redo |= dcs.flag | !si_finite_pos(sum2);
    redo |= ln.fired + 1u > max_fired;

    /* Draws of the transition after it. */
    const uint64_t c2 = ln.c + 2;
    uint32_t n0 = 0, n1 = 0, n2 = 0, n3 = 0;
    double L2 = 0.0, U2 = 0.0;
    if constexpr (NEXT) {
        philox_block(key, (c2 + 1) >> 2, n0, n1, n2, n3);
        const uint32_t ci = (uint32_t) c2 & 3u;
        const uint32_t wl = (ci == 3u) ? ln.q3 : word_of(n0, n1, n2, n3, ci);
        const uint32_t wu = word_of(n0, n1, n2, n3, (ci + 1u) & 3u);
        L2 = si_neglog_u32_spec(wl, &redo, nl);
        U2 = si_u32_to_uniform_pos(wu);
    }

    if (tau_special)
        return SSA_REDO;
    const double tn = tau + ln.t;
    if (si_dge_num(tn, next)) {
        ln.t = next;
        ln.c += 1;                            /* the waiting time's draw was used */
        return SSA_DAY_OVER;
    }
    if (redo)
        return SSA_REDO;
    ln.t = tn;
    ln.c = c2;
    ln.fired++;
#pragma unroll
    for (int cc = 0; cc < NC; cc++)
        ln.u[cc] = u2[cc];
#pragma unroll
    for (int k = 0; k < NT; k++)
        ln.rate[k] = rate2[k];
    ln.sum = sum2;
    if constexpr (NEXT) {
        ln.q0 = n0;
        ln.q1 = n1;
        ln.q2 = n2;
        ln.q3 = n3;
        ln.L = L2;
        ln.U = U2;
    }
    return SSA_FIRED;
}

/* Draws of four transitions of a node whose next waiting-time draw is c:
 * words c .. c + 7 of its stream (waiting time, selection, four times),
 * from the three Philox blocks that can hold them, as -log(u) and
 * uniform values.  The four -log(u) are independent chains of integer
 * operations that the compiler interleaves. */
__device__ __forceinline__ void draw_four(const si_rng &key, uint64_t c, double (&L)[4],
                                          double (&U)[4], const si_nl_tables *nl)
{
    uint32_t w[12];
    const uint64_t b = c >> 2;
#pragma unroll
    for (int k = 0; k < 3; k++)
        philox_block(key, b + k, w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
    const uint32_t o = (uint32_t) c & 3u;
    uint32_t x[8];
#pragma unroll
    for (int i = 0; i < 8; i++)
        x[i] = o == 0 ? w[i] : o == 1 ? w[i + 1] : o == 2 ? w[i + 2] : w[i + 3];
    int slow = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        L[j] = si_neglog_u32_spec(x[2 * j], &slow, nl);
        U[j] = si_u32_to_uniform_pos(x[2 * j + 1]);
    }
    if (slow) {
#pragma unroll
        for (int j = 0; j < 4; j++)
            L[j] = si_neglog_u32_in(x[2 * j], nl);
    }
}

/* The rest of a node's day after ssa_begin, for models whose rates do not
 * read t: straight-line steps in batches of four, their draws computed
 * together ahead of them (draw_four); a step that meets a rare case is
 * redone by ssa_step_ahead with the same draws, and the next batch starts
 * at the draw index it leaves.  The draws, and so the trajectory, are
 * those of ssa_step. */
template <class M>
__device__ __forceinline__ void ssa_run_day(SsaLane<M> &ln, const si_rng &key, double next,
                                            const double *v, const double *ld, const double *gd,
                                            const int *sS, const uint32_t *sG,
                                            unsigned max_fired, const si_nl_tables *nl)
{
    for (;;) {
        double L[4], U[4];
        draw_four(key, ln.c, L, U, nl);
        int j = 0, st;
        double Lj, Uj;
        do {
            Lj = j == 0 ? L[0] : j == 1 ? L[1] : j == 2 ? L[2] : L[3];
            Uj = j == 0 ? U[0] : j == 1 ? U[1] : j == 2 ? U[2] : U[3];
            st = ssa_step_spec<M, false>(ln, key, Lj, Uj, next, v, ld, gd, sS, sG, max_fired, nl);
        } while (st == SSA_FIRED && ++j < 4);
        if (st == SSA_DAY_OVER)
            return;
        if (st == SSA_REDO) {
            /* the exact step, with this step's draws and the Philox block
             * of its selection draw, as ssa_step_ahead expects them */
            ln.L = Lj;
            ln.U = Uj;
            philox_block(key, (ln.c + 1) >> 2, ln.q0, ln.q1, ln.q2, ln.q3);
            if (ssa_step_ahead<M>(ln, key, next, v, ld, gd, sS, sG, max_fired))
                return;
        }
    }
}

/* One step of the direct method in the reference's order: the waiting
 * time ends the day, or one transition fires.  Returns true when the
 * node's day is over. */
template <class M>
__device__ __forceinline__ bool ssa_step_in_order(SsaLane<M> &ln, const si_rng &key,
                                                  double next, const double *v,
                                                  const double *ld, const double *gd,
                                                  const int *sS, const uint32_t *sG,
                                                  unsigned max_fired,
                                                  const si_nl_tables *nl)
{
    constexpr int NC = M::NC, NT = M::NT;
    const double tn = ln.tau + ln.t;
    /* the hardware FP64 comparisons of the chain (false on NaN): one
     * instruction each, ~3% off a transition's latency */
    if (tn >= next) {
        ln.t = next;
        ln.c += 1;                            /* the waiting time's draw was used */
        return true;
    }
    ln.t = tn;
    const double rnd = ln.U * ln.sum;
    ln.c += 2;

    /* Draws of the next transition, off the chain. */
    {
        uint32_t n0, n1, n2, n3;
        philox_block(key, (ln.c + 1) >> 2, n0, n1, n2, n3);
        const uint32_t ci = (uint32_t) ln.c & 3u;
        const uint32_t wl = (ci == 3u) ? ln.q3 : word_of(n0, n1, n2, n3, ci);
        const uint32_t wu = word_of(n0, n1, n2, n3, (ci + 1u) & 3u);
        ln.q0 = n0;
        ln.q1 = n1;
        ln.q2 = n2;
        ln.q3 = n3;
        ln.L = si_neglog_u32_in(wl, nl);
        ln.U = si_u32_to_uniform_pos(wu);
    }

    int tr = select_transition<M>(ln.rate, rnd);
    double rtr = ln.rate[0];
#pragma unroll
    for (int k = 1; k < NT; k++)
        if (tr == k)
            rtr = ln.rate[k];
    if (si_is_zero(rtr)) {
        /* Back-scan to the first non-zero rate (ssm.c:171-189). */
#pragma unroll
        for (int k = NT - 1; k >= 1; k--)
            if (tr == k && si_is_zero(ln.rate[k]))
                tr = k - 1;
        double r2 = ln.rate[0];
#pragma unroll
        for (int k = 1; k < NT; k++)
            if (tr == k)
                r2 = ln.rate[k];
        if (si_is_zero(r2)) {
            ln.sum = 0.0;
            return true;
        }
    }

    if (++ln.fired > max_fired) {
        /* Bounded work per node-day: a time step that stopped advancing t
         * (a rate sum near the overflow threshold) ends the run with an
         * error instead of spinning. */
        ln.err = ERR_TIMEOUT;
        ln.err_tr = tr;
        ln.err_t = ln.t;
        ln.t = next;
        return true;
    }
    int neg = 0;
#pragma unroll
    for (int cc = 0; cc < NC; cc++) {
        const int d = sS[tr * NC + cc];
        ln.u[cc] += d;
        neg |= (d != 0) & (ln.u[cc] < 0);
    }
    if (neg) {
        ln.err = ERR_NEGATIVE_STATE;
        ln.err_tr = tr;
        ln.err_t = ln.t;
        ln.err_rate = 0.0;
    }

    /* Refresh the rates flagged in column tr of G, in row order. */
    double delta = 0.0;
    const uint32_t gm = sG[tr];
    int bad = -1;
    double bad_rate = 0.0;
#pragma unroll
    for (int k = 0; k < NT; k++) {
        if (gm & (1u << k)) {
            const double old = ln.rate[k];
            const double nr = M::rate(k, ln.u, v, ld, gd, ln.t, ln.dc);
            ln.rate[k] = nr;
            delta += nr - old;
            if (si_bad_rate(nr)) {
                bad = k;
                bad_rate = nr;
            }
        }
    }
    if (bad >= 0) {
        ln.err = ERR_INVALID_RATE;
        ln.err_tr = bad;
        ln.err_t = ln.t;
        ln.err_rate = bad_rate;
    }
    ln.sum += delta;

    if (!si_finite_pos(ln.sum)) {
        if (!le_zero(si_double_bits(ln.sum)) && !ln.err) {
            ln.err = ERR_INVALID_RATE;
            ln.err_tr = -1;
            ln.err_t = ln.t;
            ln.err_rate = ln.sum;
        }
        ln.t = next;
        return true;
    }
    ln.tau = si_div(ln.L, ln.sum);
    return false;
}

/* One step of the direct method (src/solvers/SimInf_solver_ssm.c:
 * 144-235): where the rates do not read t, the straight-line speculative
 * step, redone ahead of the waiting time on the exact path when it meets
 * a rare case. */
template <class M>
__device__ __forceinline__ bool ssa_step(SsaLane<M> &ln, const si_rng &key, double next,
                                         const double *v, const double *ld, const double *gd,
                                         const int *sS, const uint32_t *sG, unsigned max_fired,
                                                  const si_nl_tables *nl)
{
    if constexpr (M::RATES_TIME_INVARIANT) {
        const int st = ssa_step_spec<M, true>(ln, key, ln.L, ln.U, next, v, ld, gd, sS, sG,
                                              max_fired, nl);
        if (st != SSA_REDO)
            return st == SSA_DAY_OVER;
        return ssa_step_ahead<M>(ln, key, next, v, ld, gd, sS, sG, max_fired);
    } else {
        return ssa_step_in_order<M>(ln, key, next, v, ld, gd, sS, sG, max_fired, nl);
    }
}

/* A node's whole SSA day in one call (used where one thread keeps one
 * node for the whole run and the rates read t). */
template <class M>
__device__ __forceinline__ unsigned ssa_day(SsaLane<M> &ln, si_rng &r, double next,
                                            const double *v, const double *ld, const double *gd,
                                            const int *sS, const uint32_t *sG, unsigned max_fired,
                                            const si_nl_tables *nl)
{
    if (!ssa_begin<M>(ln, r, r.ctr, next, nl))
        while (!ssa_step<M>(ln, r, next, v, ld, gd, sS, sG, max_fired, nl))
            ;
    r.ctr = ln.c;
    r.have = 0;
    return ln.fired;
}

/* ------------------------------------------------------------------ */
/* One node's day by a group of lanes.                                   */
/*                                                                       */
/* A node's transitions are a serial chain -- 3,800 cycles a step when   */
/* one lane runs it -- but what is serial in a step is small: the        */
/* transition's index.  A group of W lanes therefore takes the next W    */
/* steps at once, lane l step l:                                         */
/*  - the draws of W steps are W independent Philox blocks and           */
/*    logarithms;                                                        */
/*  - each lane guesses its step's transition from the rates at the      */
/*    batch's start; with the transitions guessed, the state after every */
/*    step is a count per transition over the lanes below (ballots);     */
/*  - each lane evaluates the rates at its state and selects again; the  */
/*    lanes whose transition changed give the next round's guess.  A     */
/*    round fixes at least the first wrong lane, and as the rates move   */
/*    slowly against the selection's thresholds two or three rounds      */
/*    settle all W;                                                      */
/*  - the rate sums and times, chains of rounded additions, are then     */
/*    formed in the reference's order from the settled steps' changes,   */
/*    and every selection is checked against the exact sum.              */
/* The steps before the first one past the day's end, or before the      */
/* first that needs the exact path (zero rate selected, negative state,  */
/* invalid rate, rate sum not positive, transition bound), are kept: the */
/* same draws and the same operations as ssa_step_in_order, so the same  */
/* bits.  Rates are also evaluated at states that are guessed wrongly    */
/* (no compartment below zero), which is why only the shipped models     */
/* take this path (model_rates_total).                                   */
/* ------------------------------------------------------------------ */

/* M::rate() may be evaluated at any state without a negative compartment:
 * the shipped models, whose rates are arithmetic on u; model C code may
 * index its data by u and keeps to states that the chain reaches. */
template <class M, class = void>
struct model_rates_total {
    static constexpr bool value = false;
};
template <class M>
struct model_rates_total<M, decltype((void) M::RATES_TOTAL)> {
    static constexpr bool value = M::RATES_TOTAL && M::RATES_TIME_INVARIANT;
};

/* The chain of rounded additions x, x + d_0, (x + d_0) + d_1, ... over the W
 * lanes of a group, each lane holding its d and getting the value before it
 * (every lane of the warp calls it; x the same in a group).  While the sums
 * stay in x's binade they are whole multiples of one unit in the last
 * place, and adding d rounds d to that unit: a whole number on its own,
 * except that a tie goes to the side that makes the sum even.  The parity
 * of every sum follows from the parities below it (a tie leaves an even
 * sum), so the chain is a prefix sum of whole numbers -- about 500 cycles
 * for 32 lanes, against 2,100 for 32 dependent additions on the FP64 pipe.
 * `right` has a bit for each lane of the group whose value is right: the
 * lanes up to the first whose sum leaves the binade. */
__device__ __forceinline__ double ordered_sums(double x, double d, int W, int lane, int l,
                                               unsigned group, unsigned below, unsigned &right)
{
    const unsigned FULL = 0xFFFFFFFFu;
    const uint64_t X = si_double_bits(x), D = si_double_bits(d);
    const int ex = (int) (X >> 52) & 0x7FF;
    const uint64_t mx = (X & 0x000FFFFFFFFFFFFFULL) | 0x0010000000000000ULL;
    const int ed = (int) (D >> 52) & 0x7FF;
    const uint64_t md = ed ? (D & 0x000FFFFFFFFFFFFFULL) | 0x0010000000000000ULL : 0;
    /* d in units of x's last place: md >> sh, its remainder against a half
     * (a subnormal d is far below half a unit of a normal x) */
    int sh = ex - ed;
    const bool fits = sh >= 0 && ex > 64 && ex < 0x7FE && !(X >> 63);
    sh = sh < 0 ? 0 : sh > 60 ? 60 : sh;
    const uint64_t q = md >> sh;
    const uint64_t twice = (md - (q << sh)) << 1, unit = 1ULL << sh;
    const bool tie = twice == unit;
    uint64_t r = q + (twice > unit);
    const unsigned ties = __ballot_sync(FULL, tie) & group & below;
    const unsigned odds = __ballot_sync(FULL, !tie && (r & 1)) & group & below;
    /* lanes at and above the last tie below me (all of them without one) */
    const unsigned since = ties ? 0xFFFFFFFFu << (31 - __clz((int) ties)) : 0xFFFFFFFFu;
    const unsigned odd = (__popc(odds & since) + (ties ? 0u : (unsigned) mx)) & 1u;
    if (tie)
        r += odd ^ ((unsigned) q & 1u);
    int64_t y = (D >> 63) ? -(int64_t) r : (int64_t) r;
    for (int o = 1; o < W; o <<= 1) {
        const int64_t z = __shfl_up_sync(FULL, y, o, W);
        if (l >= o)
            y += z;
    }
    const uint64_t after = mx + (uint64_t) y;           /* after my step */
    const bool in = fits && after > (1ULL << 52) && after < (1ULL << 53) - 1;
    const unsigned out = __ballot_sync(FULL, !in) & group;
    /* the first sum outside is still added to a right one */
    right = out ? group & ((2u << (__ffs(out) - 1)) - 1u) : group;
    uint64_t b = __shfl_up_sync(FULL, after, 1, W);
    b = ((uint64_t) ex << 52) | (b & 0x000FFFFFFFFFFFFFULL);
    return l == 0 ? x : si_bits_double(b);
}

/* The same chain by additions one after the other. */
__device__ __forceinline__ double ordered_sums_serial(double x, double d, int W, int l)
{
    double before = x;
    for (int j = 0; j < W; j++) {
        const double dj = __shfl_sync(0xFFFFFFFFu, d, j, W);
        if (l == j)
            before = x;
        x = x + dj;
    }
    return before;
}

/* Every lane of the warp calls it; the W lanes of a group (W = 8, 16 or 32,
 * groups aligned) hold the same ln, key and pointers, `live` says whether
 * the group has a node.  On return the group's first lane holds the state
 * at the day's end. */
template <class M>
__device__ __forceinline__ void ssa_day_group(SsaLane<M> &ln, const si_rng &key, const int W,
                                              bool live, double next, const double *v,
                                              const double *ld, const double *gd, const int *sS,
                                              const uint32_t *sG, unsigned max_fired,
                                              const si_nl_tables *nl)
{
    constexpr int NC = M::NC, NT = M::NT;
    constexpr uint32_t ALL = NT == 32 ? 0xFFFFFFFFu : (1u << NT) - 1u;
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, l = lane & (W - 1), base = lane - l;
    const unsigned group = (W == 32 ? FULL : ((1u << W) - 1u)) << base;
    const unsigned below = (1u << lane) - 1u;       /* with `group`: the steps before mine */
    ln.fired = 0;
    bool done = !live;                              /* the same in the whole group */
    if (live && !si_finite_pos(ln.sum)) {
        /* as ssa_begin: nothing fires, or an invalid rate */
        if (!le_zero(si_double_bits(ln.sum))) {
            ln.err = ERR_INVALID_RATE;
            ln.err_tr = -1;
            ln.err_t = ln.t;
            ln.err_rate = ln.sum;
        }
        ln.t = next;
        done = true;
    }
    while (__any_sync(FULL, !done)) {
        /* the draws of step l: words c + 2 l (waiting time) and c + 2 l + 1 */
        double L, U;
        {
            const uint64_t cw = ln.c + 2u * (unsigned) l;
            const uint32_t iw = (uint32_t) cw & 3u;
            uint32_t p0, p1, p2, p3;
            philox_block(key, (cw + 1) >> 2, p0, p1, p2, p3);
            /* when the selection's word opens a block, the waiting time's is
             * the last of the block before, which the lane below holds */
            uint32_t wl = __shfl_up_sync(FULL, p3, 1, W);
            if (iw != 3u) {
                wl = word_of(p0, p1, p2, p3, iw);
            } else if (l == 0) {
                uint32_t r0, r1, r2;
                philox_block(key, cw >> 2, r0, r1, r2, wl);
            }
            L = si_neglog_u32_in(wl, nl);
            U = si_u32_to_uniform_pos(word_of(p0, p1, p2, p3, (iw + 1u) & 3u));
        }
        int tr = select_transition<M>(ln.rate, U * ln.sum);
        int u2[NC];                                 /* the state after my step */
        double ra[NT], rb[NT];                      /* the rates after and before it */
        unsigned wrong, bad;
        /* steps that start past the day's end need not settle: their start
         * times at the rate sum of the batch's start, to single precision
         * and with a margin for the sum's changes */
        bool needed;
        {
            float x = trunc_to_float(L);
            for (int o = 1; o < W; o <<= 1) {
                const float y = __shfl_up_sync(FULL, x, o, W);
                if (l >= o)
                    x += y;
            }
            const float before = __shfl_up_sync(FULL, x, 1, W);
            needed = l == 0 || !(before > 1.25f * trunc_to_float(ln.sum) *
                                              trunc_to_float(next - ln.t));
        }
        for (;;) {
            int cnt[NT];
#pragma unroll
            for (int k = 0; k < NT; k++)
                cnt[k] = __popc(__ballot_sync(FULL, tr == k) & group & (below | (1u << lane)));
            bad = 0;
#pragma unroll
            for (int c = 0; c < NC; c++) {
                int x = ln.u[c];
#pragma unroll
                for (int k = 0; k < NT; k++)
                    x += sS[k * NC + c] * cnt[k];
                bad |= x < 0;
                u2[c] = x < 0 ? 0 : x;
            }
            const uint32_t gm = sG[tr];
            const bool all_full = __all_sync(FULL, gm == ALL);
            double cum = 0.0;
            double cums[NT];
#pragma unroll
            for (int k = 0; k < NT; k++) {
                const double nr = M::rate(k, u2, v, ld, gd, ln.t, ln.dc);
                const bool g = (gm >> k) & 1u;
                bad |= g & si_bad_rate(nr);
                /* rate k before my step: the one after the last step below
                 * that refreshed it, or the batch's first */
                int j = lane - 1;
                if (!all_full)
                    j = 31 - __clz((int) (__ballot_sync(FULL, g) & group & below));
                const double r = __shfl_sync(FULL, nr, j & 31);
                rb[k] = j < base ? ln.rate[k] : r;
                ra[k] = g ? nr : rb[k];
                cum = k == 0 ? rb[0] : cum + rb[k];
                cums[k] = cum;
            }
            /* select against the sum of the rates (the exact rate sum, which
             * differs from it in its last bits, checks the choice below) */
            const double rnd = U * cum;
            int ntr = NT - 1;
#pragma unroll
            for (int k = NT - 2; k >= 0; k--)
                if (!((int64_t) si_double_bits(rnd) > (int64_t) si_double_bits(cums[k])))
                    ntr = k;
            wrong = __ballot_sync(FULL, (ntr != tr) | !needed) & group;
            const bool more = __any_sync(FULL, !done && needed && ntr != tr);
            if (!more)
                break;
            tr = ntr;
        }
        /* the change of the rate sum by each step, then the sums in order */
        double delta = 0.0;
        {
            const uint32_t gm = sG[tr];
#pragma unroll
            for (int k = 0; k < NT; k++) {
                const double d = ra[k] - rb[k];
                const double dk = k == 0 ? d : delta + d;
                delta = (gm >> k) & 1u ? dk : delta;
            }
        }
        /* the lanes whose state before the step is known: up to the first
         * unsettled one, which may still end the day */
        const unsigned known = wrong ? group & ((2u << (__ffs(wrong) - 1)) - 1u) : group;
        /* the rate sum before and after my step */
        unsigned right;
        double sb = ordered_sums(ln.sum, delta, W, lane, l, group, below, right);
        if (__any_sync(FULL, !done && (known & ~right)))
            sb = ordered_sums_serial(ln.sum, delta, W, l);
        const double sa = sb + delta;
        /* the exact selection */
        double rtr = rb[0];
#pragma unroll
        for (int k = 1; k < NT; k++)
            if (tr == k)
                rtr = rb[k];
        bad |= si_is_zero(rtr) | (select_transition<M>(rb, U * sb) != tr) | !si_finite_pos(sa);
        bad |= ln.fired + (unsigned) l + 1u > max_fired;
        /* waiting times, then the times in order */
        const double tau = si_div(L, sb);
        double tb = ordered_sums(ln.t, tau, W, lane, l, group, below, right);
        if (__any_sync(FULL, !done && (known & ~right)))
            tb = ordered_sums_serial(ln.t, tau, W, l);
        const double tn = tau + tb;
        const unsigned over = __ballot_sync(FULL, si_dge_num(tn, next)) & group;
        const unsigned cut = __ballot_sync(FULL, bad != 0) & group;
        /* steps 0 .. n - 1 fire */
        const int first_over = over ? __ffs(over) - 1 - base : W;
        const int first_wrong = wrong ? __ffs(wrong) - 1 - base : W;
        const int first_cut = cut ? __ffs(cut) - 1 - base : W;
        const bool ends = first_over < W && first_over <= first_wrong && first_over <= first_cut;
        const int n = ends ? first_over : min(first_wrong, first_cut);
        const int src = base + (n > 0 ? n - 1 : 0);
        const bool take = !done && n > 0;
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const int x = __shfl_sync(FULL, u2[c], src);
            if (take)
                ln.u[c] = x;
        }
#pragma unroll
        for (int k = 0; k < NT; k++) {
            const double x = __shfl_sync(FULL, ra[k], src);
            if (take)
                ln.rate[k] = x;
        }
        {
            const double xs = __shfl_sync(FULL, sa, src), xt = __shfl_sync(FULL, tn, src);
            if (take) {
                ln.sum = xs;
                ln.t = xt;
                ln.c += 2u * (unsigned) n;
                ln.fired += (unsigned) n;
            }
        }
        if (!done) {
            if (ends) {
                ln.t = next;
                ln.c += 1;                          /* the waiting time's draw was used */
                done = true;
            } else if (n == first_cut && n < W) {
                /* the rest of the day on the exact path, by the first lane */
                if (l == 0) {
                    const unsigned f = ln.fired;
                    if (!ssa_begin<M>(ln, key, ln.c, next, nl)) {
                        ln.fired = f;
                        while (!ssa_step_ahead<M>(ln, key, next, v, ld, gd, sS, sG, max_fired))
                            ;
                    } else {
                        ln.fired = f;
                    }
                }
                done = true;
            }
        }
    }
}

/* ------------------------------------------------------------------ */
/* Event sampling on a node's compartments uu (src/solvers/             */
/* SimInf_solver.c:62-324), drawing from the node's stream.             */
/* ------------------------------------------------------------------ */
template <int NC>
__device__ int sample_select(const DevState &s, const int *uu, int select, int n,
                             double proportion, int *ind, si_rng *r)
{
    const int *irE = s.irE, *jcE = s.jcE;
    const double *prE = s.prE;
    int i, Nstates, Nindividuals = 0, Nkinds = 0;

    for (int c = 0; c < NC; c++)
        ind[c] = 0;
    for (i = jcE[select]; i < jcE[select + 1]; i++) {
        const int nk = uu[irE[i]];
        if (nk > 0)
            Nkinds++;
        Nindividuals += nk;
    }
    Nstates = jcE[select + 1] - jcE[select];
    if (n == 0) {
        if (proportion < 0 || proportion > 1)
            return ERR_INVALID_PROPORTION;
        n = si_binomial(r, proportion, Nindividuals);
    }
    if (s.cap && n > Nindividuals)
        n = Nindividuals;
    if (Nstates <= 0 || n > Nindividuals || n < 0)
        return ERR_SAMPLE_SELECT;
    if (n == 0)
        return 0;
    if (Nindividuals == n) {
        for (i = jcE[select]; i < jcE[select + 1]; i++)
            ind[irE[i]] = uu[irE[i]];
        return 0;
    }
    if (Nstates == 1) {
        ind[irE[jcE[select]]] = n;
        return 0;
    }
    if (Nkinds == 1) {
        for (i = jcE[select]; i < jcE[select + 1]; i++) {
            if (uu[irE[i]] > 0) {
                ind[irE[i]] = n;
                break;
            }
        }
        return 0;
    }
    bool equal = true;
    for (i = jcE[select] + 1; i < jcE[select + 1]; i++)
        if (prE[i] != prE[i - 1])
            equal = false;
    if (equal) {
        /* Sequential multivariate hypergeometric. */
        for (i = jcE[select]; i < jcE[select + 1] - 1; i++) {
            if (n == 0)
                break;
            const int nk = uu[irE[i]];
            ind[irE[i]] = si_hypergeometric(r, nk, Nindividuals - nk, n);
            Nindividuals -= nk;
            n -= ind[irE[i]];
        }
        ind[irE[i]] = n;
        return 0;
    }
    /* Wallenius' noncentral hypergeometric by a biased urn. */
    while (n > 0) {
        double rand, cum = 0;
        for (i = jcE[select]; i < jcE[select + 1]; i++)
            cum += prE[i] * (uu[irE[i]] - ind[irE[i]]);
        rand = si_uniform_pos(r) * cum;
        i = jcE[select];
        cum = prE[i] * (uu[irE[i]] - ind[irE[i]]);
        while (i < jcE[select + 1] && rand > cum) {
            i++;
            if (i < jcE[select + 1])
                cum += prE[i] * (uu[irE[i]] - ind[irE[i]]);
        }
        if (i >= jcE[select + 1])
            i = jcE[select + 1] - 1;
        if ((prE[i] * (uu[irE[i]] - ind[irE[i]])) == 0.0) {
            for (; i > jcE[select] && (prE[i] * (uu[irE[i]] - ind[irE[i]])) == 0.0; i--);
            if ((prE[i] * (uu[irE[i]] - ind[irE[i]])) == 0.0)
                return ERR_SAMPLE_SELECT;
        }
        ind[irE[i]] += 1;
        n--;
    }
    return 0;
}

template <int NC>
__device__ int sample_select_enter(const DevState &s, const int *uu, int select, int n,
                                   double proportion, int *ind, si_rng *r)
{
    const int *irE = s.irE, *jcE = s.jcE;
    const double *prE = s.prE;
    int i, Nstates = jcE[select + 1] - jcE[select];
    double w_cum = 0;

    for (int c = 0; c < NC; c++)
        ind[c] = 0;
    if (n == 0) {
        if (proportion < 0 || proportion > 1)
            return ERR_INVALID_PROPORTION;
        for (i = jcE[select]; i < jcE[select + 1]; i++)
            n += uu[irE[i]];
        n = si_binomial(r, proportion, n);
    }
    if (Nstates <= 0 || n < 0)
        return ERR_SAMPLE_SELECT;
    if (n == 0)
        return 0;
    if (Nstates == 1) {
        ind[irE[jcE[select]]] = n;
        return 0;
    }
    for (i = jcE[select]; i < jcE[select + 1]; i++)
        w_cum += prE[i];
    while (n > 0) {
        double cum, rand = si_uniform_pos(r) * w_cum;
        i = jcE[select];
        cum = prE[i];
        while (i < jcE[select + 1] && rand > cum) {
            i++;
            if (i < jcE[select + 1])
                cum += prE[i];
        }
        if (i >= jcE[select + 1])
            i = jcE[select + 1] - 1;
        if (prE[i] == 0.0) {
            for (; i > jcE[select] && prE[i] == 0.0; i--);
            if (prE[i] == 0.0)
                return ERR_SAMPLE_SELECT;
        }
        ind[irE[i]] += 1;
        n--;
    }
    return 0;
}

/* Apply one E1 event to the node's compartments uu
 * (src/solvers/SimInf_solver.c:680-822).  Returns 0 or an error code. */
template <int NC>
__device__ int apply_e1(const DevState &s, int *uu, const E1Rec &e, si_rng *r)
{
    int ind[NC];
    int err;
    const int *irE = s.irE, *jcE = s.jcE;

    switch (e.kind) {
    case EV_EXIT:
        err = sample_select<NC>(s, uu, e.select, e.n, e.proportion, ind, r);
        if (err)
            return err;
        for (int i = jcE[e.select]; i < jcE[e.select + 1]; i++) {
            const int jj = irE[i];
            uu[jj] -= ind[jj];
            if (uu[jj] < 0)
                return ERR_NEGATIVE_STATE;
        }
        return 0;
    case EV_ENTER:
        err = sample_select_enter<NC>(s, uu, e.select, e.n, e.proportion, ind, r);
        if (err)
            return err;
        for (int i = jcE[e.select]; i < jcE[e.select + 1]; i++) {
            const int jj = irE[i];
            if (e.shift < 0) {
                uu[jj] += ind[jj];
                if (uu[jj] < 0)
                    return ERR_NEGATIVE_STATE;
            } else if (!s.hasN) {
                return ERR_EVENTS_N;
            } else {
                const int ll = s.Nshift[e.shift * NC + jj];
                if (jj + ll < 0 || jj + ll >= NC)
                    return ERR_SHIFT_OUT_OF_BOUNDS;
                uu[jj + ll] += ind[jj];
                if (uu[jj + ll] < 0)
                    return ERR_NEGATIVE_STATE;
            }
        }
        return 0;
    case EV_INTERNAL:
        if (!s.hasN)
            return ERR_EVENTS_N;
        if (e.shift < 0)
            return ERR_EVENT_SHIFT;
        err = sample_select<NC>(s, uu, e.select, e.n, e.proportion, ind, r);
        if (err)
            return err;
        for (int i = jcE[e.select]; i < jcE[e.select + 1]; i++) {
            const int jj = irE[i];
            const int ll = s.Nshift[e.shift * NC + jj];
            if (jj + ll < 0 || jj + ll >= NC)
                return ERR_SHIFT_OUT_OF_BOUNDS;
            uu[jj + ll] += ind[jj];
            if (uu[jj + ll] < 0)
                return ERR_NEGATIVE_STATE;
            uu[jj] -= ind[jj];
            if (uu[jj] < 0)
                return ERR_NEGATIVE_STATE;
        }
        return 0;
    default:
        return ERR_UNDEFINED_EVENT;
    }
}

/* A node's place in its E1 events: the next one and its day (NO_E1 when
 * there is none).  A day's events are found by looking at that day alone,
 * where a bisection of the node's list was up to eight dependent loads. */
enum { NO_E1 = INT_MAX };

/* The E1 events of one node-day.  Inlined: a call would make the SSA
 * kernels save the registers live across it to local memory (spills),
 * while the samplers' code, after the SSA loop, runs only on the one
 * node-day in about 250 that has events.  State and stream counter go in
 * and out by value, so the caller's copies stay in registers. */
template <int NC>
struct E1Out {
    int u[NC];
    uint64_t ctr;
    int err_code, err_event;
    int2 at;
};

template <int NC>
__device__ __forceinline__ E1Out<NC> node_e1_apply(const DevState &s, E1Out<NC> o, si_rng r, int end,
                                                int day)
{
    int k = o.at.x;
    o.at.y = NO_E1;
    for (; k < end; k++) {
        const E1Rec e = s.e1[k];
        if (e.day != day) {
            o.at.y = e.day;
            break;
        }
        const int err = apply_e1<NC>(s, o.u, e, &r);
        if (err) {
            o.err_code = err;
            o.err_event = e.index;
            break;
        }
    }
    o.at.x = k;
    o.ctr = r.ctr;
    return o;
}

/* The node's E1 events of `day` (src/solvers/SimInf_solver.c:658-822), in
 * array order, applied to u with draws from r; `at`, the node's place in
 * its events, moves past them.  Returns true when an event was applied (the
 * node is then flagged for a rate refresh). */
template <int NC>
__device__ __forceinline__ bool node_e1(const DevState &s, int (&u)[NC], int2 &at, int node, int day,
                                        si_rng &r, int &err_code, int &err_event)
{
    if (at.y != day)
        return false;
    E1Out<NC> o;
#pragma unroll
    for (int c = 0; c < NC; c++)
        o.u[c] = u[c];
    o.ctr = r.ctr;
    o.err_code = 0;
    o.err_event = -1;
    o.at = at;
    o = node_e1_apply<NC>(s, o, r, s.e1_ptr[node + 1], day);
#pragma unroll
    for (int c = 0; c < NC; c++)
        u[c] = o.u[c];
    r.ctr = o.ctr;
    r.have = 0;
    at = o.at;
    if (o.err_code) {
        err_code = o.err_code;
        err_event = o.err_event;
    }
    return true;
}

/* node_e1 as a call, for k_horizon with models of at most two
 * compartments: inlined, its samplers take the registers the one-node-a-
 * thread loop keeps live and 12 bytes spill; called, they do not (and the
 * call is made only on a day with events). */
template <int NC>
__device__ __noinline__ bool node_e1_call(const DevState &s, int (&u)[NC], int2 &at, int node,
                                          int day, si_rng &r, int &err_code, int &err_event)
{
    return node_e1<NC>(s, u, at, node, day, r, err_code, err_event);
}

/* The NC compartments of one node, loaded or stored with 16-byte (NC a
 * multiple of 4) or 8-byte (NC even) accesses: a node's block of u or of a
 * U column starts at a multiple of NC ints from a 256-byte aligned base. */
template <int NC>
__device__ __forceinline__ void load_u(const int *p, int (&u)[NC])
{
    if constexpr (NC % 4 == 0) {
#pragma unroll
        for (int c = 0; c < NC; c += 4) {
            const int4 w = *reinterpret_cast<const int4 *>(p + c);
            u[c] = w.x;
            u[c + 1] = w.y;
            u[c + 2] = w.z;
            u[c + 3] = w.w;
        }
    } else if constexpr (NC % 2 == 0) {
#pragma unroll
        for (int c = 0; c < NC; c += 2) {
            const int2 w = *reinterpret_cast<const int2 *>(p + c);
            u[c] = w.x;
            u[c + 1] = w.y;
        }
    } else {
#pragma unroll
        for (int c = 0; c < NC; c++)
            u[c] = p[c];
    }
}

/* load_u from L2, past the SM's own cache. */
template <int NC>
__device__ __forceinline__ void load_u_l2(const int *p, int (&u)[NC])
{
    if constexpr (NC % 4 == 0) {
#pragma unroll
        for (int c = 0; c < NC; c += 4) {
            const int4 w = __ldcg(reinterpret_cast<const int4 *>(p + c));
            u[c] = w.x;
            u[c + 1] = w.y;
            u[c + 2] = w.z;
            u[c + 3] = w.w;
        }
    } else if constexpr (NC % 2 == 0) {
#pragma unroll
        for (int c = 0; c < NC; c += 2) {
            const int2 w = __ldcg(reinterpret_cast<const int2 *>(p + c));
            u[c] = w.x;
            u[c + 1] = w.y;
        }
    } else {
#pragma unroll
        for (int c = 0; c < NC; c++)
            u[c] = __ldcg(p + c);
    }
}

template <int NC>
__device__ __forceinline__ void store_u(int *p, const int (&u)[NC])
{
    if constexpr (NC % 4 == 0) {
#pragma unroll
        for (int c = 0; c < NC; c += 4)
            *reinterpret_cast<int4 *>(p + c) = make_int4(u[c], u[c + 1], u[c + 2], u[c + 3]);
    } else if constexpr (NC % 2 == 0) {
#pragma unroll
        for (int c = 0; c < NC; c += 2)
            *reinterpret_cast<int2 *>(p + c) = make_int2(u[c], u[c + 1]);
    } else {
#pragma unroll
        for (int c = 0; c < NC; c++)
            p[c] = u[c];
    }
}

/* Store the node's U/V entries for columns [c0, c1) of its replicate. */
template <int NC, int ND>
__device__ __forceinline__ void store_columns(const DevState &s, int rep, int node,
                                              const int (&u)[NC], const double *vnew,
                                              int c0, int c1)
{
    for (int col = c0; col < c1; col++) {
        const size_t ccol = (size_t) rep * s.tlen + col;
        if (s.U) {
            store_u<NC>(s.U + ccol * (size_t) s.Nn * NC + (size_t) node * NC, u);
        } else if (s.jcU) {
            /* rows of this node in the sorted CSC column */
            int lo = s.jcU[ccol], hi = s.jcU[ccol + 1];
            const int row0 = node * NC;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (s.irU[mid] < row0)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            for (int k = lo; k < s.jcU[ccol + 1] && s.irU[k] < row0 + NC; k++) {
                const int c = s.irU[k] - row0;
                int val = u[0];
#pragma unroll
                for (int q = 1; q < NC; q++)
                    if (c == q)
                        val = u[q];
                s.prU[k] = (double) val;
            }
        }
        if (ND > 0) {
            if (s.V) {
                double *dst = s.V + ccol * (size_t) s.Nn * ND + (size_t) node * ND;
#pragma unroll
                for (int d = 0; d < ND; d++)
                    dst[d] = vnew[d];
            } else if (s.jcV) {
                int lo = s.jcV[ccol], hi = s.jcV[ccol + 1];
                const int row0 = node * ND;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (s.irV[mid] < row0)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                for (int k = lo; k < s.jcV[ccol + 1] && s.irV[k] < row0 + ND; k++)
                    s.prV[k] = vnew[s.irV[k] - row0];
            }
        }
    }
}

template <class M>
__device__ __forceinline__ void load_model_smem(const DevState &s, int *sS, uint32_t *sG)
{
    for (int i = threadIdx.x; i < M::NT * M::NC; i += blockDim.x)
        sS[i] = s.S[i];
    for (int i = threadIdx.x; i < M::NT; i += blockDim.x)
        sG[i] = s.Gmask[i];
    __syncthreads();
}

/* The tables of -log(u) in shared memory, for kernels whose every step
 * looks them up: a kernel starts with a cold L1, and two of the lookups
 * depend on one another.  Followed by a barrier of the caller's. */
__device__ __forceinline__ void load_nl_smem(si_nl_tables &nl)
{
    static_assert(sizeof(si_nl_tables) % sizeof(uint4) == 0, "copied 16 bytes at a time");
    const uint4 *from = reinterpret_cast<const uint4 *>(&si_nl_dev);
    uint4 *to = reinterpret_cast<uint4 *>(&nl);
    for (unsigned i = threadIdx.x; i < sizeof(si_nl_tables) / sizeof(uint4); i += blockDim.x)
        to[i] = from[i];
}

/* The start of every kernel of a day, in every thread: a chained kernel is
 * launched before its predecessor has ended, reads what no kernel writes
 * (tables, event records) and waits here until the predecessor's writes are
 * there; then the next kernel may be launched.  A day is three to a dozen
 * launches: SEIR, 100,000 nodes x 180 days 21.9 -> 20.7 ms, SISe3, 1,600 x 730
 * days 24.6 -> 23.6. */
__device__ __forceinline__ void day_begin()
{
    asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

/* ------------------------------------------------------------------ */
/* Kernels.                                                              */
/* ------------------------------------------------------------------ */

/* List g as heavy for `day` when its rate sum promises many transitions
 * in one unit of time (only for models whose rates ignore t). */
/* The heavy class of a node whose rate sum at the start of a day is
 * `sum`: 0 for sum >= 16 h, 1 for >= 4 h, 2 for >= h (h = heavy_rate),
 * -1 for a node that is not heavy or a model whose rates depend on time. */
template <class M>
__device__ __forceinline__ int heavy_class(const DevState &s, double sum)
{
    const uint64_t h = si_double_bits(s.heavy_rate), x = si_double_bits(sum);
    /* positive finite doubles compare as their bits, and 4 h and 16 h are h
     * with 2 and 4 added to its exponent: no FP64 instruction, of which two
     * a warp took 7 of k_pts_store's 60 us at 10^6 nodes */
    if (!M::RATES_TIME_INVARIANT || !(s.heavy_rate > 0.0) || !si_finite_pos(sum) || x < h)
        return -1;
    return x >= h + (4ull << 52) ? 0 : x >= h + (2ull << 52) ? 1 : 2;
}

/* Block-wide (every thread calls it): nodes with a class >= 0 join that
 * class's heavy list of `day`, up to two nodes a thread.  Places within the
 * block are taken in shared memory; one thread a class then takes the
 * block's places in the list, the three side by side (class after class and
 * warp by warp, six pushes of two round trips to L2 each, k_pts_store took
 * 14.3 us a day at 10,000 nodes, and now takes 10.5).  A list that is full
 * takes nothing more. */
__device__ __forceinline__ void push_heavy(const DevState &s, long long g1, int cls1, long long g2,
                                           int cls2, int day)
{
    __shared__ int count[HEAVY_CLASSES], base[HEAVY_CLASSES];
    if (threadIdx.x < HEAVY_CLASSES)
        count[threadIdx.x] = 0;
    __syncthreads();
    const int at1 = cls1 >= 0 ? atomicAdd(&count[cls1], 1) : 0;
    const int at2 = cls2 >= 0 ? atomicAdd(&count[cls2], 1) : 0;
    __syncthreads();
    const int q = (day & 1) * HEAVY_CLASSES;
    if (threadIdx.x < HEAVY_CLASSES && count[threadIdx.x] > 0)
        base[threadIdx.x] = atomicAdd(&s.heavy_count[q + threadIdx.x], count[threadIdx.x]);
    __syncthreads();
    if (cls1 >= 0 && base[cls1] + at1 < MAX_HEAVY) {
        s.heavy_list[(q + cls1) * MAX_HEAVY + base[cls1] + at1] = (int) g1;
        s.heavy_mark[g1] = day + 1;
    }
    if (cls2 >= 0 && base[cls2] + at2 < MAX_HEAVY) {
        s.heavy_list[(q + cls2) * MAX_HEAVY + base[cls2] + at2] = (int) g2;
        s.heavy_mark[g2] = day + 1;
    }
}

/* k_init for one (replicate, node); returns its heavy class on day 0. */
template <class M>
__device__ __forceinline__ int init_node(const DevState &s, long long g, double tt0)
{
    constexpr int NC = M::NC, NT = M::NT, ND = M::ND;
    if (s.pf_days)
        tt0 = s.pf_days[(size_t) *s.pf_interval * s.pf_days_stride].tt;
    const int node = node_of(s, g);
    int u[NC];
    load_u<NC>(s.u + g * NC, u);
    const double *v = s.vA + g * ND;
    const double *ld = s.ldata + (size_t) node * s.Nld;
    si_recip dc = si_recip_none();
    double sum = 0.0;
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const double rate = M::rate(j, u, v, ld, gdata_of(s, g), tt0, dc);
        s.t_rate[(size_t) j * s.Ntot + g] = rate;
        sum += rate;
        if (!isfinite(rate) || rate < 0.0)
            record_error(s, ERR_INVALID_RATE, PHASE_INIT, 0, g, j, -1, tt0, rate);
    }
    s.sum_rate[g] = sum;
    s.t_time[g] = tt0;
    s.ctr[g] = 0;
    if (s.crn_ctr)
        s.crn_ctr[g] = 0;
    s.update[g] = 0;
    return heavy_class<M>(s, sum);
}

template <class M>
__global__ void k_init(DevState s, double tt0)
{
    const long long g = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    int cls = -1;
    if (g < s.Ntot)
        cls = init_node<M>(s, g, tt0);
    push_heavy(s, g, cls, 0, -1, 0);
}

/* The end of a node's day: its E1 events (or its SSA error) and the state
 * written back. */
template <class M>
__device__ __forceinline__ void node_finish(const DevState &s, SsaLane<M> &ln, si_rng &r,
                                            long long g, int2 at, int day, double tt,
                                            unsigned long long &fired)
{
    constexpr int NC = M::NC, NT = M::NT;
    if (s.crn_ctr) {
        /* common random numbers: the day's SSA draws came from the SSA's
         * own stream; the events draw from the node's */
        s.crn_ctr[g] = ln.c;
        r.s1 &= ~SI_CRN_S1;
        r.ctr = s.ctr[g];
    } else {
        r.ctr = ln.c;
    }
    r.have = 0;
    fired += ln.fired;
    if (s.day_max && ln.fired > *(volatile unsigned *) (s.day_max + day))
        atomicMax(s.day_max + day, ln.fired);       /* profiling: the day's busiest node */
    if (ln.err) {
        record_error(s, ln.err, PHASE_SSA, day, g, ln.err_tr, -1, ln.err_t, ln.err_rate);
    } else {
        int e_code = 0, e_idx = -1;
        if (node_e1<NC>(s, ln.u, at, node_of(s, g), day, r, e_code, e_idx)) {
            s.update[g] = 1;
            s.e1_next[g] = at;
        }
        if (e_code)
            record_error(s, e_code, PHASE_E1, day, g, -1, e_idx, tt, 0);
    }
    store_u<NC>(s.u + g * NC, ln.u);
#pragma unroll
    for (int k = 0; k < NT; k++)
        s.t_rate[(size_t) k * s.Ntot + g] = ln.rate[k];
    s.sum_rate[g] = ln.sum;
    s.t_time[g] = ln.t;
    s.ctr[g] = r.ctr;
}

/* Node g's state at the start of its day and the key of its SSA stream. */
template <class M>
__device__ __forceinline__ void load_node(const DevState &s, long long g, SsaLane<M> &ln,
                                          si_rng &r)
{
    constexpr int NC = M::NC, NT = M::NT;
    load_u<NC>(s.u + g * NC, ln.u);
#pragma unroll
    for (int k = 0; k < NT; k++)
        ln.rate[k] = s.t_rate[(size_t) k * s.Ntot + g];
    ln.sum = s.sum_rate[g];
    ln.t = s.t_time[g];
    ln.err = 0;
    ln.err_tr = -1;
    ln.err_t = 0.0;
    ln.err_rate = 0.0;
    ln.dc = si_recip_none();
    uint64_t seed, sid;
    stream_key(s, g, seed, sid);
    si_rng_init(&r, seed, sid, 0);
    if (s.crn_ctr)
        r.s1 |= SI_CRN_S1;              /* the SSA's own stream */
}

/* The first pass of a two-pass day, one ordinary node (not in the day's
 * heavy lists) per thread: a node whose day has no transition -- rate sum
 * 0, or a first waiting time that passes the end of the day -- finishes
 * here (its E1 events, state written back), with the warp's lanes in step;
 * a node with a transition is listed in s.active for k_ssa_e1, which draws
 * the same first waiting time again (same draw index) and steps it.  The
 * draws and comparisons are those of ssa_begin and ssa_step. */
template <class M>
__global__ void __launch_bounds__(256) k_quick(DevState s, int day, double tt, double next)
{
    constexpr int NC = M::NC;
    const long long g = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    bool listed = false;
    const float left = trunc_to_float(next - tt);
    const float ulps = 1e-15f * fabsf((float) next);    /* of a time's rounding */
    day_begin();
    if (g < s.Ntot && load_flag(s.err_day) >= day && s.heavy_mark[g] != day + 1 &&
        !job_over(s, g, day)) {
        const double sum = s.sum_rate[g], t = s.t_time[g];
        uint64_t c = s.crn_ctr ? s.crn_ctr[g] : s.ctr[g];
        si_rng r;
        {
            uint64_t seed, sid;
            stream_key(s, g, seed, sid);
            si_rng_init(&r, seed, sid, 0);
            if (s.crn_ctr)
                r.s1 |= SI_CRN_S1;      /* the SSA's own stream */
        }
        int err = 0;
        if (!si_finite_pos(sum)) {
            /* nothing fires (src/solvers/SimInf_solver_ssm.c:148-151) */
            if (!le_zero(si_double_bits(sum)))
                err = ERR_INVALID_RATE;
        } else {
            uint32_t p0, p1, p2, p3;
            philox_block(r, c >> 2, p0, p1, p2, p3);
            const uint32_t w = word_of(p0, p1, p2, p3, (uint32_t) c & 3u);
            /* -log(u) against the rate sum times the day's rest in single
             * precision; where that is within its error, or the times'
             * rounding, of a tie (a few in 10^5), the quotient in double
             * precision as the SSA forms it */
            const float L = -__logf(((float) w + 0.5f) * 2.3283064365386963e-10f);
            const float fsum = trunc_to_float(sum);
            const float x = fsum * (t == tt ? left : trunc_to_float(next - t));
            const float slack = 1e-5f * (L + x) + 1e-5f + fsum * ulps;
            if (L > x + slack)
                c += 1;                         /* the waiting time's draw was used */
            else if (L < x - slack)
                listed = true;
            else if (si_dge_num(si_div(si_neglog_u32(w), sum) + t, next))
                c += 1;
            else
                listed = true;
        }
        if (!listed) {
            if (s.crn_ctr) {
                /* the SSA stream's counter is done for the day; c becomes
                 * the node stream's, which the events draw from */
                s.crn_ctr[g] = c;
                c = s.ctr[g];
                r.s1 &= ~SI_CRN_S1;
            }
            if (err) {
                record_error(s, err, PHASE_SSA, day, g, -1, -1, t, sum);
            } else {
                int2 at = s.e1_next[g];
                if (at.y == day) {
                    int u[NC];
                    load_u<NC>(s.u + g * NC, u);
                    r.ctr = c;
                    r.have = 0;
                    int e_code = 0, e_idx = -1;
                    node_e1<NC>(s, u, at, node_of(s, g), day, r, e_code, e_idx);
                    s.update[g] = 1;
                    s.e1_next[g] = at;
                    store_u<NC>(s.u + g * NC, u);
                    if (e_code)
                        record_error(s, e_code, PHASE_E1, day, g, -1, e_idx, tt, 0);
                    c = r.ctr;
                }
            }
            s.t_time[g] = next;
            s.ctr[g] = c;
        }
    }
    /* list the nodes with a transition, one atomic per warp */
    const unsigned FULL = 0xFFFFFFFFu;
    const unsigned m = __ballot_sync(FULL, listed);
    if (m) {
        const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
        unsigned long long base = 0;
        if (lane == leader)
            base = atomicAdd(&s.queue_next[4 + (day & 1)], (unsigned long long) __popc(m));
        base = __shfl_sync(FULL, base, leader);
        if (listed)
            s.active[base + __popc(m & ((1u << lane) - 1u))] = (int) g;
    }
}

/* One day of SSA and E1 events for every (replicate, node): a persistent
 * grid whose warps take nodes from the day's work queue.  The queue has two
 * parts: the heavy nodes (rate sum >= heavy_rate at the start of the day,
 * heaviest class first) and then every other node in index order.  The day
 * lasts as long as its longest chain, so heavy nodes go out first, and a
 * group of lanes steps each of them (ssa_day_group): 32 lanes a node of the
 * first class, 16 of the second, 8 of the third.  A model whose rates may
 * not be evaluated at guessed states runs them 32 to a warp, one a lane,
 * and a warp that holds one takes nothing more until they are all done.
 * Ordinary nodes go out lane by lane: a thread whose node's day is over
 * takes the next entry at once, so the lanes of a warp keep stepping
 * transitions instead of waiting for the warp's busiest node.
 * Bound: the busiest node's chain, then issue slots and the FP64 pipe.
 * SEIR of 10^6 nodes, 240 days (256,149 steps of the busiest nodes): 501 ms
 * one lane a node, 85.8 with groups and serial sums, 42.1 with the sums as
 * prefix sums of whole numbers; 10,000 nodes x 365 days 136, 22.0, 13.0. */
template <class M, int MINB>
__global__ void __launch_bounds__(SSA_BLOCK, MINB) k_ssa_e1(DevState s, int day, double tt,
                                                         double next)
{
    constexpr int NC = M::NC, NT = M::NT, ND = M::ND;
    __shared__ int sS[NT * NC];
    __shared__ uint32_t sG[NT];
    __shared__ __align__(16) si_nl_tables nl;
    const int par = day & 1, npar = (day + 1) & 1;
    load_nl_smem(nl);
    load_model_smem<M>(s, sS, sG);
    day_begin();
    /* the loads that everything waits for, all in flight at once */
    const int err_day = load_flag(s.err_day);
    int n[HEAVY_CLASSES];
#pragma unroll
    for (int c = 0; c < HEAVY_CLASSES; c++)
        n[c] = s.heavy_count[par * HEAVY_CLASSES + c];
    /* the ordinary part: every node in index order, or on two-pass days
     * the nodes k_quick listed */
    const unsigned long long Ntot = s.two_pass ? s.queue_next[4 + par]
                                               : (unsigned long long) s.Ntot;
    if (blockIdx.x == 0 && threadIdx.x < HEAVY_CLASSES)
        s.heavy_count[npar * HEAVY_CLASSES + threadIdx.x] = 0;  /* filled by this day's pts */
    if (blockIdx.x == 0 && threadIdx.x < 2)
        s.queue_next[npar * 2 + threadIdx.x] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 2)
        s.queue_next[4 + npar] = 0;                     /* filled by the next k_quick */
    unsigned long long fired = 0;
    if (err_day < day) {
        add_fired(s, fired);
        return;
    }
    unsigned long long H = 0;
#pragma unroll
    for (int c = 0; c < HEAVY_CLASSES; c++) {
        n[c] = min(n[c], (int) MAX_HEAVY);
        H += (unsigned long long) n[c];
    }
    const int lane = threadIdx.x & 31;
    const unsigned FULL = 0xFFFFFFFFu;
    /* each warp's first heavy entry is its own number, so that only later
     * ones cost an atomic's round trip */
    const unsigned nwarp = gridDim.x * (SSA_BLOCK / 32);
    const unsigned warp = blockIdx.x * (SSA_BLOCK / 32) + threadIdx.x / 32;

    SsaLane<M> ln;
    si_rng r;
    long long g = -1;
    int2 e1 = make_int2(0, NO_E1);      /* the node's place in its E1 events */
    bool alive = true, need = true, done = false, heavy = false;
    bool heavy_left = H > 0;         /* warp-uniform: the heavy part may have entries */
    const double *v = nullptr, *ld = nullptr, *gd = nullptr;
    if constexpr (model_rates_total<M>::value) {
        /* the heavy part: an entry is one node of the first class for the
         * whole warp, two of the second for 16 lanes each, or four of the
         * third for 8 */
        const unsigned end0 = n[0], end1 = end0 + (n[1] + 1) / 2, items = end1 + (n[2] + 3) / 4;
        unsigned at = warp;
        while (at < items) {
            const int c = at < end0 ? 0 : at < end1 ? 1 : 2;
            const int idx = ((int) (at - (c == 0 ? 0 : c == 1 ? end0 : end1)) << c) +
                            (lane >> (5 - c));
            bool live = idx < n[c];
            g = s.heavy_list[(par * HEAVY_CLASSES + c) * MAX_HEAVY + (live ? idx : 0)];
            live = live && !job_over(s, g, day);
            load_node<M>(s, g, ln, r);
            ln.c = s.crn_ctr ? s.crn_ctr[g] : s.ctr[g];
            e1 = s.e1_next[g];
            ssa_day_group<M>(ln, r, 32 >> c, live, next, s.vA + g * ND,
                             s.ldata + (size_t) node_of(s, g) * s.Nld, gdata_of(s, g), sS, sG,
                             s.max_fired, &nl);
            if (live && (lane & ((32 >> c) - 1)) == 0)
                node_finish<M>(s, ln, r, g, e1, day, tt, fired);
            __syncwarp();
            if (nwarp >= items)
                break;
            if (lane == 0)
                at = nwarp + (unsigned) atomicAdd(&s.queue_next[par * 2], 1ull);
            at = __shfl_sync(FULL, at, 0);
        }
        heavy_left = false;
    }
    /* lanes of a warp that take ordinary nodes: a day of few nodes is spread
     * over all warps of the grid, so that a warp steps fewer chains whose
     * branches exclude one another */
    const unsigned lanes =
        s.two_pass ? 32u : (unsigned) min(32ull, (Ntot + nwarp - 1) / nwarp);
    alive = lane < (int) max(lanes, 1u) || heavy_left;
    for (;;) {
        /* hand queue entries to the lanes without a node; while the
         * heaviest class lasts, only the first heavy_lanes lanes take them */
        unsigned want = __ballot_sync(FULL, alive && need);
        const bool holds_heavy = __any_sync(FULL, alive && !need && heavy);
        const bool from_heavy = heavy_left;
        if (from_heavy && s.heavy_lanes > 0 && s.heavy_lanes < 32 && want && !holds_heavy) {
            unsigned long long at = 0;
            if (lane == 0)
                at = *(volatile const unsigned long long *) &s.queue_next[par * 2];
            at = __shfl_sync(FULL, at, 0);
            if (at < (unsigned long long) n[0])
                want &= (1u << s.heavy_lanes) - 1u;
        }
        if (want && !holds_heavy) {
            const int leader = __ffs(want) - 1;
            unsigned long long base = 0;
            if (lane == leader)
                base = atomicAdd(&s.queue_next[par * 2 + (from_heavy ? 0 : 1)],
                                 (unsigned long long) __popc(want));
            base = __shfl_sync(FULL, base, leader);
            long long cand = -1;
            bool empty = false;
            if ((want >> lane) & 1u) {
                const unsigned long long pos = base + __popc(want & ((1u << lane) - 1u));
                if (from_heavy) {
                    if (pos < H) {
                        int idx = (int) pos, c = 0;
                        while (c < HEAVY_CLASSES - 1 && idx >= n[c]) {
                            idx -= n[c];
                            c++;
                        }
                        cand = s.heavy_list[(par * HEAVY_CLASSES + c) * MAX_HEAVY + idx];
                    } else {
                        empty = true;
                    }
                } else if (pos >= Ntot) {
                    alive = false;
                } else if (s.two_pass) {
                    cand = s.active[pos];
                } else if (s.heavy_mark[pos] != day + 1) {
                    cand = (long long) pos;     /* heavy ones come from the heavy part */
                }
                if (cand >= 0 && job_over(s, cand, day))
                    cand = -1;                  /* its model has run all its days */
            }
            if (from_heavy && __any_sync(FULL, empty))
                heavy_left = false;
            if (cand >= 0) {
                g = cand;
                heavy = from_heavy;
                load_node<M>(s, g, ln, r);
                v = s.vA + g * ND;
                ld = s.ldata + (size_t) node_of(s, g) * s.Nld;
                gd = gdata_of(s, g);
                e1 = s.e1_next[g];
                done = ssa_begin<M>(ln, r, s.crn_ctr ? s.crn_ctr[g] : s.ctr[g], next, &nl);
                need = false;
            }
        }
        if (!__any_sync(FULL, alive))
            break;
        if (alive && !need) {
            if (done) {
                node_finish<M>(s, ln, r, g, e1, day, tt, fired);
                need = true;
                heavy = false;
            } else {
                /* one step; a heavy warp has nothing else to do and runs
                 * its whole day, in batches of four steps where the rates
                 * do not read t */
                if constexpr (M::RATES_TIME_INVARIANT) {
                    if (heavy) {
                        ssa_run_day<M>(ln, r, next, v, ld, gd, sS, sG, s.max_fired, &nl);
                        done = true;
                    } else {
                        done = ssa_step<M>(ln, r, next, v, ld, gd, sS, sG, s.max_fired, &nl);
                    }
                } else {
                    do
                        done = ssa_step<M>(ln, r, next, v, ld, gd, sS, sG, s.max_fired, &nl);
                    while (heavy && !done);
                }
            }
        }
    }
    add_fired(s, fired);
}

/* One external transfer of one replicate (src/solvers/SimInf_solver.c:
 * 824-902): sample from the source, add to the destination (atomics: adds
 * into one destination commute within a wavefront), subtract from the
 * source (exclusive to this event within its wavefront).  Any transfer,
 * behind e2_apply, which handles the common ones; inlined, as a call costs
 * the waves of both kinds (SISe3, 10,000 nodes x 60 days of proportions 4.95 ms
 * of waves called, 4.18 inlined; SEIR, 20,000 nodes x 120 days of counts 3.58,
 * 3.29). */
template <class M>
__device__ __forceinline__ void e2_apply_any(const DevState &s, const E2Rec &e, int rep, int day,
                                          double tt)
{
    constexpr int NC = M::NC;
    const long long gs = (long long) rep * s.Nn + e.src;
    const long long gd = (long long) rep * s.Nn + e.dst;
    int uu[NC], ind[NC];
    for (int c = 0; c < NC; c++)
        uu[c] = __ldcg(s.u + gs * NC + c);
    si_rng r;
    {
        uint64_t seed, sid;
        stream_key(s, gs, seed, sid);
        si_rng_init(&r, seed, sid, __ldcg((const unsigned long long *) s.ctr + gs));
    }
    int err = sample_select<NC>(s, uu, e.select, e.n, e.proportion, ind, &r);
    s.ctr[gs] = r.ctr;
    if (err) {
        record_error(s, err, PHASE_E2, day, gs, -1, e.index, tt, 0);
        return;
    }
    for (int k = s.jcE[e.select]; k < s.jcE[e.select + 1]; k++) {
        const int jj = s.irE[k];
        int dj = jj;
        if (e.shift >= 0) {
            if (!s.hasN) {
                record_error(s, ERR_EVENTS_N, PHASE_E2, day, gs, -1, e.index, tt, 0);
                return;
            }
            const int ll = s.Nshift[e.shift * NC + jj];
            if (jj + ll < 0 || jj + ll >= NC) {
                record_error(s, ERR_SHIFT_OUT_OF_BOUNDS, PHASE_E2, day, gs, -1, e.index, tt, 0);
                return;
            }
            dj = jj + ll;
        }
        if (ind[jj]) {
            const int old = atomicAdd(&s.u[gd * NC + dj], ind[jj]);
            if (old + ind[jj] < 0) {
                record_error(s, ERR_NEGATIVE_STATE, PHASE_E2, day, gs, -1, e.index, tt, 0);
                return;
            }
            /* The source is exclusive to this event within the wave; a
             * self-transfer reads back its own atomic add. */
            const int nv = __ldcg(s.u + gs * NC + jj) - ind[jj];
            s.u[gs * NC + jj] = nv;
            if (nv < 0) {
                record_error(s, ERR_NEGATIVE_STATE, PHASE_E2, day, gs, -1, e.index, tt, 0);
                return;
            }
        }
    }
    s.update[gd] = 1;
    s.update[gs] = 1;
}

/* Words of a node's stream held ready for a transfer's draws: the Philox
 * blocks ctr >> 2 and the two after it, which every lane of a warp computes
 * in step (drawn one block at a time when a lane runs out, some lane would
 * be at a block's end at nearly every draw, and the warp would wait for a
 * Philox block a draw).  A thread's words lie a block of threads apart in
 * shared memory, one bank a lane. */
enum { E2_WORDS = 12 };

/* The words of blocks b, b + 1 and b + 2 of the stream in r. */
__device__ __forceinline__ void e2_words(uint32_t *words, const si_rng &r, uint64_t b)
{
#pragma unroll
    for (int j = 0; j < E2_WORDS / 4; j++) {
        uint32_t w0, w1, w2, w3;
        philox_block(r, b + j, w0, w1, w2, w3);
        words[(4 * j) * blockDim.x] = w0;
        words[(4 * j + 1) * blockDim.x] = w1;
        words[(4 * j + 2) * blockDim.x] = w2;
        words[(4 * j + 3) * blockDim.x] = w3;
    }
}

/* The next words of a long sample, out of line. */
static __device__ __noinline__ void e2_more_words(uint32_t *words, uint32_t k0, uint32_t k1,
                                                  uint32_t s0, uint32_t s1, uint64_t b)
{
    si_rng r;
    r.k0 = k0;
    r.k1 = k1;
    r.s0 = s0;
    r.s1 = s1;
    e2_words(words, r, b);
}

/* The transfer of record e: a size given as a count, sampled from a plain
 * column and moved unshifted to another node, runs here with the node's
 * compartments in registers; everything else in e2_apply_any, with the same
 * draws.  `words` is the thread's share of shared memory.  Bound: a wave's
 * chain of dependent loads (record, state, then the atomics) and draws, and
 * in waves that fill the chip instruction issue. */
template <class M>
__device__ __forceinline__ void e2_apply(const DevState &s, const E2Rec &e, int rep, int day,
                                         double tt, uint32_t *words)
{
    constexpr int NC = M::NC;
    const long long gs = (long long) rep * s.Nn + e.src;
    const long long gd = (long long) rep * s.Nn + e.dst;
    int uu[NC], ind[NC];
    load_u_l2<NC>(s.u + gs * NC, uu);
    si_rng r;
    {
        uint64_t seed, sid;
        stream_key(s, gs, seed, sid);
        si_rng_init(&r, seed, sid, __ldcg((const unsigned long long *) s.ctr + gs));
    }
    const uint32_t col = s.ecol[e.select];
    if (!(col & ECOL_PLAIN) || e.n <= 0 || e.shift >= 0 || e.src == e.dst) {
        e2_apply_any<M>(s, e, rep, day, tt);
        return;
    }
    const unsigned cols = col & ~ECOL_PLAIN;
    int total = 0, kinds = 0;
#pragma unroll
    for (int c = 0; c < NC; c++) {
        const bool in = (cols >> c) & 1u;
        total += in ? uu[c] : 0;
        kinds += in && uu[c] > 0;
        ind[c] = 0;
    }
    int n = e.n;
    if (s.cap && n > total)
        n = total;
    if (cols == 0 || n > total || n < 0) {
        record_error(s, ERR_SAMPLE_SELECT, PHASE_E2, day, gs, -1, e.index, tt, 0);
        return;
    }
    if (n > 0) {
        if (n == total || kinds == 1) {
            /* everyone, or n of the one kind there is */
#pragma unroll
            for (int c = 0; c < NC; c++)
                if (((cols >> c) & 1u) && uu[c] > 0)
                    ind[c] = n == total ? uu[c] : n;
        } else {
            uint64_t blk = r.ctr >> 2;
            e2_words(words, r, blk);
            /* sequential multivariate hypergeometric (SimInf_solver.c:
             * 139-160); the urn of each compartment is si_hypergeometric's */
            unsigned at = (unsigned) r.ctr & 3u;        /* the next draw's word */
            int left = total, want = n;
#pragma unroll
            for (int c = 0; c < NC; c++) {
                if (!((cols >> c) & 1u))
                    continue;
                const int nk = uu[c];
                if (cols >> c == 1u) {
                    ind[c] = want;                      /* the last compartment */
                } else if (nk > 0 && want > 0) {
                    const bool complement = (unsigned) want > (unsigned) (left - want);
                    const int t = complement ? left - want : want;
                    unsigned a = (unsigned) nk, rem = (unsigned) left;
                    int i = 0, k = 0;
                    while (i < t && a > 0 && a < rem) {
                        if (at == E2_WORDS) {
                            blk += E2_WORDS / 4;
                            e2_more_words(words, r.k0, r.k1, r.s0, r.s1, blk);
                            at = 0;
                        }
                        /* (2 w + 1) rem < a 2^33, in whole numbers */
                        const uint64_t w = words[at * blockDim.x];
                        const unsigned take = (uint32_t) (((2 * w + 1) * rem) >> 33) < a;
                        k += (int) take;
                        a -= take;
                        rem--;
                        at++;
                        i++;
                    }
                    if (a > 0 && a == rem)
                        k += t - i;
                    k = complement ? nk - k : k;
                    ind[c] = k;
                    want -= k;
                }
                left -= nk;
            }
            s.ctr[gs] = (blk << 2) + at;
        }
        bool neg = false;
#pragma unroll
        for (int c = 0; c < NC; c++) {
            if (ind[c])
                neg |= atomicAdd(&s.u[gd * NC + c], ind[c]) + ind[c] < 0;
            uu[c] -= ind[c];
        }
        store_u<NC>(s.u + gs * NC, uu);
        if (neg) {
            record_error(s, ERR_NEGATIVE_STATE, PHASE_E2, day, gs, -1, e.index, tt, 0);
            return;
        }
    }
    s.update[gd] = 1;
    s.update[gs] = 1;
}

template <class M>
__global__ void __launch_bounds__(512, 1) k_e2_wave(DevState s, const E2Rec *ev, int count, int day,
                                                 double tt)
{
    const long long i = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    __shared__ uint32_t words[E2_WORDS * 512];
    const bool mine = i < (long long) count * s.Nrep;
    const int rep = s.Nrep == 1 ? 0 : (int) (i / count);
    E2Rec e;
    if (mine)
        e = ev[i - (long long) rep * count];
    day_begin();
    if (!mine || load_flag(s.err_day) < day || load_flag(s.err_day_pre_e2) <= day)
        return;
    e2_apply<M>(s, e, rep, day, tt, words + threadIdx.x);
}

/* Every thread of the cluster has done its writes before any goes on, and
 * sees them (release and acquire at cluster scope are the default). */
__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory");
}

/* A day's last wavefronts in one launch, in order: the first `wide` of them
 * by a cluster of E2_CLUSTER blocks with a cluster barrier between two, the
 * smaller ones after them by the cluster's first block, where a block
 * barrier is enough.  State is read from L2, where the other blocks' writes
 * and the atomics are.  A wave on one SM is bound by that SM's issue slots
 * from about 500 transfers on, which is where the second part begins; a
 * wave that fills the cluster more than twice is better off on the whole
 * chip.  With e2_apply's common path and draws in step, a day's transfers of
 * SEIR, 10,000 nodes (9.7 waves): 79 us in three launches with a tail of one
 * block, 44 in one launch; 10^6 nodes (15 waves): 187 us, then 130.  Waves of
 * transfers off that path come here in a block's size only
 * (launch_day_waves). */
template <class M>
__global__ void __launch_bounds__(E2_TAIL_BLOCK, 1) k_e2_tail(DevState s, const E2Rec *ev,
                                                           E2Tail tail, int day, double tt)
{
    __shared__ uint32_t words[E2_WORDS * E2_TAIL_BLOCK];
    const long long me = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    E2Rec e;
    if (me < tail.count[0] * (long long) s.Nrep)
        e = ev[tail.off[0] + (s.Nrep == 1 ? me : me % tail.count[0])];
    day_begin();
    if (load_flag(s.err_day) < day || load_flag(s.err_day_pre_e2) <= day)
        return;                                     /* the same for every thread */
    for (int w = 0; w < tail.n; w++) {
        const bool wide = w < tail.wide;
        if (!wide && blockIdx.x > 0)
            return;
        const int count = tail.count[w];
        const E2Rec *wev = ev + tail.off[w];
        const long long items = (long long) count * s.Nrep;
        const long long step = wide ? (long long) gridDim.x * blockDim.x : blockDim.x;
        for (long long i = me; i < items; i += step) {
            const int rep = s.Nrep == 1 ? 0 : (int) (i / count);
            if (i != me)
                e = wev[i - (long long) rep * count];
            e2_apply<M>(s, e, rep, day, tt, words + threadIdx.x);
        }
        /* the thread's first record of the next wave, before the wait */
        if (w + 1 < tail.n) {
            const int nc = tail.count[w + 1];
            if (me < nc * (long long) s.Nrep)
                e = ev[tail.off[w + 1] + (s.Nrep == 1 ? me : me % nc)];
        }
        if (wide)
            cluster_barrier();
        else
            __syncthreads();
    }
}

/* Batches: node g's share of its job's prevalence sums at columns c0 ..
 * c1 - 1 (integer sums, so the order of the additions does not matter).  The
 * lanes here that share a job add up first: a model of 50,000 nodes would
 * send 100,000 atomics a day to two words. */
template <int NC>
__device__ __forceinline__ void add_prevalence(const DevState &s, long long g, const int (&u)[NC],
                                               int c0, int c1)
{
    const int j = s.job_of[g];
    unsigned long long num = 0, den = 0;
#pragma unroll
    for (int c = 0; c < NC; c++) {
        const unsigned long long x = (unsigned long long) (long long) u[c];
        if (s.prev_num_mask & (1u << c))
            num += x;
        if (s.prev_den_mask & (1u << c))
            den += x;
    }
    const unsigned here = __activemask();
    const unsigned mates = __match_any_sync(here, j);
    bool first = true;
    if (!__any_sync(mates, (num | den) >> 32)) {
        /* 32 halves of 16 bits add up within 32 bits */
        const unsigned n0 = __reduce_add_sync(mates, (unsigned) num & 0xFFFFu),
                       n1 = __reduce_add_sync(mates, (unsigned) num >> 16),
                       d0 = __reduce_add_sync(mates, (unsigned) den & 0xFFFFu),
                       d1 = __reduce_add_sync(mates, (unsigned) den >> 16);
        num = n0 + ((unsigned long long) n1 << 16);
        den = d0 + ((unsigned long long) d1 << 16);
        first = (threadIdx.x & 31) == __ffs((int) mates) - 1;
    }
    const int tl = s.job_tlen[j];
    for (int col = c0; first && col < c1 && col < tl; col++) {
        unsigned long long *p = s.prev + 2 * (s.job_col0[j] + col);
        atomicAdd(p, num);
        atomicAdd(p + 1, den);
    }
}

enum { NEEDS_REFRESH = -2 };

/* k_pts_store for one (replicate, node): post-time-step function, U/V
 * columns, prevalence.  Returns NEEDS_REFRESH when its rates must be
 * recomputed (an event touched it, or the post-time-step function changed
 * v), else its heavy class on the next day. */
template <class M>
__device__ __forceinline__ int pts_node(const DevState &s, long long g, int day, double tt,
                                        int c0, int c1, const double *v_in, double *v_out)
{
    constexpr int NC = M::NC, ND = M::ND;
    const int rep = rep_of(s, g), node = node_of(s, g);
    int u[NC];
    load_u<NC>(s.u + g * NC, u);
    const double *vi = v_in + g * ND;
    double *vo = v_out + g * ND;
    const double *ld = s.ldata + (size_t) node * s.Nld;
    const double *gd = gdata_of(s, g);
    /* a post-time-step function that reads other nodes (by offsets from
     * its node, src/models/SISe_sp.c:127-134) gets the node's place in the
     * replicate's arrays; every node's external transfers are done */
    const int rc = M::PTS_LOCAL ? M::pts(vo, u, vi, ld, gd, node, tt)
                                : M::pts(vo, s.u + g * NC, vi, ld, gd, node, tt);
    store_columns<NC, ND>(s, rep, node, u, vo, c0, c1);
    if (s.prev && c1 > c0)
        add_prevalence<NC>(s, g, u, c0, c1);
    if (rc < 0)
        record_error(s, rc, PHASE_PTS, day, g, -1, -1, tt, 0);
    else if (rc > 0 || s.update[g])
        return NEEDS_REFRESH;
    return job_over(s, g, day + 1) ? -1 : heavy_class<M>(s, s.sum_rate[g]);
}

/* The rate refresh of the day's end (src/solvers/SimInf_solver_ssm.c:
 * 285-306): every rate recomputed with v_new at tt, their changes added to
 * the rate sum in transition order.  Returns the heavy class on the next
 * day. */
template <class M>
__device__ __forceinline__ int refresh_node(const DevState &s, long long g, int day, double tt,
                                            const double *v_out)
{
    constexpr int NC = M::NC, NT = M::NT, ND = M::ND;
    const int node = node_of(s, g);
    int u[NC];
    load_u<NC>(s.u + g * NC, u);
    const double *vo = v_out + g * ND;
    const double *ld = s.ldata + (size_t) node * s.Nld;
    const double *gd = gdata_of(s, g);
    si_recip dc = si_recip_none();
    double delta = 0.0;
#pragma unroll
    for (int k = 0; k < NT; k++) {
        const double old = s.t_rate[(size_t) k * s.Ntot + g];
        const double nr = M::rate(k, u, vo, ld, gd, tt, dc);
        s.t_rate[(size_t) k * s.Ntot + g] = nr;
        delta += nr - old;
        if (si_bad_rate(nr))
            record_error(s, ERR_INVALID_RATE, PHASE_PTS, day, g, k, -1, tt, nr);
    }
    s.sum_rate[g] += delta;
    s.update[g] = 0;
    return job_over(s, g, day + 1) ? -1 : heavy_class<M>(s, s.sum_rate[g]);
}

template <class M>
__global__ void __launch_bounds__(256) k_pts_store(DevState s, int day, double tt, int c0, int c1,
                                                   const double *v_in, double *v_out)
{
    /* The block's nodes whose rates need a refresh are gathered first and
     * refreshed by the block's first threads: the refresh is FP64 work,
     * and the FP64 pipe issues a warp instruction at the same cost however
     * few of its lanes are active. */
    __shared__ int listed[256];
    __shared__ int nlisted;
    if (threadIdx.x == 0)
        nlisted = 0;
    __syncthreads();
    day_begin();
    const long long g0 = blockIdx.x * (long long) blockDim.x;
    const long long g = g0 + threadIdx.x;
    int cls = -1;
    if (g < s.Ntot && load_flag(s.err_day) >= day && !job_over(s, g, day)) {
        cls = pts_node<M>(s, g, day, tt, c0, c1, v_in, v_out);
        if (cls == NEEDS_REFRESH) {
            listed[atomicAdd(&nlisted, 1)] = threadIdx.x;
            cls = -1;
        }
    }
    __syncthreads();
    long long gr = 0;
    int cls2 = -1;
    if (threadIdx.x < nlisted) {
        gr = g0 + listed[threadIdx.x];
        cls2 = refresh_node<M>(s, gr, day, tt, v_out);
    }
    push_heavy(s, g, cls, gr, cls2, day + 1);
}

/* ------------------------------------------------------------------ */
/* All-events method (src/solvers/SimInf_solver_aem.c), a lane for each  */
/* transition of a node during its day (k_aem_day), a thread a node at   */
/* its start and end.  Transition j of node g draws from its own stream, */
/* keyed (seed, AEM_SID | (g * Nt + j)); the next event is the smallest  */
/* event time, the lowest transition among equal times.                  */
/* ------------------------------------------------------------------ */
#define AEM_SID (1ULL << 63)

__device__ __forceinline__ double aem_neglog(uint64_t seed, long long g, int Nt, int j,
                                             uint64_t &ctr, const si_nl_tables *nl)
{
    si_rng r;
    si_rng_init(&r, seed, AEM_SID | ((uint64_t) g * (uint64_t) Nt + (uint64_t) j), ctr);
    const double x = si_neglog_u32_in(si_next_u32(&r), nl);
    ctr = r.ctr;
    return x;
}

/* calcTimes (src/solvers/SimInf_solver_aem.c:52-75), with its three
 * quotients -- a new waiting time -log(u) / new_rate, a sleeping time
 * inf / new_rate, a rescaling old_rate / new_rate -- formed by one division
 * (one copy of the division's code in the kernel).  Addition commutes
 * exactly, so tt + q and q + tt are the same double. */
__device__ __forceinline__ void aem_calc_times(double &time, double &inf, double tt,
                                               double old_rate, double new_rate, uint64_t seed,
                                               long long g, int Nt, int j, uint64_t &ctr,
                                               const si_nl_tables *nl)
{
    const double oldtime = time;
    int kind;                           /* 0: q + tt, 1: q * (oldtime - tt) + tt, 2: none */
    bool draw = false;
    double num = 0.0;
    if (isinf(oldtime)) {
        if (inf == 0.0) {
            draw = true;
            kind = 0;
        } else if (new_rate > 0.0) {
            num = inf;
            kind = 0;
        } else {
            kind = 2;
        }
    } else if (new_rate >= DBL_MIN) {
        if (oldtime == tt) {
            draw = true;
            kind = 0;
        } else {
            num = old_rate;
            kind = 1;
        }
    } else {
        inf = (oldtime - tt) * old_rate;
        time = si_bits_double(0x7FF0000000000000ULL);
        return;
    }
    if (kind == 2)
        return;
    if (draw)
        num = aem_neglog(seed, g, Nt, j, ctr, nl);
    const double q = si_div(num, new_rate);
    time = kind == 0 ? q + tt : (q * (oldtime - tt)) + tt;
}

/* Initial rates and event times (src/solvers/SimInf_solver_aem.c:113-158). */
template <class M>
__device__ __forceinline__ int aem_init_node(const DevState &s, long long g, double tt0);

template <class M>
__global__ void k_aem_init(DevState s, double tt0)
{
    const long long g = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    int cls = -1;
    if (g < s.Ntot)
        cls = aem_init_node<M>(s, g, tt0);
    push_heavy(s, g, cls, 0, -1, 0);
}

/* k_aem_init for one node; returns its heavy class on day 0 (from the sum
 * of its rates, for the order of the work queue only). */
template <class M>
__device__ __forceinline__ int aem_init_node(const DevState &s, long long g, double tt0)
{
    constexpr int NC = M::NC, NT = M::NT, ND = M::ND;
    const int node = node_of(s, g);
    int u[NC];
    load_u<NC>(s.u + g * NC, u);
    const double *v = s.vA + g * ND;
    const double *ld = s.ldata + (size_t) node * s.Nld;
    si_recip dc = si_recip_none();
    double sum = 0.0;
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const double rate = M::rate(j, u, v, ld, gdata_of(s, g), tt0, dc);
        const size_t k = (size_t) j * s.Ntot + g;
        s.t_rate[k] = rate;
        if (!isfinite(rate) || rate < 0.0)
            record_error(s, ERR_INVALID_RATE, PHASE_INIT, 0, g, j, -1, tt0, rate);
        uint64_t c = 0;
        double t = si_div(aem_neglog(s.seed, g, NT, j, c, SI_NL_GLOBAL), rate) + tt0;
        if (t <= 0.0)
            t = si_bits_double(0x7FF0000000000000ULL);
        s.react_time[k] = t;
        s.react_inf[k] = 0.0;
        s.react_ctr[k] = c;
        sum += rate;
    }
    s.t_time[g] = tt0;
    s.ctr[g] = 0;
    s.update[g] = 0;
    return heavy_class<M>(s, sum);
}

/* One node's state in k_aem_pts. */
template <class M>
struct AemNode {
    int u[M::NC];
    double rate[M::NT], time[M::NT], inf[M::NT];
    uint64_t ctr[M::NT];
    int err, err_tr;
    double err_t, err_rate;
};

/* Rate j refreshed at time t (rate functions) and its event time at tc
 * (calcTimes), recording an invalid rate. */
template <class M>
__device__ __forceinline__ void aem_refresh(const DevState &s, AemNode<M> &a, long long g, int j,
                                            const double *v, const double *ld, const double *gd,
                                            double t, double tc, si_recip &dc)
{
    const double old = a.rate[j];
    const double nr = M::rate(j, a.u, v, ld, gd, t, dc);
    a.rate[j] = nr;
    if (si_bad_rate(nr)) {
        a.err = ERR_INVALID_RATE;
        a.err_tr = j;
        a.err_t = t;
        a.err_rate = nr;
    }
    aem_calc_times(a.time[j], a.inf[j], tc, old, nr, s.seed, g, M::NT, j, a.ctr[j],
                   SI_NL_GLOBAL);
}

/* Lanes a node has in k_aem_day: one a transition, to a power of two. */
template <class M>
struct AemLanes {
    static constexpr int value = M::NT <= 1    ? 1
                                 : M::NT <= 2  ? 2
                                 : M::NT <= 4  ? 4
                                 : M::NT <= 8  ? 8
                                 : M::NT <= 16 ? 16
                                               : 32;
};

/* One day of every node under the all-events method, then its E1 events: a
 * persistent grid whose groups of AemLanes lanes take nodes from the
 * day's work queue, first the heavy nodes (rate sum >= heavy_rate at the
 * start of the day, listed by the previous day's end, heaviest class first),
 * then every other node in index order.  Lane j of a group holds transition
 * j's rate, event time, sleeping time and stream (src/solvers/
 * SimInf_solver_aem.c:179-307): the group finds the smallest event time (the
 * lowest transition among equal ones), every lane applies that transition
 * to its copy of u, and the transition and its dependents in G's column
 * each refresh their own rate and time, side by side: one division a step
 * where one lane did NT of them one after the other.  Bound: the busiest
 * node's chain.  SEIR, 100,000 nodes x 120 days: 50.3 ms with a lane a node,
 * 23.1 with four.
 * With WIDE, for many nodes a group (Launch::aem_day), a warp looks through
 * the ordinary part 32 nodes at a time, a lane a node: one whose event times
 * all pass the day's end, and without an E1 event, is done, and the groups
 * take the others.  Handed out a group a node, a day of 500,000 nodes without
 * an infected one took 55 us, 25 with a lane a node, and takes 20. */
template <class M, bool WIDE>
__global__ void __launch_bounds__(SSA_BLOCK, 4) k_aem_day(DevState s, int day, double tt,
                                                          double next)
{
    constexpr int NC = M::NC, NT = M::NT, ND = M::ND, G = AemLanes<M>::value;
    __shared__ int sS[NT * NC];
    __shared__ uint32_t sG[NT];
    __shared__ __align__(16) si_nl_tables nl;
    load_nl_smem(nl);
    load_model_smem<M>(s, sS, sG);
    day_begin();
    const int par = day & 1, npar = (day + 1) & 1;
    const int err_day = load_flag(s.err_day);
    int n[HEAVY_CLASSES];
    unsigned long long H = 0;
#pragma unroll
    for (int c = 0; c < HEAVY_CLASSES; c++) {
        n[c] = min(s.heavy_count[par * HEAVY_CLASSES + c], (int) MAX_HEAVY);
        H += (unsigned long long) n[c];
    }
    if (blockIdx.x == 0 && threadIdx.x < HEAVY_CLASSES)
        s.heavy_count[npar * HEAVY_CLASSES + threadIdx.x] = 0;  /* filled by this day's end */
    if (blockIdx.x == 0 && threadIdx.x < 2)
        s.queue_next[npar * 2 + threadIdx.x] = 0;
    unsigned long long fired = 0;
    if (err_day < day) {
        add_fired(s, fired);
        return;
    }
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, j = lane & (G - 1), base = lane - j;
    const unsigned group = (G == 32 ? FULL : ((1u << (G & 31)) - 1u)) << base;
    const bool own = j < NT;                /* the lane holds a transition */
    long long g = 0;
    bool alive = true, need = true;         /* the same in the whole group */
    int u[NC];
    double rate = 0.0, time = 0.0, inf = 0.0;
    uint64_t ctr = 0;
    int err = 0, err_tr = -1;
    double err_t = 0.0, err_rate = 0.0;
    unsigned nfired = 0;
    const double *v = nullptr, *ld = nullptr, *gd = nullptr;
    si_recip dc = si_recip_none();
    /* WIDE, the same in the whole warp: the heavy part and the ordinary one
     * may have entries; the lanes whose `mine` is a node to hand out */
    bool heavy_left = H > 0, more = true;
    unsigned listed = 0;
    long long mine = 0;
    for (;;) {
        /* groups without a node take the queue's next entries */
        const unsigned want = __ballot_sync(FULL, alive && need && j == 0);
        if (want) {
            const unsigned place = __popc(want & ((1u << base) - 1u));  /* the group's among them */
            long long cand = -1;
            if (!WIDE || heavy_left) {
                unsigned long long at = 0;
                if (lane == __ffs((int) want) - 1)
                    at = atomicAdd(&s.queue_next[par * 2], (unsigned long long) __popc(want));
                at = __shfl_sync(FULL, at, __ffs((int) want) - 1);
                heavy_left = at + __popc(want) < H;
                if (alive && need) {
                    const unsigned long long pos = at + place;
                    if (pos < H) {
                        int idx = (int) pos, c = 0;
                        while (c < HEAVY_CLASSES - 1 && idx >= n[c]) {
                            idx -= n[c];
                            c++;
                        }
                        cand = s.heavy_list[(par * HEAVY_CLASSES + c) * MAX_HEAVY + idx];
                    } else if (!WIDE) {
                        if (pos - H >= (unsigned long long) s.Ntot)
                            alive = false;
                        else if (H == 0 || s.heavy_mark[pos - H] != day + 1)
                            cand = (long long) (pos - H);
                    }
                }
            } else {
                while (!listed && more) {
                    unsigned long long at = 0;
                    if (lane == 0)
                        at = atomicAdd(&s.queue_next[par * 2 + 1], 32ull);
                    at = __shfl_sync(FULL, at, 0);
                    more = at + 32 < (unsigned long long) s.Ntot;
                    mine = (long long) at + lane;
                    bool take = mine < s.Ntot && (H == 0 || s.heavy_mark[mine] != day + 1);
                    if (take) {
                        double t = s.react_time[mine];
#pragma unroll
                        for (int k = 1; k < NT; k++) {
                            const double x = s.react_time[(size_t) k * s.Ntot + mine];
                            if (x < t)
                                t = x;
                        }
                        if ((isinf(t) || t >= next) && s.e1_next[mine].y != day) {
                            s.t_time[mine] = next;
                            take = false;
                        }
                    }
                    listed = __ballot_sync(FULL, take);
                }
                /* the k-th group takes the k-th node of the list */
                const unsigned from = __fns(listed, 0, (int) place + 1);
                const unsigned last = __fns(listed, 0, __popc(want));
                const long long c = __shfl_sync(FULL, mine, (int) (from & 31u));
                if (alive && need) {
                    if (from < 32)
                        cand = c;
                    else if (!more)
                        alive = false;
                }
                listed = last < 32 ? listed & ~((2u << last) - 1u) : 0u;
            }
            if (cand >= 0) {
                g = cand;
                load_u<NC>(s.u + g * NC, u);
                const size_t k = (size_t) (own ? j : 0) * s.Ntot + g;
                rate = s.t_rate[k];
                time = s.react_time[k];
                inf = s.react_inf[k];
                ctr = s.react_ctr[k];
                v = s.vA + g * ND;
                ld = s.ldata + (size_t) node_of(s, g) * s.Nld;
                gd = gdata_of(s, g);
                dc = si_recip_none();
                err = 0;
                err_tr = -1;
                err_t = err_rate = 0.0;
                nfired = 0;
                need = false;
            }
        }
        if (!__any_sync(FULL, alive))
            break;
        /* the smallest event time, the lowest transition among equal ones;
         * the comparisons are those of a scan from transition 0: a time that
         * is not a number is passed over, and in place 0 it stays */
        const uint64_t tb = si_double_bits(time);
        int64_t key = si_isnan_bits(tb) ? (j == 0 ? INT64_MIN : INT64_MAX) : si_dkey(tb);
        int tr = j;
        if (!own)
            key = INT64_MAX;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const int64_t k2 = __shfl_xor_sync(FULL, key, o);
            const int t2 = __shfl_xor_sync(FULL, tr, o);
            if (k2 < key || (k2 == key && t2 < tr)) {
                key = k2;
                tr = t2;
            }
        }
        const double t = __shfl_sync(FULL, time, base + tr);
        const bool busy = alive && !need;
        bool done = busy && (isinf(t) || t >= next);
        bool bad = false;
        double nr = 0.0;
        if (busy && !done) {
            if (++nfired > s.max_fired) {
                err = ERR_TIMEOUT;
                err_tr = tr;
                err_t = t;
                done = true;
            } else {
                int neg = 0;
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    const int x = sS[tr * NC + c];
                    u[c] += x;
                    neg |= (x != 0) & (u[c] < 0);
                }
                if (neg) {
                    err = ERR_NEGATIVE_STATE;
                    err_tr = tr;
                    err_t = t;
                    err_rate = 0.0;
                }
                if (own && (j == tr || ((sG[tr] >> j) & 1u))) {
                    const double old = rate;
#pragma unroll
                    for (int k = 0; k < NT; k++)
                        if (k == j)
                            nr = M::rate(k, u, v, ld, gd, t, dc);
                    rate = nr;
                    bad = si_bad_rate(nr);
                    aem_calc_times(time, inf, t, old, nr, s.seed, g, NT, j, ctr, &nl);
                }
            }
        }
        const unsigned bads = __ballot_sync(FULL, bad);
        if (bads) {
            /* the dependents are refreshed in order, the fired transition
             * last: the last invalid rate is the one reported */
            const unsigned mine = bads & group;
            const int at = !mine ? lane
                           : (mine >> (base + tr)) & 1u ? base + tr : 31 - __clz((int) mine);
            const double r = __shfl_sync(FULL, nr, at);
            if (mine) {
                err = ERR_INVALID_RATE;
                err_tr = at - base;
                err_t = t;
                err_rate = r;
            }
        }
        if (done) {
            /* the end of the node's day: its error, or its E1 events */
            if (j == 0) {
                if (err) {
                    record_error(s, err, PHASE_SSA, day, g, err_tr, -1, err_t, err_rate);
                } else {
                    int2 at = s.e1_next[g];
                    if (at.y == day) {
                        si_rng r;
                        uint64_t seed, sid;
                        int e_code = 0, e_idx = -1;
                        stream_key(s, g, seed, sid);
                        si_rng_init(&r, seed, sid, s.ctr[g]);
                        node_e1<NC>(s, u, at, node_of(s, g), day, r, e_code, e_idx);
                        s.update[g] = 1;
                        s.e1_next[g] = at;
                        s.ctr[g] = r.ctr;
                        if (e_code)
                            record_error(s, e_code, PHASE_E1, day, g, -1, e_idx, tt, 0);
                    }
                }
                store_u<NC>(s.u + g * NC, u);
                s.t_time[g] = next;
                fired += nfired;
            }
            if (own) {
                const size_t k = (size_t) j * s.Ntot + g;
                s.t_rate[k] = rate;
                s.react_time[k] = time;
                s.react_inf[k] = inf;
                s.react_ctr[k] = ctr;
            }
            need = true;
        }
        __syncwarp();
    }
    add_fired(s, fired);
}

/* The day's end (src/solvers/SimInf_solver_aem.c:329-381): post-time-step
 * function, U/V columns, and for a node an event touched or whose v
 * changed, every rate recomputed with v_new at tt and its event time
 * rescaled at the node's time (the end of the day). */
template <class M>
__device__ __forceinline__ int aem_pts_node(const DevState &s, long long g, int day, double tt,
                                            int c0, int c1, const double *v_in, double *v_out);

template <class M>
__global__ void __launch_bounds__(256) k_aem_pts(DevState s, int day, double tt, int c0, int c1,
                                                 const double *v_in, double *v_out)
{
    day_begin();
    const long long g = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    int cls = -1;
    if (g < s.Ntot && load_flag(s.err_day) >= day)
        cls = aem_pts_node<M>(s, g, day, tt, c0, c1, v_in, v_out);
    push_heavy(s, g, cls, 0, -1, day + 1);
}

/* k_aem_pts for one node; returns its heavy class on the next day. */
template <class M>
__device__ __forceinline__ int aem_pts_node(const DevState &s, long long g, int day, double tt,
                                            int c0, int c1, const double *v_in, double *v_out)
{
    constexpr int NC = M::NC, NT = M::NT, ND = M::ND;
    const int rep = rep_of(s, g), node = node_of(s, g);
    AemNode<M> a;
    load_u<NC>(s.u + g * NC, a.u);
    const double *vi = v_in + g * ND;
    double *vo = v_out + g * ND;
    const double *ld = s.ldata + (size_t) node * s.Nld;
    const double *gd = gdata_of(s, g);
    const int rc = M::PTS_LOCAL ? M::pts(vo, a.u, vi, ld, gd, node, tt)
                                : M::pts(vo, s.u + g * NC, vi, ld, gd, node, tt);
    store_columns<NC, ND>(s, rep, node, a.u, vo, c0, c1);
    if (rc < 0) {
        record_error(s, rc, PHASE_PTS, day, g, -1, -1, tt, 0);
        return -1;
    }
    double sum = 0.0;
    if (rc == 0 && !s.update[g]) {
#pragma unroll
        for (int j = 0; j < NT; j++)
            sum += s.t_rate[(size_t) j * s.Ntot + g];
        return heavy_class<M>(s, sum);
    }
    const double tc = s.t_time[g];
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const size_t k = (size_t) j * s.Ntot + g;
        a.rate[j] = s.t_rate[k];
        a.time[j] = s.react_time[k];
        a.inf[j] = s.react_inf[k];
        a.ctr[j] = s.react_ctr[k];
    }
    a.err = 0;
    si_recip dc = si_recip_none();
#pragma unroll
    for (int j = 0; j < NT; j++) {
        aem_refresh<M>(s, a, g, j, vo, ld, gd, tt, tc, dc);
        if (a.err) {
            record_error(s, ERR_INVALID_RATE, PHASE_PTS, day, g, j, -1, tt, a.err_rate);
            a.err = 0;
        }
    }
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const size_t k = (size_t) j * s.Ntot + g;
        s.t_rate[k] = a.rate[j];
        s.react_time[k] = a.time[j];
        s.react_inf[k] = a.inf[j];
        s.react_ctr[k] = a.ctr[j];
        sum += a.rate[j];
    }
    s.update[g] = 0;
    return heavy_class<M>(s, sum);
}

/* M::pts() writes every entry of v_new, whatever the day: the shipped
 * models.  The C code of a compiled model may leave an entry alone, which
 * then holds the value of two days before: v and v_new are two buffers that
 * change places at each day's end. */
template <class M, class = void>
struct model_pts_sets_v {
    static constexpr bool value = M::ND == 0;
};
template <class M>
struct model_pts_sets_v<M, decltype((void) M::PTS_SETS_V)> {
    static constexpr bool value = M::PTS_SETS_V;
};

/* A rate sum of 64 or more: a day of a lone chain, not of a node among many. */
__device__ __forceinline__ bool busy_sum(double sum)
{
    return (unsigned) (si_double_bits(sum) >> 32) - 0x40500000u < 0x7FF00000u - 0x40500000u;
}

/* Every day of one node, for rates that ignore t: each pass of the loop is
 * one draw of a waiting time.  It ends in a transition or in the end of a
 * day, and both end in the same code: the rates at the new state (u after a
 * transition, v after a day's post time step) and their changes to the rate
 * sum.  The lanes of a warp so go through their days each at its own pace,
 * and a pass costs them one evaluation of the rates, where a loop over days
 * waits each day for the warp's busiest node: 35 draws and 7 post time steps
 * a week of the particle filter's SISe, against about 21 passes.  What a
 * step meets rarely (a division off the integer path, a zero rate selected,
 * a negative state, an invalid rate, the transition bound) is redone on the
 * exact path, to the end of that day.
 * With BUSY, a warp whose every node fires 64 times a day or more (busy_sum)
 * runs its nodes to the end of the day as ssa_run_day does: lanes at
 * different days gain nothing there, and a draw a pass is a longer chain than
 * a quarter of a batch of four.  Its test costs the other warps 1 to 3%
 * (1,000 to 40,000 nodes of 100), and where warps are many a chain's latency
 * is hidden, so it is for the smaller runs (Launch::horizon).
 * Every lane of the warp calls it; `alive` says whether it has a node. */
template <class M, bool BUSY>
__device__ __forceinline__ void horizon_passes(const DevState &s, const DayInfo *days, int ndays,
                                               long long g, bool alive, SsaLane<M> &ln, si_rng &r,
                                               uint64_t &c_other, const int *sS,
                                               const uint32_t *sG, const si_nl_tables *nl,
                                               unsigned long long &fired)
{
    constexpr int NC = M::NC, NT = M::NT, ND = M::ND;
    constexpr uint32_t ALL = NT == 32 ? 0xFFFFFFFFu : (1u << NT) - 1u;
    const unsigned FULL = 0xFFFFFFFFu;
    const int rep = rep_of(s, g), node = node_of(s, g);
    const double *ld = s.ldata + (size_t) node * s.Nld;
    const double *gd = gdata_of(s, g);
    /* v, and the other buffer's values where a post time step may keep some */
    constexpr bool KEEPS = !model_pts_sets_v<M>::value;
    double v[ND > 0 ? ND : 1], vo[ND > 0 ? ND : 1];
#pragma unroll
    for (int d = 0; d < ND; d++) {
        v[d] = s.vA[g * ND + d];
        if (KEEPS)
            vo[d] = s.vB[g * ND + d];
    }
    int2 e1;
    e1.x = s.e1_ptr[node];
    e1.y = e1.x < s.e1_ptr[node + 1] ? s.e1[e1.x].day : NO_E1;
    const bool mine = alive;
    int d = 0, err_day = INT_MAX;
    DayInfo di = {0.0, 0.0, 0, 0};
    if (ndays > 0)
        di = days[0];
    else
        alive = false;
    ln.c = r.ctr;
    ln.fired = 0;
    ln.err = 0;
    ln.q3 = 0;
    uint64_t have = ~0ULL;              /* the Philox block whose last word ln.q3 is */
    bool day_over = false;              /* the day ended on the exact path */
    bool busy = false;                  /* a long day is ahead of the node */
    for (;;) {
        enum { NONE, FIRES, ENDS, REDO };
        if (__builtin_expect(!__any_sync(FULL, alive && !busy), 0)) {
            if (!BUSY || !__any_sync(FULL, alive))
                break;
            /* every node here is busy: their days in batches of four draws */
            if (alive) {
                ln.err_tr = -1;
                ln.err_t = 0.0;
                ln.err_rate = 0.0;
                ssa_run_day<M>(ln, r, di.next, v, ld, gd, sS, sG, s.max_fired, nl);
                have = ~0ULL;
                day_over = true;
                if (ln.err) {
                    record_error(s, ln.err, PHASE_SSA, d, g, ln.err_tr, -1, ln.err_t, ln.err_rate);
                    fired += ln.fired;
                    alive = false;
                }
            }
            __syncwarp();
        }
        int kind = alive ? ENDS : NONE;
        const bool draws = alive && !day_over && si_finite_pos(ln.sum);
        double L = 0.0, U = 0.0, tn = ln.t;
        uint32_t n0 = 0, n1 = 0, n2 = 0, n3 = 0;
        int u2[NC], redo = 0;
        uint32_t mask = 0;
#pragma unroll
        for (int c = 0; c < NC; c++)
            u2[c] = ln.u[c];
        if (draws) {
            const uint32_t iw = (uint32_t) ln.c & 3u;
            philox_block(r, (ln.c + 1) >> 2, n0, n1, n2, n3);
            uint32_t wl = word_of(n0, n1, n2, n3, iw);
            if (iw == 3u) {
                wl = ln.q3;
                if (have != ln.c >> 2) {
                    uint32_t x0, x1, x2;
                    philox_block(r, ln.c >> 2, x0, x1, x2, wl);
                }
            }
            have = (ln.c + 1) >> 2;
            ln.q3 = n3;
            L = si_neglog_u32_in(wl, nl);
            U = si_u32_to_uniform_pos(word_of(n0, n1, n2, n3, (iw + 1u) & 3u));
            const double tau = si_div_spec(L, ln.sum, &redo);
            tn = tau + ln.t;
            kind = redo ? REDO : si_dge_num(tn, di.next) ? ENDS : FIRES;
        }
        if (kind == FIRES) {
            const int tr = select_transition<M>(ln.rate, U * ln.sum);
            double rtr = ln.rate[0];
#pragma unroll
            for (int k = 1; k < NT; k++)
                if (tr == k)
                    rtr = ln.rate[k];
            redo = si_is_zero(rtr) | (ln.fired + 1u > s.max_fired);
#pragma unroll
            for (int c = 0; c < NC; c++) {
                u2[c] = ln.u[c] + sS[tr * NC + c];
                redo |= u2[c] < 0;
            }
            mask = sG[tr];
        }
        double vn[ND > 0 ? ND : 1];
#pragma unroll
        for (int c = 0; c < ND; c++)
            vn[c] = KEEPS && kind == ENDS ? vo[c] : v[c];
        if (kind == ENDS) {
            if (draws)
                ln.c += 1;                  /* the waiting time's draw was used */
            else if (!day_over && !le_zero(si_double_bits(ln.sum)))
                ln.err = ERR_INVALID_RATE;
            /* the exact path sets the time itself: all rates zero under a
             * positive sum leaves it at that step */
            if (!day_over)
                ln.t = di.next;
            fired += ln.fired;
            if (ln.err) {
                record_error(s, ln.err, PHASE_SSA, d, g, -1, -1, tn, ln.sum);
                alive = false;
                kind = NONE;
            }
        }
        if (kind == ENDS) {
            int e_code = 0, e_idx = -1;
            bool upd = false;
            if (e1.y == d) {
                /* the events draw from the node's stream: with common random
                 * numbers its own counter, else the SSA's */
                r.ctr = s.crn_ctr ? c_other : ln.c;
                r.have = 0;
                if (s.crn_ctr)
                    r.s1 ^= SI_CRN_S1;
                if constexpr (NC <= 2)
                    upd = node_e1_call<NC>(s, u2, e1, node, d, r, e_code, e_idx);
                else
                    upd = node_e1<NC>(s, u2, e1, node, d, r, e_code, e_idx);
                if (s.crn_ctr) {
                    r.s1 ^= SI_CRN_S1;
                    c_other = r.ctr;
                } else {
                    ln.c = r.ctr;
                }
            }
            int rc = 0;
            if (!e_code)
                rc = M::pts(vn, u2, v, ld, gd, node, di.tt);
            if (e_code || rc < 0) {
                record_error(s, e_code ? e_code : rc, e_code ? PHASE_E1 : PHASE_PTS, d, g, -1,
                             e_idx, di.tt, 0);
#pragma unroll
                for (int c = 0; c < NC; c++)
                    ln.u[c] = u2[c];
                alive = false;
                kind = NONE;
            }
            mask = rc > 0 || upd ? ALL : 0u;
        }
        __syncwarp();
        /* the rates that the pass refreshes, in order, and the rate sum */
        double rate2[NT], sum2 = ln.sum;
        if (mask != 0 && kind != NONE) {
            double delta = 0.0;
#pragma unroll
            for (int k = 0; k < NT; k++) {
                const double nr = M::rate(k, u2, vn, ld, gd, ln.t, ln.dc);
                const bool m = (mask >> k) & 1u;
                rate2[k] = m ? nr : ln.rate[k];
                const double dk = k == 0 ? nr - ln.rate[k] : delta + (nr - ln.rate[k]);
                delta = m ? dk : delta;
                if (m && si_bad_rate(nr)) {
                    redo = 1;
                    if (kind == ENDS) {
                        record_error(s, ERR_INVALID_RATE, PHASE_PTS, d, g, k, -1, di.tt, nr);
                        alive = false;
                    }
                }
            }
            sum2 = ln.sum + delta;
        } else {
#pragma unroll
            for (int k = 0; k < NT; k++)
                rate2[k] = ln.rate[k];
        }
        if (kind == FIRES) {
            /* a sum of zero or below ends the day at the next pass; one that
             * is not a number is the exact path's error */
            redo |= !si_finite_pos(sum2) && !le_zero(si_double_bits(sum2));
            if (redo)
                kind = REDO;
        }
        if (kind == REDO) {
            ln.L = L;
            ln.U = U;
            ln.q0 = n0;
            ln.q1 = n1;
            ln.q2 = n2;
            ln.err_tr = -1;
            ln.err_t = 0.0;
            ln.err_rate = 0.0;
            while (!ssa_step_ahead<M>(ln, r, di.next, v, ld, gd, sS, sG, s.max_fired))
                ;
            have = ~0ULL;
            day_over = true;
            busy = false;
            if (ln.err) {
                record_error(s, ln.err, PHASE_SSA, d, g, ln.err_tr, -1, ln.err_t, ln.err_rate);
                fired += ln.fired;
                alive = false;
            }
        } else if (kind != NONE) {
#pragma unroll
            for (int c = 0; c < NC; c++)
                ln.u[c] = u2[c];
#pragma unroll
            for (int k = 0; k < NT; k++)
                ln.rate[k] = rate2[k];
            ln.sum = sum2;
            if (kind == FIRES) {
                ln.t = tn;
                ln.c += 2;
                ln.fired++;
                busy = BUSY && busy_sum(sum2);
            } else if (alive) {
                busy = false;
                store_columns<NC, ND>(s, rep, node, ln.u, vn, di.c0, di.c1);
#pragma unroll
                for (int c = 0; c < ND; c++) {
                    if (KEEPS)
                        vo[c] = v[c];
                    v[c] = vn[c];
                }
                ln.fired = 0;
                day_over = false;
                d++;
                /* an error elsewhere stops the run; read a day ahead of its
                 * use, off the chain */
                if (d >= ndays || err_day < d) {
                    alive = false;
                } else {
                    err_day = load_flag(s.err_day);
                    di = days[d];
                }
            }
        }
    }
    if (mine) {
#pragma unroll
        for (int c = 0; c < ND; c++) {
            s.vA[g * ND + c] = v[c];
            if (KEEPS)
                s.vB[g * ND + c] = vo[c];
        }
    }
    r.ctr = ln.c;
}

/* Whole horizon of one (replicate, node) in one thread: valid when no
 * external transfer couples nodes and the post-time-step function reads
 * only its own node. */
template <class M, bool BUSY>
__global__ void __launch_bounds__(HORIZON_BLOCK, M::NT <= 4 ? 4 : 2)
k_horizon(DevState s, const DayInfo *days, int ndays, int lanes)
{
    if (s.pf_days)
        days = s.pf_days + (size_t) *s.pf_interval * s.pf_days_stride;
    constexpr int NC = M::NC, NT = M::NT, ND = M::ND;
    __shared__ int sS[NT * NC];
    __shared__ uint32_t sG[NT];
    __shared__ __align__(16) si_nl_tables nl;
    load_nl_smem(nl);
    load_model_smem<M>(s, sS, sG);
    const int lane = threadIdx.x & 31;
    const long long at =
        (blockIdx.x * (long long) (HORIZON_BLOCK / 32) + threadIdx.x / 32) * lanes + lane;
    unsigned long long fired = 0;
    const bool have = lane < lanes && at < s.Ntot;
    const long long g = have ? at : 0;          /* a lane without a node reads node 0 */
    SsaLane<M> ln;
    load_u<NC>(s.u + g * NC, ln.u);
#pragma unroll
    for (int k = 0; k < NT; k++)
        ln.rate[k] = s.t_rate[(size_t) k * s.Ntot + g];
    ln.sum = s.sum_rate[g];
    ln.t = s.t_time[g];
    ln.dc = si_recip_none();
    si_rng r;
    uint64_t c_other = 0;       /* common random numbers: the other stream's counter */
    {
        uint64_t seed, sid;
        stream_key(s, g, seed, sid);
        if (s.crn_ctr) {
            /* r holds the SSA's own stream; the events switch to the node's */
            si_rng_init(&r, seed, sid, s.crn_ctr[g]);
            r.s1 |= SI_CRN_S1;
            c_other = s.ctr[g];
        } else {
            si_rng_init(&r, seed, sid, s.ctr[g]);
        }
    }
    if constexpr (M::RATES_TIME_INVARIANT) {
        horizon_passes<M, BUSY>(s, days, ndays, g, have, ln, r, c_other, sS, sG, &nl, fired);
    } else if (have) {
        const int rep = rep_of(s, g), node = node_of(s, g);
        double *v = s.vA + g * ND, *vn = s.vB + g * ND;
        const double *ld = s.ldata + (size_t) node * s.Nld;
        const double *gd = gdata_of(s, g);
        int2 at;
        at.x = s.e1_ptr[node];
        at.y = at.x < s.e1_ptr[node + 1] ? s.e1[at.x].day : NO_E1;
        for (int d = 0; d < ndays; d++) {
            if (load_flag(s.err_day) < d)
                break;
            const DayInfo di = days[d];
            ln.err = 0;
            ln.err_tr = -1;
            ln.err_t = 0.0;
            ln.err_rate = 0.0;
            fired += ssa_day<M>(ln, r, di.next, v, ld, gd, sS, sG, s.max_fired, &nl);
            if (ln.err) {
                record_error(s, ln.err, PHASE_SSA, d, g, ln.err_tr, -1, ln.err_t, ln.err_rate);
                break;
            }
            int e_code = 0, e_idx = -1;
            if (s.crn_ctr) {
                const uint64_t t = r.ctr;   /* to the node's stream */
                r.ctr = c_other;
                c_other = t;
                r.s1 ^= SI_CRN_S1;
                r.have = 0;
            }
            bool upd = false;
            if constexpr (NC <= 2) {
                if (at.y == d)
                    upd = node_e1_call<NC>(s, ln.u, at, node, d, r, e_code, e_idx);
            } else {
                upd = node_e1<NC>(s, ln.u, at, node, d, r, e_code, e_idx);
            }
            if (s.crn_ctr) {
                const uint64_t t = r.ctr;   /* back to the SSA's */
                r.ctr = c_other;
                c_other = t;
                r.s1 ^= SI_CRN_S1;
                r.have = 0;
            }
            if (e_code) {
                record_error(s, e_code, PHASE_E1, d, g, -1, e_idx, di.tt, 0);
                break;
            }
            const int rc = M::pts(vn, ln.u, v, ld, gd, node, di.tt);
            if (rc < 0) {
                record_error(s, rc, PHASE_PTS, d, g, -1, -1, di.tt, 0);
                break;
            }
            if (rc > 0 || upd) {
                double delta = 0.0;
                bool bad = false;
#pragma unroll
                for (int k = 0; k < NT; k++) {
                    const double old = ln.rate[k];
                    const double nr = M::rate(k, ln.u, vn, ld, gd, di.tt, ln.dc);
                    ln.rate[k] = nr;
                    delta += nr - old;
                    if (si_bad_rate(nr)) {
                        record_error(s, ERR_INVALID_RATE, PHASE_PTS, d, g, k, -1, di.tt, nr);
                        bad = true;
                    }
                }
                ln.sum += delta;
                if (bad)
                    break;
            }
            store_columns<NC, ND>(s, rep, node, ln.u, vn, di.c0, di.c1);
            double *tmp = v;
            v = vn;
            vn = tmp;
        }
    }
    if (have) {
        store_u<NC>(s.u + g * NC, ln.u);
#pragma unroll
        for (int k = 0; k < NT; k++)
            s.t_rate[(size_t) k * s.Ntot + g] = ln.rate[k];
        s.sum_rate[g] = ln.sum;
        s.t_time[g] = ln.t;
        if (s.crn_ctr) {
            s.crn_ctr[g] = r.ctr;
            s.ctr[g] = c_other;
        } else {
            s.ctr[g] = r.ctr;
        }
    }
    add_fired(s, fired);
}

/* ------------------------------------------------------------------ */
/* Launchers, one table per model.                                      */
/* ------------------------------------------------------------------ */

static inline unsigned blocks_for(long long n, int threads)
{
    return (unsigned) ((n + threads - 1) / threads);
}

static inline int sm_count()
{
    static const int n = [] {           /* once, whichever thread comes first */
        int dev = 0, count = 1;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
        return count;
    }();
    return n;
}

/* Launch a day's kernel; chained, it may start while the kernel before it in
 * the stream drains, and waits in day_begin() for that kernel's writes. */
template <class K, class... A>
static cudaError_t launch_day(bool chained, unsigned cluster, K kernel, unsigned grid,
                              unsigned block, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[2] = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cfg.attrs = at;
    if (chained) {
        at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        at[cfg.numAttrs].val.clusterDim.x = cluster;
        at[cfg.numAttrs].val.clusterDim.y = at[cfg.numAttrs].val.clusterDim.z = 1;
        cfg.numAttrs++;
    }
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <class M>
struct Launch {
    static cudaError_t init(const DevState &s, double tt0, cudaStream_t st)
    {
        k_init<M><<<blocks_for(s.Ntot, 256), 256, 0, st>>>(s, tt0);
        return cudaGetLastError();
    }
    static cudaError_t horizon(const DevState &s, const DayInfo *days, int ndays, cudaStream_t st)
    {
        /* a warp for each of the chip's schedulers before more lanes a warp:
         * fewer lanes wait for one another's branches (SIR, 1,000 nodes x
         * 150 days: 0.91 ms with 32 lanes, 0.74 with 2; 20,000 nodes x 365
         * days: 1.42 ms with 32 lanes, 1.54 with 16) */
        int lanes = 32;
        while (lanes > 1 && (s.Ntot + lanes / 2 - 1) / (lanes / 2) <= 4ll * sm_count())
            lanes /= 2;
        const unsigned grid = blocks_for(s.Ntot, lanes * (HORIZON_BLOCK / 32));
        /* up to four warps a scheduler, busy days in batches of four draws
         * (SIR, nodes of 3,000 x 40 days: 40,000 nodes 12.5 ms without, 11.8
         * with; 80,000 22.3, 21.3; 160,000 35.3, 37.3; one node of 200,000 x
         * 60 days 326, 206) */
        if constexpr (M::RATES_TIME_INVARIANT) {
            if (s.Ntot <= 4 * 32 * 4ll * sm_count()) {
                k_horizon<M, true><<<grid, HORIZON_BLOCK, 0, st>>>(s, days, ndays, lanes);
                return cudaGetLastError();
            }
        }
        k_horizon<M, false><<<grid, HORIZON_BLOCK, 0, st>>>(s, days, ndays, lanes);
        return cudaGetLastError();
    }
    /* k_ssa_e1 is persistent: as many blocks as can be resident at once
     * (looked up once per model), fewer for small models. */
    /* The SSA kernel's two register budgets: blocks of SSA_BLOCK threads
     * resident per SM that __launch_bounds__ asks for (the default keeps
     * larger models within their registers; the other trades warps for
     * registers). */
    static constexpr int SSA_MINB0 = M::NT <= 4 ? 4 : 3;
    static constexpr int SSA_MINB1 = M::NT <= 4 ? 3 : 2;
    template <int MINB>
    static int ssa_resident_blocks()
    {
        static int blocks = 0;
        if (!blocks) {
            int dev = 0, nsm = 1, per = 0;
            cudaGetDevice(&dev);
            cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_ssa_e1<M, MINB>, SSA_BLOCK, 0);
            blocks = nsm * (per > 0 ? per : 1);
        }
        return blocks;
    }
    template <int MINB>
    static cudaError_t ssa_e1_with(const DevState &s, int day, double tt, double next,
                                   cudaStream_t st)
    {
        /* a warp of its own for every node where the chip has room for it */
        const long long need = (long long) blocks_for(s.Ntot, SSA_BLOCK / 32);
        const int resident = ssa_resident_blocks<MINB>();
        const int grid = (int) (need < resident ? need : resident);
        return launch_day(s.chained, 1, k_ssa_e1<M, MINB>, grid, SSA_BLOCK, st, s, day, tt, next);
    }
    static cudaError_t quick(const DevState &s, int day, double tt, double next, cudaStream_t st)
    {
        return launch_day(s.chained, 1, k_quick<M>, blocks_for(s.Ntot, 256), 256, st, s, day, tt,
                          next);
    }
    static cudaError_t ssa_e1(const DevState &s, int day, double tt, double next, cudaStream_t st)
    {
        /* the larger register budget also where its warps have at most two
         * nodes each: a model that small has no use for more warps (SISe3,
         * 1,600 nodes: 100 bytes a thread spilled under the smaller one) */
        const bool small = model_rates_total<M>::value &&
                           (long long) blocks_for(s.Ntot, SSA_BLOCK / 16) <=
                               ssa_resident_blocks<SSA_MINB1>();
        return s.ssa_variant == 1 || small
                   ? ssa_e1_with<SSA_MINB1>(s, day, tt, next, st)
                   : ssa_e1_with<SSA_MINB0>(s, day, tt, next, st);
    }
    static cudaError_t e2_tail(const DevState &s, const E2Rec *ev, const E2Tail &tail, int day,
                               double tt, cudaStream_t st)
    {
        const unsigned blocks = tail.wide > 0 ? E2_CLUSTER : 1;
        return launch_day(s.chained, blocks, k_e2_tail<M>, blocks, E2_TAIL_BLOCK, st, s, ev, tail,
                          day, tt);
    }
    static cudaError_t e2_wave(const DevState &s, const E2Rec *ev, int count, int day, double tt,
                               cudaStream_t st)
    {
        const long long n = (long long) count * s.Nrep;
        if (n == 0)
            return cudaSuccess;
        const int b = (s.wave_block == 256 || s.wave_block == 512) ? s.wave_block : 128;
        return launch_day(s.chained, 1, k_e2_wave<M>, blocks_for(n, b), b, st, s, ev, count, day, tt);
    }
    static cudaError_t pts_store(const DevState &s, int day, double tt, int c0, int c1,
                                 const double *v_in, double *v_out, cudaStream_t st)
    {
        /* small models in small blocks, over more SMs: the FP64 pipe takes a
         * warp instruction in 64 cycles, and two warps would share one */
        const int b = s.Ntot <= 65536 ? 64 : 256;
        return launch_day(s.chained, 1, k_pts_store<M>, blocks_for(s.Ntot, b), b, st, s, day, tt, c0,
                          c1, v_in, v_out);
    }
    static cudaError_t aem_init(const DevState &s, double tt0, cudaStream_t st)
    {
        k_aem_init<M><<<blocks_for(s.Ntot, 256), 256, 0, st>>>(s, tt0);
        return cudaGetLastError();
    }
    template <bool WIDE>
    static int aem_resident_blocks()
    {
        static const int blocks = [] {
            int per = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_aem_day<M, WIDE>, SSA_BLOCK, 0);
            return sm_count() * (per > 0 ? per : 1);
        }();
        return blocks;
    }
    template <bool WIDE>
    static cudaError_t aem_day_with(const DevState &s, int day, double tt, double next,
                                    cudaStream_t st)
    {
        const long long need = (long long) blocks_for(s.Ntot, SSA_BLOCK / AemLanes<M>::value);
        const int resident = aem_resident_blocks<WIDE>();
        const int grid = (int) (need < resident ? need : resident);
        return launch_day(s.chained, 1, k_aem_day<M, WIDE>, grid, SSA_BLOCK, st, s, day, tt, next);
    }
    static cudaError_t aem_day(const DevState &s, int day, double tt, double next, cudaStream_t st)
    {
        /* from eight nodes a resident group, quiet ones are looked through by
         * lanes (SEIR of 1% infected nodes, 10^6 x 20 days 9.8 ms without, 8.3
         * with; 300,000 x 30 5.6, 5.1; at five nodes a group SIS, 200,000 x 40,
         * 3.9, 4.1) */
        const long long groups =
            (long long) aem_resident_blocks<true>() * (SSA_BLOCK / AemLanes<M>::value);
        return s.Ntot >= 8 * groups ? aem_day_with<true>(s, day, tt, next, st)
                                    : aem_day_with<false>(s, day, tt, next, st);
    }
    static cudaError_t aem_pts(const DevState &s, int day, double tt, int c0, int c1,
                               const double *v_in, double *v_out, cudaStream_t st)
    {
        return launch_day(s.chained, 1, k_aem_pts<M>, blocks_for(s.Ntot, 256), 256, st, s, day, tt,
                          c0, c1, v_in, v_out);
    }
    static const Launchers *table()
    {
        static const Launchers t = {M::NC, M::NT, M::ND, M::NGD, M::PTS_LOCAL,
                                    M::RATES_TIME_INVARIANT, model_rates_total<M>::value,
                                    model_pts_sets_v<M>::value, init, horizon, quick, ssa_e1,
                                    e2_wave, pts_store, aem_init, aem_day, aem_pts, e2_tail};
        return &t;
    }
};

}  // namespace siminf

#endif
