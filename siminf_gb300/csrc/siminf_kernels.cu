/*
 * siminf_kernels.cu -- the lookup of the models the library ships
 * (siminf_models.cuh; their kernels are instantiated in siminf_models_a.cu,
 * _b.cu and _c.cu), and the particle filter's kernels, which do not depend
 * on the model.
 */
#include "siminf_kernels.cuh"

namespace siminf {

/* ------------------------------------------------------------------ */
/* Particle filter (R/pfilter.R:417-452, src/misc/SimInf_particle_filter.c: */
/* 33-67): log-weights, normalisation, ESS, systematic resampling and   */
/* the ancestors' state copy.  Sums are rounded addition by addition in */
/* particle or node order, so that every bit matches the CPU            */
/* restatement; a warp forms them as prefix sums (ordered_sums).        */
/* ------------------------------------------------------------------ */
#define PF_LOG_FLOOR (-690.0)

__device__ __forceinline__ double pf_logdens(const double *lfact, int tablen, int k, int n,
                                             double logp, double logq)
{
    if (k < 0 || n < 0 || k > n || n >= tablen)
        return PF_LOG_FLOOR;
    return (((lfact[n] - lfact[k]) - lfact[n - k]) + si_i2d(k) * logp) + si_i2d(n - k) * logq;
}

/* x + d(0), then + d(1), ... + d(n - 1), each sum rounded: the last one, and
 * every one in out[] when it is not NULL.  A whole warp calls it.  The warp
 * takes PF_CHUNK additions at once, PF_LANE to a lane: while the sums stay
 * in one binade and no addition is a tie, each adds a whole number of units
 * in the last place, whatever the sum.  A chunk where that fails goes 32
 * additions at a time (ordered_sums, which knows ties), and where that
 * fails, one by one.  4,096 additions: 262,000 cycles one by one. */
enum { PF_LANE = 4, PF_CHUNK = 32 * PF_LANE };

template <class D>
__device__ double pf_ordered(double x, int n, D &&d, double *out)
{
    const unsigned FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    for (int at = 0; at < n; at += PF_CHUNK) {
        const uint64_t X = si_double_bits(x);
        const int ex = (int) (X >> 52) & 0x7FF;
        const uint64_t mx = (X & 0x000FFFFFFFFFFFFFULL) | 0x0010000000000000ULL;
        bool good = ex > 64 && ex < 0x7FE && !(X >> 63);
        int64_t y[PF_LANE], sum = 0;
#pragma unroll
        for (int k = 0; k < PF_LANE; k++) {
            const int i = at + lane * PF_LANE + k;
            const uint64_t D64 = i < n ? si_double_bits(d(i)) : 0;
            const int ed = (int) (D64 >> 52) & 0x7FF;
            const uint64_t md = ed ? (D64 & 0x000FFFFFFFFFFFFFULL) | 0x0010000000000000ULL : 0;
            int sh = ex - ed;
            good &= sh >= 0;
            sh = sh < 0 ? 0 : sh > 60 ? 60 : sh;
            const uint64_t q = md >> sh, twice = (md - (q << sh)) << 1, unit = 1ULL << sh;
            good &= twice != unit;
            const int64_t r = (int64_t) (q + (twice > unit));
            sum += (D64 >> 63) ? -r : r;
            y[k] = sum;
        }
        int64_t upto = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t z = __shfl_up_sync(FULL, upto, o);
            if (lane >= o)
                upto += z;
        }
        const uint64_t before = mx + (uint64_t) (upto - sum);
#pragma unroll
        for (int k = 0; k < PF_LANE; k++) {
            const uint64_t s = before + (uint64_t) y[k];
            good &= s > (1ULL << 52) && s < (1ULL << 53) - 1;
        }
        if (__all_sync(FULL, good)) {
            const uint64_t top = (uint64_t) ex << 52;
#pragma unroll
            for (int k = 0; k < PF_LANE; k++) {
                const int i = at + lane * PF_LANE + k;
                if (out && i < n)
                    out[i] = si_bits_double(top | ((before + (uint64_t) y[k]) &
                                                   0x000FFFFFFFFFFFFFULL));
            }
            const uint64_t last = __shfl_sync(FULL, before + (uint64_t) y[PF_LANE - 1], 31);
            x = si_bits_double(top | (last & 0x000FFFFFFFFFFFFFULL));
            continue;
        }
        for (int c = at; c < n && c < at + PF_CHUNK; c += 32) {
            const int i = c + lane;
            const double di = i < n ? d(i) : 0.0;
            unsigned right;
            double sb = ordered_sums(x, di, 32, lane, lane, FULL, (1u << lane) - 1u, right);
            if (right != FULL)
                sb = ordered_sums_serial(x, di, 32, lane);
            const double sa = sb + di;
            if (out && i < n)
                out[i] = sa;
            x = __shfl_sync(FULL, sa, min(31, n - 1 - c));
        }
    }
    return x;
}

/* A warp a particle: the terms side by side, their sum in node order (of the
 * negated terms: the same roundings, and sums that grow upward).  Bound: the
 * FP64 pipe.  500 nodes: 4,096 particles 233 us with a thread a particle, 94
 * with a warp; 256 particles 224 us, then 27. */
__global__ void __launch_bounds__(128) k_pf_weights(const int *U, int tlen, int Nn, int Nc, int Np,
                                                    const int *obs_row, int obs_c,
                                                    const double *lfact, int tablen, double logp,
                                                    double logq, double *w, const int *interval)
{
    const int p = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    if (p >= Np)
        return;
    if (interval)
        obs_row += (size_t) *interval * Nn;     /* obs_row is the first interval's row */
    const int *last = U + ((size_t) p * tlen + tlen - 1) * (size_t) Nn * Nc;
    const double acc = pf_ordered(0.0, Nn, [&](int node) {
        return -pf_logdens(lfact, tablen, obs_row[node], last[(size_t) node * Nc + obs_c], logp,
                           logq);
    }, nullptr);
    if ((threadIdx.x & 31) == 0)
        w[p] = 0.0 - acc;
}

/* One cluster of PF_CLUSTER blocks; w has room for 3 Np values, the weights
 * and two prefix sums.  The exponentials, the normalisation and the
 * ancestors' searches are spread over the cluster; the three sums in
 * particle order (of the weights, of their squares, the cumulative weights
 * with the resampling points) are a warp's each.  Bound: those sums.  4,096
 * particles: 1,255 us with one thread for the sums on one SM, 123 now; 256
 * particles 85, then 47. */
enum { PF_CLUSTER = 8, PF_BLOCK = 512 };

__global__ void __launch_bounds__(PF_BLOCK)
k_pf_finalize(double *w, int Np, double log_np, double *loglik, double *ess, int i, uint64_t seed,
              uint64_t sid, int *anc, int *anc_out, int *interval, const uint64_t *seed_dev)
{
    if (seed_dev)
        seed = *seed_dev;               /* graph replay: the pass's seed */
    if (interval) {
        /* graph replay: the interval, its resampling stream and its row of
         * ancestors come from the device counter, which moves on at the end */
        i = *interval;
        sid += (uint64_t) i;
        if (anc_out)
            anc_out += (size_t) i * Np;
    }
    __shared__ double red[PF_BLOCK];
    __shared__ double s_x;
    double *cum = w + Np, *points = w + 2 * (size_t) Np;
    const int me = blockIdx.x * blockDim.x + threadIdx.x, all = gridDim.x * blockDim.x;
    const bool first_warp = threadIdx.x < 32;
    double m = -INFINITY;
    for (int p = threadIdx.x; p < Np; p += blockDim.x)
        m = fmax(m, __ldcg(w + p));
    red[threadIdx.x] = m;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o)
            red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + o]);
        __syncthreads();
    }
    const double max_w = red[0];
    cluster_barrier();                  /* every block has read the weights */
    for (int p = me; p < Np; p += all)
        w[p] = si_exp(w[p] - max_w);
    cluster_barrier();
    /* every block forms the sum for itself, and block 0 keeps it */
    if (first_warp) {
        const double sum = pf_ordered(0.0, Np, [&](int p) { return __ldcg(w + p); }, nullptr);
        if (threadIdx.x == 0) {
            s_x = sum;
            if (blockIdx.x == 0)
                *loglik = ((*loglik + max_w) + si_log(sum)) - log_np;
        }
    }
    __syncthreads();
    cluster_barrier();                  /* every block has read the exponentials */
    for (int p = me; p < Np; p += all)
        w[p] = si_div(w[p], s_x);
    cluster_barrier();
    if (blockIdx.x == 0 && first_warp) {
        /* systematic resampling: cumulative weights, then the points */
        const double total = pf_ordered(0.0, Np, [&](int p) { return __ldcg(w + p); }, cum);
        si_rng r;
        si_rng_init(&r, seed, sid, 0);
        const double du = si_div(total, si_i2d(Np));
        const double u = du * si_uniform_pos(&r);
        if (threadIdx.x == 0)
            points[0] = u;
        pf_ordered(u, Np - 1, [&](int) { return du; }, points + 1);
    }
    if (blockIdx.x == 1 && first_warp) {
        const double sq = pf_ordered(0.0, Np, [&](int p) {
            const double x = __ldcg(w + p);
            return x * x;
        }, nullptr);
        if (threadIdx.x == 0)
            ess[i] = si_div(1.0, sq);
    }
    cluster_barrier();
    /* the ancestor of point p: the first particle whose cumulative weight is
     * not below it, or the last */
    for (int p = me; p < Np; p += all) {
        const double u = __ldcg(points + p);
        int lo = 0, hi = Np - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (u > __ldcg(cum + mid))
                lo = mid + 1;
            else
                hi = mid;
        }
        anc[p] = lo;
        if (anc_out)
            anc_out[p] = lo + 1;
    }
    if (interval && me == 0)
        *interval = i + 1;              /* every block has read it: barriers above */
}

__global__ void k_pf_gather(const int *U, const double *V, int tlen, long long nu, long long nv,
                            const int *anc, int Np, int *u0, double *v0)
{
    const long long idx = blockIdx.x * (long long) blockDim.x + threadIdx.x;
    if (idx < (long long) Np * nu) {
        const int p = (int) (idx / nu);
        const long long r = idx - (long long) p * nu;
        u0[idx] = U[((size_t) anc[p] * tlen + tlen - 1) * nu + r];
    }
    if (V && idx < (long long) Np * nv) {
        const int p = (int) (idx / nv);
        const long long r = idx - (long long) p * nv;
        v0[idx] = V[((size_t) anc[p] * tlen + tlen - 1) * nv + r];
    }
}

cudaError_t pf_weights(const int *U, int tlen, int Nn, int Nc, int Np, const int *obs_row,
                       int obs_c, const double *lfact, int tablen, double logp, double logq,
                       double *w, cudaStream_t st, const int *interval)
{
    k_pf_weights<<<(Np + 3) / 4, 128, 0, st>>>(U, tlen, Nn, Nc, Np, obs_row, obs_c, lfact,
                                               tablen, logp, logq, w, interval);
    return cudaGetLastError();
}

cudaError_t pf_finalize(double *w, int Np, double log_np, double *loglik, double *ess, int i,
                        uint64_t seed, uint64_t sid, int *anc, int *anc_out, cudaStream_t st,
                        int *interval, const uint64_t *seed_dev)
{
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    cfg.gridDim = dim3(PF_CLUSTER);
    cfg.blockDim = dim3(PF_BLOCK);
    cfg.stream = st;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = PF_CLUSTER;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_pf_finalize, w, Np, log_np, loglik, ess, i, seed, sid, anc,
                              anc_out, interval, seed_dev);
}

cudaError_t pf_gather(const int *U, const double *V, int tlen, long long nu, long long nv,
                      const int *anc, int Np, int *u0, double *v0, cudaStream_t st)
{
    const long long n = (long long) Np * (nu > nv ? nu : nv);
    k_pf_gather<<<(unsigned) ((n + 255) / 256), 256, 0, st>>>(U, V, tlen, nu, nv, anc, Np, u0, v0);
    return cudaGetLastError();
}

/* The shipped models' launcher tables, instantiated in three translation
 * units (siminf_models_a.cu, _b.cu, _c.cu) that compile in parallel. */
const Launchers *launchers_shipped_a(const char *name);
const Launchers *launchers_shipped_b(const char *name);
const Launchers *launchers_shipped_c(const char *name);

const Launchers *launchers_for(const char *name)
{
    const Launchers *t = launchers_shipped_a(name);
    if (!t)
        t = launchers_shipped_b(name);
    return t ? t : launchers_shipped_c(name);
}

}  // namespace siminf
