// pb_interp64.cu -- FP64 point interpolation kernels (reference arithmetic).
// Compiled with -fmad=false so that every expression is the IEEE result of the
// reference's operation order (no FMA contraction).
#include "pb_internal.h"
#include "pb_fp64_impl.cuh"

namespace pb {

template <int STRAT, int KT>
__global__ void __launch_bounds__(128) k_points64w(DevTree T, DevCatalog C, int64_t nq, const double *__restrict__ qx,
                                                   const double *__restrict__ qy, const double *__restrict__ qz,
                                                   const uint32_t *__restrict__ perm, int64_t npts,
                                                   unsigned long long *counter)
{
    __shared__ __align__(16) double sterm[4][TBUF];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    for (;;) {
        int64_t j = next_query(counter, lane);
        if (j >= nq) break;
        int64_t qi = perm ? (int64_t)__ldg(perm + j) : j;
        if (qi >= npts) continue;
        const double px = __ldg(qx + qi), py = __ldg(qy + qi), pz = __ldg(qz + qi);
        const int64_t bnear = STRAT != SCATTER ? nearest_leaf(T, px, py, pz) : -1;
        points64_query<STRAT, KT>(T, C, px, py, pz, bnear, qi, sterm[wib], lane, 1);
    }
}

// Two-phase form: the walked queries' runs are read (deal_runs) instead of walking, with the
// same per-slot terms and the same in-order column sums, so the values are those of k_points64w
// bit for bit.  The queries of a higher size class than block_min leaves, which are the first of
// the order, are taken by whole blocks (pairs64_block), the others by single
// warps once no such query is left.
// number of queries at the front of the order (descending size classes, deferred queries last) of a
// higher class than `above` accepted leaves: a 32-way search, the same in every warp
__device__ __forceinline__ int64_t count_above(const RunPool &P, int64_t m, const uint32_t *__restrict__ order,
                                               unsigned above, int lane)
{
    if (above == 0xffffffffu) return 0;
    int64_t lo = 0, hi = m;   // the answer lies in [lo, hi]
    while (lo < hi) {
        const int64_t step = (hi - lo + 31) / 32, t = lo + lane * step;
        bool more = false;
        if (t < hi) {
            const uint32_t j = __ldg(order + t);
            more = !__ldg(P.qflag + j) && count_class(__ldg(P.qacc + j)) > count_class(above);
        }
        const int k = __popc(__ballot_sync(0xffffffffu, more));   // the first k probes are above
        if (k == 0) return lo;
        hi = min(hi, lo + k * step);
        lo = lo + (k - 1) * step + 1;
    }
    return lo;
}

template <int STRAT, int KT, int CAT>
__global__ void __launch_bounds__(128, minb64<STRAT, CAT>()) k_pairs64w(
    DevTree T, DevCatalog C, RunPool P, int64_t m, unsigned block_min, const uint32_t *__restrict__ ql,
    const uint32_t *__restrict__ order, const double *__restrict__ qx, const double *__restrict__ qy,
    const double *__restrict__ qz, unsigned long long *counter)
{
    __shared__ __align__(16) double sterm[BLOCK64_BUFS][nterms64<CAT>() * TROW];
    __shared__ unsigned long long s_next;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t nblk = count_above(P, m, order, block_min, lane);
    if (nblk > 0) {
        unsigned long long nxt = 0;
        if (threadIdx.x == 0) nxt = atomicAdd(counter, 1ULL);
        for (;;) {
            if (threadIdx.x == 0) s_next = nxt;
            __syncthreads();   // also: every warp is done with the previous query's term buffers
            const int64_t t = (int64_t)s_next;
            if (t >= nblk) break;
            if (threadIdx.x == 0) nxt = atomicAdd(counter, 1ULL);
            const int64_t j = __ldg(order + t);
            if (!__ldg(P.qflag + j)) {
                const int64_t qi = __ldg(ql + j);
                pairs64_block<STRAT, KT, CAT>(T, C, P, j, qi, __ldg(qx + qi), __ldg(qy + qi), __ldg(qz + qi),
                                              STRAT != SCATTER ? (int64_t)__ldg(P.bnear + j) : -1,
                                              (int)__ldg(P.qacc + j), sterm[0], wib, lane);
            }
            __syncthreads();   // s_next has been read by every warp
        }
    }
    // the next query's position in the order is fetched (lane 0's atomic) while the current
    // one is summed, so the counter's latency overlaps the work; which warp sums a query does
    // not change its value
    unsigned long long nxt = 0;
    if (lane == 0) nxt = atomicAdd(counter + 1, 1ULL);
    int64_t t = nblk + (int64_t)__shfl_sync(0xffffffffu, nxt, 0);
    while (t < m) {
        if (lane == 0) nxt = atomicAdd(counter + 1, 1ULL);
        const int64_t j = order ? (int64_t)__ldg(order + t) : t;
        if (!__ldg(P.qflag + j)) {
            const int64_t qi = __ldg(ql + j);
            const double px = __ldg(qx + qi), py = __ldg(qy + qi), pz = __ldg(qz + qi);
            pairs64_query<STRAT, KT, CAT>(T, C, P, j, qi, px, py, pz,
                                          STRAT != SCATTER ? (int64_t)__ldg(P.bnear + j) : -1, sterm[wib], lane);
        }
        t = nblk + (int64_t)__shfl_sync(0xffffffffu, nxt, 0);
    }
}

static int persistent_grid(const void *kern, int bs)
{
    int dev = 0, sms = 148, per = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, bs, 0);
    return sms * (per > 0 ? per : 1);
}

// run-time (strategy, kernel family) -> F::run<STRAT, KT>()
template <int STRAT, typename F>
static void dispatch_kernel(int kernel, F &f)
{
    switch (kernel) {
    case 0: f.template run<STRAT, 0>(); break;
    case 1: f.template run<STRAT, 1>(); break;
    case 2: f.template run<STRAT, 2>(); break;
    case 3: f.template run<STRAT, 3>(); break;
    case 4: f.template run<STRAT, 4>(); break;
    default: f.template run<STRAT, 5>(); break;
    }
}

template <typename F>
static void dispatch(int strategy, int kernel, F &f)
{
    switch (strategy) {
    case GATHER: dispatch_kernel<GATHER>(kernel, f); break;
    case SCATTER: dispatch_kernel<SCATTER>(kernel, f); break;
    default: dispatch_kernel<SYMMETRIC>(kernel, f); break;
    }
}

namespace {

struct PointsLaunch {
    Handle *H;
    const DevTree &T;
    const DevCatalog &C;
    int64_t nq;
    const double *qx, *qy, *qz;
    const uint32_t *perm;
    int64_t npts;
    unsigned long long *ctr;
    template <int STRAT, int KT>
    void run()
    {
        k_points64w<STRAT, KT><<<persistent_grid((const void *)k_points64w<STRAT, KT>, 128), 128, 0, H->stream>>>(
            T, C, nq, qx, qy, qz, perm, npts, ctr);
    }
};

struct PairsLaunch {
    Handle *H;
    const DevTree &T;
    const DevCatalog &C;
    const RunPool &P;
    int64_t m;
    unsigned block_min;
    const uint32_t *ql, *order;
    const double *qx, *qy, *qz;
    unsigned long long *ctr;
    template <int STRAT, int KT, int CAT>
    void one()
    {
        k_pairs64w<STRAT, KT, CAT><<<persistent_grid((const void *)k_pairs64w<STRAT, KT, CAT>, 128), 128, 0, H->stream>>>(
            T, C, P, m, block_min, ql, order, qx, qy, qz, ctr);
    }
    template <int STRAT, int KT>
    void run()
    {
        switch (catalog_shape(C)) {
        case CAT_GDC4: one<STRAT, KT, CAT_GDC4>(); break;
        case CAT_C4: one<STRAT, KT, CAT_C4>(); break;
        case CAT_S1: one<STRAT, KT, CAT_S1>(); break;
        case CAT_SG1: one<STRAT, KT, CAT_SG1>(); break;
        default: one<STRAT, KT, CAT_ANY>(); break;
        }
    }
};

}  // namespace

cudaError_t launch_points_fp64(Handle *H, const DevTree &T, const DevCatalog &C, int strategy, int64_t nq,
                               const double *qx, const double *qy, const double *qz, const uint32_t *perm,
                               int64_t npts)
{
    cudaError_t e = H->counter.reserve(sizeof(unsigned long long));
    if (e) return e;
    unsigned long long *ctr = H->counter.as<unsigned long long>();
    cudaMemsetAsync(ctr, 0, sizeof(unsigned long long), H->stream);
    PointsLaunch f{H, T, C, nq, qx, qy, qz, perm, npts, ctr};
    dispatch(strategy, T.kernel, f);
    H->launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_pairs_fp64(Handle *H, const DevTree &T, const DevCatalog &C, int strategy, const RunPool &P,
                              int64_t m, unsigned block_min, const uint32_t *ql, const uint32_t *order,
                              const double *qx, const double *qy, const double *qz)
{
    cudaError_t e = H->counter.reserve(2 * sizeof(unsigned long long));
    if (e) return e;
    unsigned long long *ctr = H->counter.as<unsigned long long>();
    cudaMemsetAsync(ctr, 0, 2 * sizeof(unsigned long long), H->stream);
    PairsLaunch f{H, T, C, P, m, block_min, ql, order, qx, qy, qz, ctr};
    dispatch(strategy, T.kernel, f);
    H->launches += 1;
    return cudaGetLastError();
}

}  // namespace pb
