// pb_walk.cu -- the traversal half of the two-phase point interpolation.
//
// 1. k_nearest_list: the nearest particle of every query (gather/symmetric strategies;
//    LBVH_find_nearest_h, LinearBVHQueries.jl:118-140), one thread per query.
// 2. k_walk: one warp per query of the (Morton-ordered) list writes the runs of its accepted
//    leaves (pb_walk_impl.cuh).
#include "pb_internal.h"
#include "pb_walk_impl.cuh"

namespace pb {

// Queries whose nearest particle's h is within a factor 8 of the largest have the longest walks (the
// walk's work grows with the surface of the support).  The nearest search lists them, and the walk
// takes them first: in Morton order they come last where a grid's corner lies far from the particles,
// and the launch waited for them (SMs busy 72 % of the walk of 131,072 particles on 64^3 points).
// Where h varies by less than that (a box of even density) every query would be on the list, walked out of
// Morton order, a ticket each, and passed over again: the list is not used where fewer than one query in
// LONG_OTHERS is off it.  On discs up to 0.95 of the points may be on it, with gain.  Nearest search and walk,
// always used / not from a half on / not from 7/8 on: 1e6 even particles, 2e6 points 11.40 / 10.74 / 10.74 ms;
// 131,072 disc particles, 64^3 points (0.58 on the list) 2.15 / 2.83 / 2.15; 400,000 on 80 x 80 x 24 (0.57) 1.92 / 2.95 /
// 1.93; 300,878 clumped, 129 x 138 x 63 (gather, 0.52) 9.94 / 10.65 / 9.93.
constexpr int LONG_OTHERS = 8;

__device__ __forceinline__ bool long_walk(const DevTree &T, int b)
{
    if (T.root == 0 || b < 0) return false;
    return 8.f * (float)ldg4(T.leaf + b).w >= __ldg(T.node_hmax + (T.root - 1));
}

struct LongList {
    uint32_t *list;    // cap entries; NULL: none
    unsigned *count;   // above cap: the list is not used
    unsigned cap;
    __device__ __forceinline__ void add(const DevTree &T, int64_t j, int b) const
    {
        if (!list || !long_walk(T, b)) return;
        const unsigned at = atomicAdd(count, 1u);
        if (at < cap) list[at] = (uint32_t)j;
    }
    __device__ __forceinline__ int64_t used() const { return list && *count <= cap ? (int64_t)*count : 0; }
};

// the list of a launch over m queries
static unsigned long_cap(int64_t m) { return (unsigned)(m - m / LONG_OTHERS); }

static LongList long_list(Handle *H, int64_t m, bool listed)
{
    return LongList{listed ? H->long_list.as<uint32_t>() : nullptr, H->long_count.as<unsigned>(), long_cap(m)};
}

__global__ void __launch_bounds__(128) k_nearest_list(DevTree T, int64_t m, const uint32_t *__restrict__ ql,
                                                      const double *__restrict__ qx, const double *__restrict__ qy,
                                                      const double *__restrict__ qz, int *bnear, LongList longs)
{
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t qi = __ldg(ql + j);
        const int b = (int)nearest_leaf(T, __ldg(qx + qi), __ldg(qy + qi), __ldg(qz + qi));
        bnear[j] = b;
        longs.add(T, j, b);
    }
}

// few queries: a warp each (nearest_leaf_warp)
__global__ void __launch_bounds__(128) k_nearest_list_warp(DevTree T, int64_t m, const uint32_t *__restrict__ ql,
                                                           const double *__restrict__ qx, const double *__restrict__ qy,
                                                           const double *__restrict__ qz, int *bnear, LongList longs)
{
    __shared__ int s_stack[4][WSTACK];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    for (int64_t j = blockIdx.x * (int64_t)4 + wib; j < m; j += (int64_t)gridDim.x * 4) {
        const uint32_t qi = __ldg(ql + j);
        const int b = (int)nearest_leaf_warp(T, __ldg(qx + qi), __ldg(qy + qi), __ldg(qz + qi), s_stack[wib], lane);
        if (lane == 0) {
            bnear[j] = b;
            longs.add(T, j, b);
        }
    }
}

// A warp takes WALK_TICKET queries at a time from the queue (one counter for millions of short
// walks would be the bottleneck).
constexpr int WALK_TICKET = 4;

template <int STRAT>
__global__ void __launch_bounds__(128, 8) k_walk(DevTree T, RunPool P, int64_t m, const uint32_t *__restrict__ ql,
                                                 const double *__restrict__ qx, const double *__restrict__ qy,
                                                 const double *__restrict__ qz, int ticket, LongList longs,
                                                 unsigned long long *counter)
{
    __shared__ int s_walk[4][RUN_WALK_SMEM];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const double K = kernel_valid(T.kernel);
    const int scan = walk_scan<STRAT>(T);
    const int64_t nlong = longs.used();
    // tickets: the listed queries one by one, then all others, `ticket` at a time
    for (;;) {
        const int64_t t = next_query(counter, lane);
        const int64_t first = (t - nlong) * ticket;
        if (t >= nlong && first >= m) break;
        const int64_t end = t < nlong ? first + 1 : min(first + ticket, m);
        for (int64_t k = first; k < end; ++k) {
            const int64_t j = t < nlong ? (int64_t)longs.list[t] : k;
            if (nlong > 0 && t >= nlong && long_walk(T, P.bnear[j])) continue;   // walked already
            const uint32_t qi = __ldg(ql + j);
            walk_query<STRAT>(T, P, j, qi, __ldg(qx + qi), __ldg(qy + qi), __ldg(qz + qi), K, scan, s_walk[wib], lane);
        }
    }
}

// 8-bit pair order: the heavy queries (more than light_max accepted leaves), then the others, by
// descending size class (count_class) in each part; deferred queries last
__global__ void k_lpt_keys(int64_t m, const unsigned *__restrict__ qacc, const int *__restrict__ qflag,
                           unsigned light_max, uint32_t *keys, uint32_t *vals)
{
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
        const unsigned a = qacc[j];
        keys[j] = qflag[j] ? 255u : (a > light_max ? 127u : 255u) - count_class(a);
        vals[j] = (uint32_t)j;
    }
}

// queries (not deferred) with more than `light_max` accepted leaves, and the accepted pairs of
// the heavy and of the light queries (pairs[0], pairs[1]); one set of atomics per block
__global__ void k_count_heavy(int64_t m, const unsigned *__restrict__ qacc, const int *__restrict__ qflag,
                              unsigned light_max, unsigned *count, unsigned long long *pairs)
{
    __shared__ unsigned long long s_pairs[2];
    __shared__ unsigned s_count;
    if (threadIdx.x == 0) {
        s_pairs[0] = s_pairs[1] = 0ULL;
        s_count = 0u;
    }
    __syncthreads();
    unsigned c = 0;
    unsigned long long ph = 0, pl = 0;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
        if (qflag[j]) continue;
        const unsigned a = qacc[j];
        if (a > light_max) {
            ++c;
            ph += a;
        } else {
            pl += a;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        c += __shfl_down_sync(0xffffffffu, c, off);
        ph += __shfl_down_sync(0xffffffffu, ph, off);
        pl += __shfl_down_sync(0xffffffffu, pl, off);
    }
    if ((threadIdx.x & 31) == 0) {
        if (c) atomicAdd(&s_count, c);
        if (ph) atomicAdd(&s_pairs[0], ph);
        if (pl) atomicAdd(&s_pairs[1], pl);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_count) atomicAdd(count, s_count);
        if (s_pairs[0]) atomicAdd(pairs, s_pairs[0]);
        if (s_pairs[1]) atomicAdd(pairs + 1, s_pairs[1]);
    }
}

// plain schedule: a stable partition, heavy queries first, input order kept in each part
__global__ void k_heavy_keys(int64_t m, const unsigned *__restrict__ qacc, const int *__restrict__ qflag,
                             unsigned light_max, uint32_t *keys, uint32_t *vals)
{
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x) {
        keys[j] = (!qflag[j] && qacc[j] > light_max) ? 0u : 1u;
        vals[j] = (uint32_t)j;
    }
}

__global__ void k_iota(int64_t m, uint32_t *out)
{
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < m; j += (int64_t)gridDim.x * blockDim.x)
        out[j] = (uint32_t)j;
}

static int persistent_blocks(const void *kern, int bs)
{
    int dev = 0, sms = 148, per = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, bs, 0);
    return sms * (per > 0 ? per : 1);
}

cudaError_t launch_nearest_list(Handle *H, const DevTree &T, int64_t m, const uint32_t *ql, const double *qx,
                                const double *qy, const double *qz, int *bnear, bool listed)
{
    cudaError_t e;
    if (listed && ((e = H->long_list.reserve(sizeof(uint32_t) * long_cap(m))) || (e = H->long_count.reserve(sizeof(unsigned))) ||
                   (e = cudaMemsetAsync(H->long_count.p, 0, sizeof(unsigned), H->stream))))
        return e;
    const LongList L = long_list(H, m, listed);
    if (m <= nearest_warp_max(T.n))
        k_nearest_list_warp<<<grid_for(m, 4, 1 << 30), 128, 0, H->stream>>>(T, m, ql, qx, qy, qz, bnear, L);
    else k_nearest_list<<<grid_for(m, 128, 1 << 30), 128, 0, H->stream>>>(T, m, ql, qx, qy, qz, bnear, L);
    H->launches += 1;
    return cudaGetLastError();
}

template <int STRAT>
static void launch_walk_strat(Handle *H, const DevTree &T, const RunPool &P, int64_t m, const uint32_t *ql,
                              const double *qx, const double *qy, const double *qz, const LongList &longs,
                              unsigned long long *counter)
{
    const int warps = 4 * persistent_blocks((const void *)k_walk<STRAT>, 128);
    const int ticket = m >= (int64_t)warps * 16 ? WALK_TICKET : 1;
    k_walk<STRAT><<<grid_for(m, 4, warps / 4), 128, 0, H->stream>>>(T, P, m, ql, qx, qy, qz, ticket, longs, counter);
}

cudaError_t launch_walk(Handle *H, const DevTree &T, int strategy, const RunPool &P, int64_t m, const uint32_t *ql,
                        const double *qx, const double *qy, const double *qz, bool listed, unsigned long long *counter)
{
    if (m <= 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), H->stream);
    if (e) return e;
    const LongList L = long_list(H, m, listed);
    switch (strategy) {
    case GATHER: launch_walk_strat<GATHER>(H, T, P, m, ql, qx, qy, qz, L, counter); break;
    case SCATTER: launch_walk_strat<SCATTER>(H, T, P, m, ql, qx, qy, qz, L, counter); break;
    default: launch_walk_strat<SYMMETRIC>(H, T, P, m, ql, qx, qy, qz, L, counter); break;
    }
    H->launches += 1;
    return cudaGetLastError();
}

// pair order of a walked slice, heavy queries first, by descending size class unless `plain` (then the
// stable heavy/light partition of the walk order); the word after *P.n_deferred counts the heavy
// queries, and the accepted pairs of the heavy and the light queries are added to pairs[0], pairs[1]
cudaError_t launch_split_order(Handle *H, const RunPool &P, int64_t m, unsigned light_max, bool plain,
                               uint32_t **order, unsigned long long *pairs)
{
    cudaError_t e;
    if ((e = H->lpt_k.reserve(4 * m)) || (e = H->lpt_v.reserve(4 * m)) || (e = H->lpt_ka.reserve(4 * m)) ||
        (e = H->lpt_va.reserve(4 * m)))
        return e;
    uint32_t *k = H->lpt_k.as<uint32_t>(), *v = H->lpt_v.as<uint32_t>();
    if (plain) k_heavy_keys<<<grid_for(m, 256), 256, 0, H->stream>>>(m, P.qacc, P.qflag, light_max, k, v);
    else k_lpt_keys<<<grid_for(m, 256), 256, 0, H->stream>>>(m, P.qacc, P.qflag, light_max, k, v);
    H->launches += 1;
    if ((e = cudaGetLastError())) return e;
    if ((e = sort_pairs_u32(H, k, v, H->lpt_ka.as<uint32_t>(), H->lpt_va.as<uint32_t>(), m, 8, order))) return e;
    unsigned *cnt = reinterpret_cast<unsigned *>(P.n_deferred) + 1;
    if ((e = cudaMemsetAsync(cnt, 0, sizeof(unsigned), H->stream))) return e;
    k_count_heavy<<<grid_for(m, 256), 256, 0, H->stream>>>(m, P.qacc, P.qflag, light_max, cnt, pairs);
    H->launches += 1;
    return cudaGetLastError();
}

// the FP32C/FP64 split of a walked slice, left on the device: *count (zeroed here) = queries
// with more than light_max accepted leaves, pairs[0..1] += their pairs / the other queries' pairs
cudaError_t launch_count_heavy(Handle *H, const RunPool &P, int64_t m, unsigned light_max, unsigned *count,
                               unsigned long long *pairs)
{
    cudaError_t e = cudaMemsetAsync(count, 0, sizeof(unsigned), H->stream);
    if (e) return e;
    k_count_heavy<<<grid_for(m, 256), 256, 0, H->stream>>>(m, P.qacc, P.qflag, light_max, count, pairs);
    H->launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_iota(Handle *H, int64_t m, uint32_t *out)
{
    k_iota<<<grid_for(m, 256), 256, 0, H->stream>>>(m, out);
    H->launches += 1;
    return cudaGetLastError();
}

}  // namespace pb
