// pb_query.cu -- batched neighbour-search entry points on a built LBVH:
//   LBVH_find_nearest_h / LBVH_find_nearest (LinearBVHQueries.jl:79-140)
//   LBVH_query! (LinearBVHQueries.jl:183-211) as count + fill passes (CSR output)
// These are the bit-exact probes of the neighbour sets: the walk is the point path's (WarpWalk), so
// accepted leaves appear in ascending sorted-leaf order exactly as in the reference.  One thread
// per query with FP64 box tests used 4 % of the warp slots for 20,000 queries (4.2e6 particles):
// 15.6 ms; a warp per query 0.23 ms, and 0.21 ms for the closest leaf (a nearest search of its own).
// Many queries with few leaves each take k_query_short first.
#include "pb_internal.h"
#include "pb_walk_impl.cuh"

namespace pb {

__global__ void k_nearest(DevTree T, int64_t nq, const double *__restrict__ qx, const double *__restrict__ qy,
                          const double *__restrict__ qz, double *h_out, int64_t *idx_out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nq; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t b = nearest_leaf(T, qx[i], qy[i], qz[i]);
        if (h_out) h_out[i] = b < 0 ? __longlong_as_double(0x7ff8000000000000LL) : T.leaf[b].w;
        if (idx_out) idx_out[i] = b;
    }
}

__global__ void __launch_bounds__(128) k_nearest_warp(DevTree T, int64_t nq, const double *__restrict__ qx,
                                                      const double *__restrict__ qy, const double *__restrict__ qz,
                                                      double *h_out, int64_t *idx_out)
{
    __shared__ int s_stack[4][WSTACK];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    for (int64_t i = blockIdx.x * (int64_t)4 + wib; i < nq; i += (int64_t)gridDim.x * 4) {
        const int64_t b = nearest_leaf_warp(T, __ldg(qx + i), __ldg(qy + i), __ldg(qz + i), s_stack[wib], lane);
        if (lane == 0) {
            if (h_out) h_out[i] = b < 0 ? __longlong_as_double(0x7ff8000000000000LL) : T.leaf[b].w;
            if (idx_out) idx_out[i] = b;
        }
    }
}

// A query's accepted leaves, counted and (with a pool) listed in DFS order; a list longer than its
// `cap` flags ST_POOL and is cut there.
struct ListSink {
    int64_t *pool;   // NULL: count only
    int64_t cap;
    int *status;
    int lane;
    int64_t count = 0;

    __device__ __forceinline__ bool append(unsigned done, int lo, int hi)
    {
        const int len = (done >> lane) & 1u ? hi - lo + 1 : 0;
        if (!pool) {
            count += __reduce_add_sync(0xffffffffu, len);   // disjoint ranges: at most n <= 2^30
            return true;
        }
        int inc = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        const int tot = __shfl_sync(0xffffffffu, inc, 31);
        if (len == 1 && count + inc - 1 < cap) pool[count + inc - 1] = lo;
        for (unsigned big = __ballot_sync(0xffffffffu, len > 1); big; big &= big - 1) {
            const int l = __ffs(big) - 1;
            const int first = __shfl_sync(0xffffffffu, lo, l), n = __shfl_sync(0xffffffffu, len, l);
            const int64_t at = count + __shfl_sync(0xffffffffu, inc, l) - n;
            for (int i = lane; i < n; i += 32)
                if (at + i < cap) pool[at + i] = first + i;
        }
        if (count + tot > cap && lane == 0) flag(status, ST_POOL);
        count += tot;
        return true;
    }
};

// gather predicate d2 <= radius^2 (LinearBVHTraversalMacros.jl:26-108), one warp per query (WarpWalk);
// pool == nullptr counts only.  rest: the number of queries and the queries to take; NULL: all
__global__ void __launch_bounds__(128, 8) k_query(DevTree T, int64_t nq, const double *__restrict__ qx,
                                                  const double *__restrict__ qy, const double *__restrict__ qz,
                                                  const double *__restrict__ radius,
                                                  const int64_t *__restrict__ offsets, int64_t *counts, int64_t *pool,
                                                  const uint32_t *__restrict__ rest)
{
    __shared__ int s_walk[4][WALK_SMEM];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t todo = rest ? (int64_t)__ldg(rest) : nq;
    for (int64_t k = blockIdx.x * (int64_t)4 + wib; k < todo; k += (int64_t)gridDim.x * 4) {
        const int64_t i = rest ? (int64_t)__ldg(rest + 1 + k) : k;
        const double px = __ldg(qx + i), py = __ldg(qy + i), pz = __ldg(qz + i), r = __ldg(radius + i);
        const double r2 = __dmul_rn(r, r);
        const int64_t base = pool ? __ldg(offsets + i) : 0;
        ListSink S{pool ? pool + base : nullptr, pool ? __ldg(offsets + i + 1) - base : 0, T.status, lane};
        if (T.root == 0) {
            if (d2_point(px, py, pz, ldg4(T.leaf)) <= r2) S.append(1u, 0, 0);
        } else {
            WarpWalk<GATHER, ListSink> W(T, S, s_walk[wib], lane, WALK_SCAN);
            W.run(px, py, pz, 0.0, r2);
        }
        if (counts && lane == 0) counts[i] = S.count;
    }
}

// From QUERY_SHORT_MIN queries on a thread takes up to QUERY_STEPS nodes and leaves of its query's
// depth-first walk first; a query that is not done then is listed in `rest` and taken by a warp (k_query,
// which writes the same leaves again, and k_closest_rest).  A query of few leaves needs no more, and a warp's
// rounds would be mostly idle on it; for others the thread's steps come on top.  Counts on 1e6 particles, a
// thread for the whole walk / a warp / this: 100,000 points of 0.4 leaves each 0.45 / 0.63 / 0.36 ms, of 15 leaves
// 1.31 / 0.67 / 0.48, of 339 leaves 8.7 / 0.91 / 0.98; 40,000 points 0.30 / 0.31 / 0.23, 1.09 / 0.33 / 0.28 and
// 8.2 / 0.46 / 0.53; 20,000 points 0.24 / 0.17 / 0.16, 0.98 / 0.18 / 0.19 and 8.0 / 0.25 / 0.35.  Steps of 64 / 96 /
// 128 / 192 at 100,000 points: 0.38 / 0.37 / 0.41 / 0.43 (0.4 leaves) and 0.54 / 0.48 / 0.49 / 0.50 (15 leaves).
constexpr int QUERY_STEPS = 96;
constexpr int64_t QUERY_SHORT_MIN = 24576;

__global__ void __launch_bounds__(128) k_query_short(DevTree T, int64_t nq, const double *__restrict__ qx,
                                                     const double *__restrict__ qy, const double *__restrict__ qz,
                                                     const double *__restrict__ radius,
                                                     const int64_t *__restrict__ offsets, int64_t *counts, int64_t *pool,
                                                     int64_t *nearest, double *nearest_d2, uint32_t *rest)
{
    const int n = (int)T.n;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nq; i += (int64_t)gridDim.x * blockDim.x) {
        const double px = __ldg(qx + i), py = __ldg(qy + i), pz = __ldg(qz + i), r = __ldg(radius + i);
        const double r2 = __dmul_rn(r, r);
        const QBox q = make_qbox(px, py, pz);
        const float r2_up = __double2float_ru(r2);
        const int64_t base = pool ? __ldg(offsets + i) : 0, cap = pool ? __ldg(offsets + i + 1) - base : 0;
        int node = T.root, ci = -1;
        int64_t cnt = 0;
        double cd = INFINITY;
        for (int s = 0; s < QUERY_STEPS && node != 0; ++s) {
            if (node >= n) {
                const int b = node - n;
                const double d2 = d2_point(px, py, pz, ldg4(T.leaf + b));
                node = __ldg(T.leaf_escape + b);
                if (d2 <= r2) {
                    if (cnt < cap) pool[base + cnt] = b;
                    ++cnt;
                    if (d2 < cd) {
                        cd = d2;
                        ci = b;
                    }
                }
            } else {
                const NodeF nd = load_node(T.node + (node - 1));
                node = node_pruned<GATHER>(T, nd, node, q, 0.f, r2_up) ? nd.escape : nd.left;
            }
        }
        if (node != 0 || T.root == 0) {
            rest[1 + atomicAdd(rest, 1u)] = (uint32_t)i;
            continue;
        }
        if (pool && cnt > 0 && cnt > cap) flag(T.status, ST_POOL);   // an empty list fits any offsets
        if (counts) counts[i] = cnt;
        if (nearest) nearest[i] = ci;
        if (nearest_d2) nearest_d2[i] = cd;
    }
}

// the closest accepted leaf of a query: the nearest leaf of all within the radius.  It is the
// first strictly closer one in DFS order (LinearBVHQueries.jl:33-39,196-203): nearest[i] its index (-1
// if none), nearest_d2[i] its squared distance (+Inf if none).
__device__ __forceinline__ void store_closest(const DevTree &T, int64_t i, int64_t b, double px, double py, double pz,
                                              int64_t *nearest, double *nearest_d2)
{
    if (nearest) nearest[i] = b;
    if (nearest_d2) nearest_d2[i] = b < 0 ? INFINITY : d2_point(px, py, pz, ldg4(T.leaf + b));
}

template <typename REST>
__device__ __forceinline__ void closest_by_warps(const DevTree &T, int64_t todo, const double *__restrict__ qx,
                                                 const double *__restrict__ qy, const double *__restrict__ qz,
                                                 const double *__restrict__ radius, int64_t *nearest, double *nearest_d2,
                                                 REST query)
{
    __shared__ int s_stack[4][WSTACK];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    for (int64_t k = blockIdx.x * (int64_t)4 + wib; k < todo; k += (int64_t)gridDim.x * 4) {
        const int64_t i = query(k);
        const double px = __ldg(qx + i), py = __ldg(qy + i), pz = __ldg(qz + i), r = __ldg(radius + i);
        const int64_t b = nearest_leaf_warp<true>(T, px, py, pz, s_stack[wib], lane, __dmul_rn(r, r));
        if (lane == 0) store_closest(T, i, b, px, py, pz, nearest, nearest_d2);
    }
}

__global__ void __launch_bounds__(128) k_closest_warp(DevTree T, int64_t nq, const double *__restrict__ qx,
                                                      const double *__restrict__ qy, const double *__restrict__ qz,
                                                      const double *__restrict__ radius, int64_t *nearest,
                                                      double *nearest_d2)
{
    closest_by_warps(T, nq, qx, qy, qz, radius, nearest, nearest_d2, [](int64_t k) { return k; });
}

// the queries that k_query_short left: a warp each for up to NEAREST_WARP_MAX of them, a thread each for more
__global__ void __launch_bounds__(128) k_closest_rest(DevTree T, const double *__restrict__ qx,
                                                      const double *__restrict__ qy, const double *__restrict__ qz,
                                                      const double *__restrict__ radius, int64_t *nearest,
                                                      double *nearest_d2, const uint32_t *__restrict__ rest)
{
    const int64_t todo = __ldg(rest);
    if (todo <= NEAREST_WARP_MAX) {
        closest_by_warps(T, todo, qx, qy, qz, radius, nearest, nearest_d2, [&](int64_t k) { return (int64_t)__ldg(rest + 1 + k); });
        return;
    }
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < todo; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = __ldg(rest + 1 + k);
        const double px = __ldg(qx + i), py = __ldg(qy + i), pz = __ldg(qz + i), r = __ldg(radius + i);
        store_closest(T, i, nearest_leaf<true>(T, px, py, pz, __dmul_rn(r, r)), px, py, pz, nearest, nearest_d2);
    }
}

// Event counts of the reference algorithm itself (leaf size 1, Karras tree, left-first DFS,
// FP64 boxes and the reference's pruning tests, LinearBVHTraversalMacros.jl:26-371): per
// query [nearest-pass internal visits, nearest-pass leaf tests, main-pass internal visits,
// main-pass leaf tests, accepted neighbours].  Used for the algorithmic-bytes roofline model
// and as exact per-query work labels.
struct Tree64 {
    const double *bmin, *bmax, *hmax;
};

__device__ __forceinline__ double d2_box64(const Tree64 &B, int64_t nin, int64_t i0, double px, double py, double pz)
{
    double p[3] = {px, py, pz};
    double s = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double a = B.bmin[d * nin + i0], b = B.bmax[d * nin + i0];
        double t = p[d] < a ? __dsub_rn(a, p[d]) : (p[d] > b ? __dsub_rn(p[d], b) : 0.0);
        s = __dadd_rn(s, __dmul_rn(t, t));
    }
    return s;
}

__global__ void k_stats(DevTree T, Tree64 B, int strategy, int64_t nq, const double *__restrict__ qx,
                        const double *__restrict__ qy, const double *__restrict__ qz, int64_t *stats)
{
    const int64_t n = T.n, nin = n - 1;
    const double K = kernel_valid(T.kernel);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nq; i += (int64_t)gridDim.x * blockDim.x) {
        double px = qx[i], py = qy[i], pz = qz[i];
        int64_t nv = 0, nl = 0, mv = 0, ml = 0, acc = 0;
        int64_t guard, limit = 4 * n + 64;
        double ha = 0.0;
        if (strategy != SCATTER) {
            double best = INFINITY;
            int64_t bi = -1;
            if (T.root == 0) {
                double d2 = d2_point(px, py, pz, ldg4(T.leaf));
                ++nl;
                if (d2 < best) bi = 0;
            } else {
                int node = T.root;
                guard = 0;
                while (node != 0) {
                    if (++guard > limit) { flag(T.status, ST_TRAVERSAL); break; }
                    if (node >= n) {
                        int64_t b = node - n;
                        double d2 = d2_point(px, py, pz, ldg4(T.leaf + b));
                        ++nl;
                        if (d2 < best) { best = d2; bi = b; }
                        node = __ldg(T.leaf_escape + b);
                    } else {
                        ++nv;
                        NodeF nd = load_node(T.node + (node - 1));
                        node = (d2_box64(B, nin, node - 1, px, py, pz) > best) ? nd.escape : nd.left;
                    }
                }
            }
            ha = bi < 0 ? __longlong_as_double(0x7ff8000000000000LL) : T.leaf[bi].w;
        }
        double ra = __dmul_rn(K, ha), r2a = __dmul_rn(ra, ra);
        int node = T.root;
        int64_t bi = 0;
        bool brute = (node == 0);
        guard = 0;
        while (brute ? (bi < n) : (node != 0)) {
            if (++guard > limit) { flag(T.status, ST_TRAVERSAL); break; }
            if (brute || node >= n) {
                int64_t b = brute ? bi++ : (int64_t)(node - n);
                double4 L = ldg4(T.leaf + b);
                double r = __dmul_rn(K, L.w), rr = __dmul_rn(r, r);
                double r2 = strategy == GATHER ? r2a : (strategy == SCATTER ? rr : (r2a > rr ? r2a : rr));
                ++ml;
                if (d2_point(px, py, pz, L) <= r2) ++acc;
                if (!brute) node = __ldg(T.leaf_escape + b);
            } else {
                ++mv;
                NodeF nd = load_node(T.node + (node - 1));
                double r = __dmul_rn(K, B.hmax[node - 1]), rr = __dmul_rn(r, r);
                double r2 = strategy == GATHER ? r2a : (strategy == SCATTER ? rr : (r2a > rr ? r2a : rr));
                node = (d2_box64(B, nin, node - 1, px, py, pz) > r2) ? nd.escape : nd.left;
            }
        }
        int64_t *s = stats + 5 * i;
        s[0] = nv; s[1] = nl; s[2] = mv; s[3] = ml; s[4] = acc;
    }
}

cudaError_t launch_stats(Handle *H, const DevTree &T, int strategy, int64_t nq, const double *qx, const double *qy,
                         const double *qz, int64_t *stats)
{
    Tree64 B{H->bmin64.as<double>(), H->bmax64.as<double>(), H->hmax64.as<double>()};
    k_stats<<<grid_for(nq, 128, 1 << 30), 128, 0, H->stream>>>(T, B, strategy, nq, qx, qy, qz, stats);
    H->launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_nearest(Handle *H, const DevTree &T, int64_t nq, const double *qx, const double *qy,
                           const double *qz, double *h_out, int64_t *idx_out)
{
    if (nq <= nearest_warp_max(T.n))
        k_nearest_warp<<<grid_for(nq, 4, 1 << 30), 128, 0, H->stream>>>(T, nq, qx, qy, qz, h_out, idx_out);
    else k_nearest<<<grid_for(nq, 128, 1 << 30), 128, 0, H->stream>>>(T, nq, qx, qy, qz, h_out, idx_out);
    H->launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_query(Handle *H, const DevTree &T, int64_t nq, const double *qx, const double *qy,
                         const double *qz, const double *radius, const int64_t *offsets, int64_t *counts,
                         int64_t *pool, int64_t *nearest, double *nearest_d2)
{
    uint32_t *rest = nullptr;   // what is left after the short queries, if there are many
    if (nq >= QUERY_SHORT_MIN && nq < 0xffffffffLL) {
        cudaError_t e = H->q_rest.reserve(sizeof(uint32_t) * (nq + 1));
        if (!e) e = cudaMemsetAsync(H->q_rest.p, 0, sizeof(uint32_t), H->stream);
        if (e) return e;
        rest = H->q_rest.as<uint32_t>();
        k_query_short<<<grid_for(nq, 128, 1 << 30), 128, 0, H->stream>>>(T, nq, qx, qy, qz, radius, offsets, counts, pool,
                                                                         nearest, nearest_d2, rest);
        H->launches += 1;
    }
    int sms = 148, per = 1;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, H->device);
    if (counts || pool) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_query, 128, 0);
        k_query<<<grid_for(nq, 4, (rest ? 1 : 4) * sms * (per > 0 ? per : 1)), 128, 0, H->stream>>>(
            T, nq, qx, qy, qz, radius, offsets, counts, pool, rest);
        H->launches += 1;
    }
    if (nearest || nearest_d2) {
        if (rest) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_closest_rest, 128, 0);
            k_closest_rest<<<sms * (per > 0 ? per : 1), 128, 0, H->stream>>>(T, qx, qy, qz, radius, nearest, nearest_d2, rest);
        } else {
            k_closest_warp<<<grid_for(nq, 4, 1 << 30), 128, 0, H->stream>>>(T, nq, qx, qy, qz, radius, nearest, nearest_d2);
        }
        H->launches += 1;
    }
    return cudaGetLastError();
}

// Sample points of a structured grid, generated on the device (coordinate_grid + flatten,
// StructuredGrid.jl:126-204, transform.jl:53-66): column-major linear order, the first axis
// fastest; coord 0 Cartesian (a0, a1, a2), 2 cylindrical (s cos phi, s sin phi, z), 3 spherical
// (r sin(theta) cos(phi), r sin(theta) sin(phi), r cos(theta)) with the host's operation order.
__global__ void k_grid_points(int coord, const double *__restrict__ a0, int64_t n0, const double *__restrict__ a1,
                              int64_t n1, const double *__restrict__ a2, int64_t n2, double *x, double *y, double *z)
{
    const int64_t n = n0 * n1 * n2;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i0 = i % n0, i1 = (i / n0) % n1, i2 = i / (n0 * n1);
        const double u = a0[i0], v = a1[i1], w = a2[i2];
        if (coord == 2) {
            x[i] = __dmul_rn(u, cos(v));
            y[i] = __dmul_rn(u, sin(v));
            z[i] = w;
        } else if (coord == 3) {
            const double st = sin(w);
            x[i] = __dmul_rn(__dmul_rn(u, st), cos(v));
            y[i] = __dmul_rn(__dmul_rn(u, st), sin(v));
            z[i] = __dmul_rn(u, cos(w));
        } else {
            x[i] = u;
            y[i] = v;
            z[i] = w;
        }
    }
}

cudaError_t launch_grid_points(Handle *H, int coord, const double *a0, int64_t n0, const double *a1, int64_t n1,
                               const double *a2, int64_t n2, double *x, double *y, double *z)
{
    k_grid_points<<<grid_for(n0 * n1 * n2, 256), 256, 0, H->stream>>>(coord, a0, n0, a1, n1, a2, n2, x, y, z);
    H->launches += 1;
    return cudaGetLastError();
}

// Lines of an image (LineSamples of a column-density map): line k = i + n0 * j starts at
// (c + a0[i] e1) + a1[j] e2 and runs along d; no FMA, so the values equal the host's
// per-component expression.
__global__ void k_line_image(const double *__restrict__ a0, int64_t n0, const double *__restrict__ a1, int64_t n1,
                             LineFrame F, double *ox, double *oy, double *oz, double *dx, double *dy, double *dz)
{
    const int64_t n = n0 * n1;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const double u = a0[k % n0], v = a1[k / n0];
        ox[k] = __dadd_rn(__dadd_rn(F.c[0], __dmul_rn(u, F.e1[0])), __dmul_rn(v, F.e2[0]));
        oy[k] = __dadd_rn(__dadd_rn(F.c[1], __dmul_rn(u, F.e1[1])), __dmul_rn(v, F.e2[1]));
        oz[k] = __dadd_rn(__dadd_rn(F.c[2], __dmul_rn(u, F.e1[2])), __dmul_rn(v, F.e2[2]));
        dx[k] = F.d[0];
        dy[k] = F.d[1];
        dz[k] = F.d[2];
    }
}

cudaError_t launch_line_image(Handle *H, const double *a0, int64_t n0, const double *a1, int64_t n1, const LineFrame &F,
                              double *ox, double *oy, double *oz, double *dx, double *dy, double *dz)
{
    k_line_image<<<grid_for(n0 * n1, 256), 256, 0, H->stream>>>(a0, n0, a1, n1, F, ox, oy, oz, dx, dy, dz);
    H->launches += 1;
    return cudaGetLastError();
}

}  // namespace pb
