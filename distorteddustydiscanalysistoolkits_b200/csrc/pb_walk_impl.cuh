// pb_walk_impl.cuh -- the walk of the two-phase point path: a warp walks one query's tree and writes
// its accepted leaves, merged into runs of consecutive sorted indices, to extents of a shared pool.
// Shared by the walk kernels (pb_walk.cu) and the batched walk (pb_batch.cu).
//
// The warp keeps a stack of tree entries whose top is the next one in DFS order.  Each round its
// lanes take the top 32: a subtree that the query does not reach is dropped; one inside the
// query's radius, one of few leaves (WALK_SCAN) and a leaf stay; any other is replaced by its two
// children.  The entries that stay and come before the first one opened are the next ones in DFS
// order: they collect until there are 32, then their leaves are tested 32 at a time (those of a
// subtree inside the radius pass as a whole) and what is accepted is appended to the runs.  The node
// decisions are next_item's (node_pruned, box_upper) and the leaf test is exact, so the accepted set
// and its order are the reference's.
//
// A thread per (query, subtree) item, as before, kept 6.7 of 32 lanes busy (paths of different length,
// and leaf, prune, accept and emit steps in turn) and needed a cut of the tree, a prefilter, a sorted
// work list and 64 item records a query; here the 32 lanes test 32 entries of one query.  Walk phase
// before and now: 2.1e6 particles and 4.2e6 points 133 -> 102 ms, 131,072 particles on 64^3 points
// 3.9 -> 2.5 ms, 1e5 tracers (scatter) 1.43 -> 0.72 ms.
#pragma once
#include "pb_interp_impl.cuh"

namespace pb {

// Leaves of a subtree that are tested instead of opening it: a test is a 32-byte load and ten FP64
// operations, batched over the lanes, an opening two more box tests.  Walk phase at 1 / 4 / 8 / 16 / 32:
// 2.1e6 particles, 4.2e6 points 147 / 119 / 107 / 102 / 109 ms; 131,072 particles, 64^3 points 3.2 / 2.7 /
// 2.5 / 2.5 / 2.6; scatter, 1e5 tracers 0.82 / 0.72 / 0.71 / 0.72 / 0.76.
// A scanned leaf skips the tests of the nodes between it and the subtree; they could only have cut it
// off where its radius exceeds theirs, that is where an h is negative: such trees are opened to the leaves.
constexpr int WALK_SCAN = 16;
template <int STRAT>
__device__ __forceinline__ int walk_scan(const DevTree &T)
{
    return STRAT != GATHER && (__ldg(T.odd) & ODD_NEGATIVE_H) ? 1 : WALK_SCAN;
}
constexpr int WSTACK = 512;   // entries; taken one at a time above WSTACK - 160, where a round adds at most one
constexpr int WALK_SMEM = WSTACK + 128;       // ints of shared memory per warp of a WarpWalk
constexpr int RUN_WALK_SMEM = WALK_SMEM + 128;   // and of one into a RunSink

// where a walk's accepted ranges go: a query's runs in the shared pool
struct RunSink {
    const RunPool &P;
    int *rlo, *rhi;           // 64 runs not written yet, the last one still open
    int lane;
    int cnt = 0;              // runs in rlo/rhi
    int first = -1, cur = -1, nruns = 0;
    int nacc = 0;             // this lane's share of the accepted leaves

    __device__ __forceinline__ RunSink(const RunPool &p, int *smem, int l) : P(p), rlo(smem), rhi(smem + 64), lane(l) {}

    // writes the first k <= 32 runs as one chunk; false if the pool is full
    __device__ __forceinline__ bool flush(int k)
    {
        nruns += k;
        if (P.count_only) return true;
        if (cur < 0 || (cur & (RUN_EXTENT - 1)) == RUN_EXTENT - 1) {
            unsigned long long c = 0;
            if (lane == 0) c = atomicAdd(P.used, (unsigned long long)RUN_EXTENT);
            c = __shfl_sync(0xffffffffu, c, 0);
            if (c + RUN_EXTENT > P.cap) return false;
            if (cur < 0) first = (int)c;
            else if (lane == 0) P.next[cur] = (int)c;
            cur = (int)c;
        } else {
            ++cur;
        }
        if (lane < k)
            P.runs[(int64_t)cur * RUN_CHUNK + lane] = make_uint2((unsigned)rlo[lane], (unsigned)(rhi[lane] - rlo[lane] + 1));
        return true;
    }
    // appends the ranges [lo, hi] of the lanes of `done` (at least one), in lane order; false if the
    // pool is full
    __device__ __forceinline__ bool append(unsigned done, int lo, int hi)
    {
        const unsigned self = 1u << lane, below = self - 1u;
        const bool on = done & self;
        const unsigned before = done & below, after = done & ~(below | self);
        const int prev = __shfl_sync(0xffffffffu, hi, before ? 31 - __clz(before) : 0);
        const int open = cnt > 0 ? rhi[cnt - 1] : -2;
        const bool start = on && lo != (before ? prev : open) + 1;
        const unsigned starts = __ballot_sync(0xffffffffu, start);
        const int r = cnt - 1 + __popc(starts & (below | self));   // the run this range belongs to
        __syncwarp();   // every lane has read the open run
        if (start) rlo[r] = lo;
        if (on && (!after || ((starts >> (__ffs(after) - 1)) & 1u))) rhi[r] = hi;   // the run's last range
        if (on) nacc += hi - lo + 1;
        cnt += __popc(starts);
        __syncwarp();
        if (cnt > 32) {
            if (!flush(32)) return false;
            cnt -= 32;
            const int a = rlo[32 + lane], b = rhi[32 + lane];
            __syncwarp();
            rlo[lane] = a;
            rhi[lane] = b;
            __syncwarp();
        }
        return true;
    }
    __device__ __forceinline__ bool finish() { return cnt == 0 || flush(cnt); }
};

template <int STRAT, typename SINK>
struct WarpWalk {
    const DevTree &T;
    SINK &sink;
    int *stack;               // WSTACK entries
    int *clo, *clen;          // 64 candidates in DFS order: first leaf, and the number of leaves to be tested
                              // or minus the number of leaves accepted as a whole
    int lane;
    int scan;                 // walk_scan of the tree
    int cand = 0;             // candidates

    __device__ __forceinline__ WarpWalk(const DevTree &t, SINK &s, int *smem, int l, int sc)
        : T(t), sink(s), stack(smem), clo(smem + WSTACK), clen(smem + WSTACK + 64), lane(l), scan(sc)
    {
    }
    // tests the leaves of the first k <= 32 candidates, passes on what is accepted and removes them;
    // false if the sink refused a range
    __device__ __forceinline__ bool settle(int k, double px, double py, double pz, double K, double r2a)
    {
        const int c0 = lane < k ? clo[lane] : 0, len = lane < k ? clen[lane] : 0;
        const int width = len < 0 ? 1 : len;   // positions: one per leaf to be tested, one per accepted range
        int inc = width;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        const int tot = __shfl_sync(0xffffffffu, inc, 31), ex = inc - width;
        for (int tb = 0; tb < tot; tb += 32) {
            // the candidate of position tb + lane: that of position tb plus the candidates that start
            // between them
            const int r0 = __popc(__ballot_sync(0xffffffffu, inc <= tb)), s = ex - tb;
            const unsigned starts = __reduce_or_sync(0xffffffffu, s > 0 && s < 32 && width > 0 ? 1u << s : 0u);
            const int r = (r0 + __popc(starts & (0xffffffffu >> (31 - lane)))) & 31;
            const int l = __shfl_sync(0xffffffffu, c0, r), n = __shfl_sync(0xffffffffu, len, r),
                      e = __shfl_sync(0xffffffffu, ex, r);
            bool on = tb + lane < tot;
            int lo = l, hi = l - n - 1;
            if (on && n > 0) {
                lo = hi = l + (tb + lane - e);
                const double4 L = ldg4(T.leaf + lo);
                double r2;
                if (STRAT == GATHER) r2 = r2a;
                else {
                    const double rad = __dmul_rn(K, L.w);
                    const double rr = __dmul_rn(rad, rad);
                    r2 = STRAT == SCATTER ? rr : (r2a > rr ? r2a : rr);
                }
                on = d2_point(px, py, pz, L) <= r2;
            }
            const unsigned done = __ballot_sync(0xffffffffu, on);
            if (done && !sink.append(done, lo, hi)) return false;
        }
        __syncwarp();
        cand -= k;
        if (cand > 0) {
            const int a = clo[32 + lane], b = clen[32 + lane];
            __syncwarp();
            clo[lane] = a;
            clen[lane] = b;
        }
        __syncwarp();
        return true;
    }
    // the walk from the root; false if the sink refused a range
    __device__ __forceinline__ bool run(double px, double py, double pz, double K, double r2a)
    {
        const int n = (int)T.n;
        const QBox q = make_qbox(px, py, pz);
        const float Kf = (float)K;
        const float r2a_up = __double2float_ru(r2a);
        const float bulk_lim = __fmul_rd(__double2float_rd(r2a), MARGIN_DN);
        const unsigned below = (1u << lane) - 1u;
        const unsigned limit = 2u * (unsigned)n + 64u;   // every round settles or opens at least one entry
        unsigned guard = 0;
        int size = 1;
        if (lane == 0) stack[0] = T.root;
        __syncwarp();
        while (size > 0) {
            if (++guard > limit || size > WSTACK - 2) {
                flag(T.status, ST_TRAVERSAL);
                break;
            }
            const int k = size > WSTACK - 160 ? 1 : (size < 32 ? size : 32);
            int c = 0, e0 = 0, e1 = 0, lo = 0, len = 1;   // c: entries that replace this one
            if (lane < k) {
                e0 = stack[size - 1 - lane];
                c = 1;
                lo = e0 - n;
                if (e0 < n) {
                    const int id = e0;
                    const int2 rg = __ldg(T.range + (id - 1));
                    const NodeF nd = load_node(T.node + (id - 1));
                    lo = rg.x;
                    len = rg.y - rg.x + 1;
                    if (node_pruned<STRAT>(T, nd, id, q, Kf, r2a_up)) {
                        c = 0;
                    } else if (STRAT != SCATTER && box_upper(q, nd) <= bulk_lim) {
                        len = -len;
                    } else if (len > scan) {
                        // the children of a Karras node meet at the split, which the left child's id
                        // gives; a child of one leaf is that leaf
                        c = 2;
                        e0 = nd.left;
                        const int split = nd.left >= n ? nd.left - (n - 1) : nd.left;   // 1-based
                        e1 = split == rg.y ? n + rg.y : split + 1;
                    }
                }
            }
            __syncwarp();
            const unsigned open = __ballot_sync(0xffffffffu, c == 2), stay = __ballot_sync(0xffffffffu, c >= 1);
            const unsigned pre = open ? (open & -open) - 1u : 0xffffffffu;   // lanes before the first open one
            const unsigned done = stay & pre, kept = stay & ~pre;
            size += __popc(kept) + __popc(open) - k;
            if (c >= 1) {
                if ((done >> lane) & 1u) {
                    const int at = cand + __popc(done & below);
                    clo[at] = lo;
                    clen[at] = len;
                } else {
                    const int at = size - 1 - __popc(kept & below) - __popc(open & below);
                    stack[at] = e0;
                    if (c == 2) stack[at - 1] = e1;
                }
            }
            cand += __popc(done);
            __syncwarp();
            if (cand >= 32 && !settle(32, px, py, pz, K, r2a)) return false;
        }
        return cand == 0 || settle(cand, px, py, pz, K, r2a);
    }
};

// nearest_leaf by a warp: the 32 leaves around the point's place in the Morton order give a first
// distance, then the lanes take 32 tree entries a round and keep those that may hold a leaf at most
// that far.  The result is nearest_leaf's: the least squared distance and, among equal ones, the
// smallest sorted index; WITHIN as there.  Every lane of the warp calls it; smem holds WSTACK ints.
template <bool WITHIN = false>
__device__ __forceinline__ int64_t nearest_leaf_warp(const DevTree &T, double px, double py, double pz, int *stack,
                                                     int lane, double within = INFINITY)
{
    const int n = (int)T.n;
    double best = INFINITY;
    int bi = -1;
    if (WITHIN && within < INFINITY) {
        best = within;
        bi = n;
    }
    if (WITHIN && !(within >= 0.0)) return -1;   // NaN
    // the warp's least (d2, index) over its lanes' candidates and the best so far
    auto take = [&](double d2, int b) {
        if (!__any_sync(0xffffffffu, d2 < best || (d2 == best && b < bi))) return;
        if (!(d2 < best || (d2 == best && b < bi))) { d2 = best; b = bi; }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double v = __shfl_xor_sync(0xffffffffu, d2, o);
            const int vb = __shfl_xor_sync(0xffffffffu, b, o);
            if (v < d2 || (v == d2 && vb < b)) { d2 = v; b = vb; }
        }
        best = d2;
        bi = b;
    };
    if (T.root == 0) {
        take(lane == 0 ? d2_point(px, py, pz, ldg4(T.leaf)) : INFINITY, 0);
        return !WITHIN || bi < n ? bi : -1;
    }
    uint64_t code = 0;
    {
        const double p[3] = {px, py, pz};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double f = T.qp->flat[d] ? 0.5 : (p[d] - T.qp->vmin[d]) * T.qp->inv[d];
            const uint64_t c = f > 0.0 ? (uint64_t)(fmin(f, 1.0) * 2097151.0) : 0;   // NaN: 0
            code |= expand_bits3(c) << (2 - d);
        }
    }
    int lo = 0, hi = n;
    while (hi - lo > 32) {
        const int step = (hi - lo + 31) / 32, t = lo + lane * step;
        const int k = __popc(__ballot_sync(0xffffffffu, t < hi && __ldg(T.codes + t) < code));
        hi = min(hi, lo + max(k, 1) * step);
        lo = lo + (k > 0 ? (k - 1) * step : 0);
    }
    {
        const int b = max(0, min((lo + hi) / 2 - 16, n - 32)) + lane;
        take(b < n ? d2_point(px, py, pz, ldg4(T.leaf + b)) : INFINITY, b);
    }
    const QBox q = make_qbox(px, py, pz);
    const unsigned below = (1u << lane) - 1u;
    const unsigned limit = 2u * (unsigned)n + 64u;
    unsigned guard = 0;
    int size = 1;
    __syncwarp();
    if (lane == 0) stack[0] = T.root;
    __syncwarp();
    while (size > 0) {
        if (++guard > limit || size > WSTACK - 2) {
            flag(T.status, ST_TRAVERSAL);
            break;
        }
        const int k = size > WSTACK - 160 ? 1 : (size < 32 ? size : 32);
        // a subtree is skipped only when its lower bound exceeds the best distance by the margin
        const float lim = __fmul_ru(__double2float_ru(best), MARGIN_UP);
        int e0 = 0, e1 = 0, b = -1;
        bool open = false;
        if (lane < k) {
            const int e = stack[size - 1 - lane];
            if (e >= n) {
                b = e - n;
            } else {
                const NodeF nd = load_node(T.node + (e - 1));
                open = !(box_lower(q, nd) > lim);
                const int2 rg = __ldg(T.range + (e - 1));
                e0 = nd.left;
                const int split = nd.left >= n ? nd.left - (n - 1) : nd.left;   // 1-based
                e1 = split == rg.y ? n + rg.y : split + 1;
            }
        }
        take(b >= 0 ? d2_point(px, py, pz, ldg4(T.leaf + b)) : INFINITY, b >= 0 ? b : n);
        const unsigned o = __ballot_sync(0xffffffffu, open);
        size += 2 * __popc(o) - k;
        if (open) {
            const int at = size - 1 - 2 * __popc(o & below);
            stack[at] = e0;
            stack[at - 1] = e1;
        }
        __syncwarp();
    }
    return !WITHIN || bi < n ? bi : -1;
}

// The walk of the j-th listed query (sample point qi at px, py, pz; nearest sorted leaf P.bnear[j]):
// its run list, its number of accepted leaves, and whether the pool was full (the query is then
// listed as deferred).  scan is walk_scan of the tree.  Every lane of the warp calls it; smem holds RUN_WALK_SMEM ints.
template <int STRAT>
__device__ __forceinline__ void walk_query(const DevTree &T, const RunPool &P, int64_t j, uint32_t qi, double px,
                                           double py, double pz, double K, int scan, int *smem, int lane)
{
    RunSink R(P, smem + WALK_SMEM, lane);
    WarpWalk<STRAT, RunSink> W(T, R, smem, lane, scan);
    bool ok = P.count_only || *(volatile unsigned long long *)P.used < P.cap;   // else the pool is exhausted
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (ok) {
        double ha = 0.0;
        if (STRAT != SCATTER) {
            const int b = P.bnear[j];
            ha = b < 0 ? __longlong_as_double(0x7ff8000000000000LL) : ldg4(T.leaf + b).w;
        }
        const double ra = __dmul_rn(K, ha), r2a = __dmul_rn(ra, ra);
        if (T.root == 0) {
            double4 L;
            double d2;
            if (single_leaf_accepted<STRAT>(T, px, py, pz, K, r2a, L, d2)) ok = R.append(1u, 0, 0);
        } else {
            ok = W.run(px, py, pz, K, r2a);
        }
        ok = ok && R.finish();
    }
    const int nacc = __reduce_add_sync(0xffffffffu, R.nacc);   // at most n <= 2^30
    if (lane == 0) {
        P.qacc[j] = (unsigned)nacc;
        P.qflag[j] = ok ? 0 : 1;
        if (!P.count_only) {
            P.items[j] = ok ? make_int2(R.first, R.nruns) : make_int2(RUN_DEFERRED, 0);
            if (!ok) P.deferred[atomicAdd(P.n_deferred, 1u)] = qi;
        }
    }
    __syncwarp();
}

}  // namespace pb
