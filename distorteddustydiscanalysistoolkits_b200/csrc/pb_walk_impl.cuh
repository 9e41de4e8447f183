// pb_walk_impl.cuh -- the walk of the two-phase point path: a warp walks one query's tree and writes
// its accepted leaves, merged into runs of consecutive sorted indices, to extents of a shared pool.
// Shared by the walk kernels (pb_walk.cu) and the batched walk (pb_batch.cu).
//
// The warp keeps a stack of tree entries whose top is the next one in DFS order.  Each round its
// lanes take the top 32: an entry that the query does not reach is dropped, a subtree inside the
// query's radius or an accepted leaf stays as an accepted range, any other subtree is replaced by
// its two children.  The accepted ranges before the first subtree still open are the next ones in
// DFS order and are appended to the runs.  The decisions are those of next_item (node_pruned,
// box_upper, the exact leaf test), so the accepted set and its order are the reference's.
//
// A thread per (query, subtree) item, as before, kept 6.7 of 32 lanes busy (paths of different length,
// and leaf, prune, accept and emit steps in turn) and needed a cut of the tree, a prefilter, a sorted
// work list and 64 item records a query; here the 32 lanes test 32 entries of one query.
#pragma once
#include "pb_interp_impl.cuh"

namespace pb {

constexpr int WSTACK = 512;   // entries; taken one at a time above WSTACK - 160, where a round adds at most one
constexpr int WALK_SMEM = WSTACK + 128;   // ints of shared memory per warp

template <int STRAT>
struct WarpWalk {
    const DevTree &T;
    const RunPool &P;
    int *stack, *rlo, *rhi;   // WSTACK entries; 64 runs not written yet, the last one still open
    int lane;
    int cnt = 0;              // runs in rlo/rhi
    int first = -1, cur = -1, nruns = 0;
    int nacc = 0;             // this lane's share of the accepted leaves

    __device__ __forceinline__ WarpWalk(const DevTree &t, const RunPool &p, int *smem, int l)
        : T(t), P(p), stack(smem), rlo(smem + WSTACK), rhi(smem + WSTACK + 64), lane(l)
    {
    }
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
    // appends the ranges [lo, hi] of the lanes of `done`, in lane order; false if the pool is full
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
    // the walk from the root; false if the pool is full
    __device__ __forceinline__ bool run(double px, double py, double pz, double K, double r2a)
    {
        const int n = (int)T.n;
        const QBox q = make_qbox(px, py, pz);
        const float Kf = (float)K;
        const float r2a_up = __double2float_ru(r2a);
        const float bulk_lim = __fmul_rd(__double2float_rd(r2a), MARGIN_DN);
        const unsigned below = (1u << lane) - 1u;
        const int64_t limit = 4 * T.n + 64;
        int64_t guard = 0;
        int size = 1;
        if (lane == 0) stack[0] = T.root;
        __syncwarp();
        while (size > 0) {
            if (++guard > limit || size > WSTACK - 2) {
                flag(T.status, ST_TRAVERSAL);
                break;
            }
            const int k = size > WSTACK - 160 ? 1 : (size < 32 ? size : 32);
            int c = 0, e0 = 0, e1 = 0, lo = 0, hi = 0;   // c: entries that replace this one
            if (lane < k) {
                const int e = stack[size - 1 - lane];
                const int id = e & 0x7fffffff;
                if (id >= n) {
                    lo = hi = id - n;
                    c = 1;
                    if (e >= 0) {
                        const double4 L = ldg4(T.leaf + lo);
                        double r2;
                        if (STRAT == GATHER) r2 = r2a;
                        else {
                            const double r = __dmul_rn(K, L.w);
                            const double rr = __dmul_rn(r, r);
                            r2 = STRAT == SCATTER ? rr : (r2a > rr ? r2a : rr);
                        }
                        if (!(d2_point(px, py, pz, L) <= r2)) c = 0;
                    }
                    e0 = (int)((unsigned)id | 0x80000000u);
                } else {
                    const int2 rg = __ldg(T.range + (id - 1));
                    lo = rg.x;
                    hi = rg.y;
                    if (e < 0) {   // accepted whole in an earlier round
                        c = 1;
                        e0 = e;
                    } else {
                        const NodeF nd = load_node(T.node + (id - 1));
                        if (node_pruned<STRAT>(T, nd, id, q, Kf, r2a_up)) {
                            c = 0;
                        } else if (STRAT != SCATTER && box_upper(q, nd) <= bulk_lim) {
                            c = 1;
                            e0 = (int)((unsigned)id | 0x80000000u);
                        } else {
                            // the children of a Karras node meet at the split, which the left child's
                            // id gives; a child of one leaf is that leaf
                            c = 2;
                            e0 = nd.left;
                            const int split = nd.left >= n ? nd.left - (n - 1) : nd.left;   // 1-based
                            e1 = split == hi ? n + hi : split + 1;
                        }
                    }
                }
            }
            __syncwarp();
            const unsigned open = __ballot_sync(0xffffffffu, c == 2);
            const int firstopen = open ? __ffs(open) - 1 : 32;
            const unsigned done = __ballot_sync(0xffffffffu, c == 1 && lane < firstopen);
            const unsigned kept = __ballot_sync(0xffffffffu, c >= 1 && lane >= firstopen);
            size += __popc(kept) + __popc(open) - k;
            if (c >= 1 && lane >= firstopen) {
                const int at = size - 1 - __popc(kept & below) - __popc(open & below);
                stack[at] = e0;
                if (c == 2) stack[at - 1] = e1;
            }
            __syncwarp();
            if (done && !append(done, lo, hi)) return false;
        }
        return cnt == 0 || flush(cnt);
    }
};

// The walk of the j-th listed query (sample point qi at px, py, pz; nearest sorted leaf P.bnear[j]):
// its run list, its number of accepted leaves, and whether the pool was full (the query is then
// listed as deferred).  Every lane of the warp calls it; smem holds WALK_SMEM ints.
template <int STRAT>
__device__ __forceinline__ void walk_query(const DevTree &T, const RunPool &P, int64_t j, uint32_t qi, double px,
                                           double py, double pz, double K, int *smem, int lane)
{
    WarpWalk<STRAT> W(T, P, smem, lane);
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
            if (single_leaf_accepted<STRAT>(T, px, py, pz, K, r2a, L, d2)) ok = W.append(1u, 0, 0) && W.flush(1);
        } else {
            ok = W.run(px, py, pz, K, r2a);
        }
    }
    const int nacc = __reduce_add_sync(0xffffffffu, W.nacc);   // at most n <= 2^30
    if (lane == 0) {
        P.qacc[j] = (unsigned)nacc;
        P.qflag[j] = ok ? 0 : 1;
        if (!P.count_only) {
            P.items[j] = ok ? make_int2(W.first, W.nruns) : make_int2(RUN_DEFERRED, 0);
            if (!ok) P.deferred[atomicAdd(P.n_deferred, 1u)] = qi;
        }
    }
    __syncwarp();
}

}  // namespace pb
