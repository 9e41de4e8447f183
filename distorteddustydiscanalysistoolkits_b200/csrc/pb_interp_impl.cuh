// pb_interp_impl.cuh -- the traversal building blocks shared by the interpolation units:
// nearest-h search, the stackless left/escape DFS of the ball query
// (LinearBVHTraversalMacros.jl:26-371) in its warp-uniform form (next_item), the dealing of a
// query's accepted runs to the lanes of a warp (deal_runs) and the FP64 accumulator of the
// reference's arithmetic.
//
// Included by pb_interp64.cu (-fmad=false; FP64 terms in the reference's expressions and
// order, bit-exact with the FP64 oracle), pb_interp32.cu (FP32 per-pair terms with double-float
// offsets, FP64 accumulation of FP32 chunk sums) and
// pb_walk.cu (the walk kernels).
//
// Accepted neighbours are visited in ascending sorted-leaf order (DFS preorder), exactly as
// in the reference, so the per-query summation order does not depend on the launch shape.
// Node pruning uses FP32 boxes rounded outward: it visits a superset of the reference's
// nodes and accepts exactly the same leaves.
#pragma once
#include "pb_device.cuh"

namespace pb {

template <int N, typename T>
__device__ __forceinline__ T pick(const T (&a)[N], int i)
{
    T r = a[0];
#pragma unroll
    for (int k = 1; k < N; ++k)
        if (i == k) r = a[k];
    return r;
}

// Compile-time shape of a launch's catalog, for the pair kernels (FP64 and FP32C).  CAT 0 reads everything from
// the DevCatalog at run time; 1: four columns, gradient + divergence + curl; 2: four columns,
// curl only; 3: one column, scalars only.  A specialised kernel performs exactly the
// operations, in the same order, that the generic one performs for such a catalog.
constexpr int CAT_ANY = 0, CAT_GDC4 = 1, CAT_C4 = 2, CAT_S1 = 3, CAT_SG1 = 4;   // SG1: one column, scalar + gradient

template <int CAT>
struct CatShape {
    __device__ static __forceinline__ int nu(const DevCatalog &C)
    {
        return (CAT == CAT_GDC4 || CAT == CAT_C4) ? 4 : ((CAT == CAT_S1 || CAT == CAT_SG1) ? 1 : C.nU);
    }
    __device__ static __forceinline__ bool grad(const DevCatalog &C)
    {
        return (CAT == CAT_GDC4 || CAT == CAT_SG1) ? true : (CAT == CAT_ANY ? C.n_grad > 0 : false);
    }
    __device__ static __forceinline__ bool div(const DevCatalog &C)
    {
        return CAT == CAT_GDC4 ? true : (CAT == CAT_ANY ? C.n_div > 0 : false);
    }
    __device__ static __forceinline__ bool curl(const DevCatalog &C)
    {
        return (CAT == CAT_GDC4 || CAT == CAT_C4) ? true : (CAT == CAT_ANY ? C.n_curl > 0 : false);
    }
    __device__ static __forceinline__ bool any(const DevCatalog &C) { return grad(C) || div(C) || curl(C); }
    __device__ static __forceinline__ int stride(int s)
    {
        return (CAT == CAT_GDC4 || CAT == CAT_C4) ? 4 : ((CAT == CAT_S1 || CAT == CAT_SG1) ? 3 : s);
    }
};

inline int catalog_shape(const DevCatalog &C)
{
    if (C.nU == 4 && C.n_grad == 1 && C.g_u[0] == 0 && C.n_div == 1 && C.n_curl == 1) return CAT_GDC4;
    if (C.nU == 4 && C.n_grad == 0 && C.n_div == 0 && C.n_curl == 1) return CAT_C4;
    if (C.nU == 1 && C.n_grad == 0 && C.n_div == 0 && C.n_curl == 0) return CAT_S1;
    if (C.nU == 1 && C.n_grad == 1 && C.g_u[0] == 0 && C.n_div == 0 && C.n_curl == 0) return CAT_SG1;
    return CAT_ANY;
}

__device__ __forceinline__ void flag(int *status, int bit) { atomicOr(status, bit); }

__device__ __forceinline__ NodeF load_node(const NodeF *p)
{
    NodeF nd;   // the 32-byte record in one 256-bit load
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(nd.lox), "=f"(nd.loy), "=f"(nd.loz), "=r"(nd.left), "=f"(nd.hix), "=f"(nd.hiy), "=f"(nd.hiz), "=r"(nd.escape)
        : "l"(p));
    return nd;
}

// ------------------------------------------------------------------------------------
// a / b, correctly rounded, from y = RN(1/b): Markstein's theorem (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990; Muller et al., Handbook of
// Floating-Point Arithmetic, on division with a correctly rounded reciprocal): if q is
// within one ulp of a/b, RN(q + y RN(a - b q)) is RN(a/b).  a y can be off by 1.5 ulp, so one step
// brings q within an ulp and the second one gives the quotient.  `safe` says that both operands
// are in the exponent range where no step can under- or overflow (exp_safe); otherwise (zero,
// infinities and NaN included) they are divided.
__device__ __forceinline__ double div_by(double a, double b, double y, bool safe)
{
    if (!safe) return a / b;
    double q = a * y;
    q = fma(fma(-q, b, a), y, q);
    return fma(fma(-q, b, a), y, q);
}

// --------------------------------------------------------------------------------------
// FP32 box tests with directed rounding.  The query point is kept as round-down/round-up
// floats; gaps, squares and sums are rounded toward the safe side, so `lower` never exceeds
// the exact box distance^2 and `upper` is never below the exact farthest-corner distance^2.
// Decisions then carry a relative margin of 2^-20, far above FP64 rounding (2^-53), so a
// subtree is pruned only if every leaf in it fails its FP64 acceptance test and is
// bulk-accepted only if every leaf passes it -- exactly the decisions of the FP64 walk.
struct QBox {
    float dn[3], up[3];
};

__device__ __forceinline__ QBox make_qbox(double px, double py, double pz)
{
    QBox q;
    q.dn[0] = __double2float_rd(px); q.up[0] = __double2float_ru(px);
    q.dn[1] = __double2float_rd(py); q.up[1] = __double2float_ru(py);
    q.dn[2] = __double2float_rd(pz); q.up[2] = __double2float_ru(pz);
    return q;
}

constexpr float MARGIN_UP = 1.0f + 9.5367431640625e-07f;   // 1 + 2^-20
constexpr float MARGIN_DN = 1.0f - 9.5367431640625e-07f;

__device__ __forceinline__ float box_lower(const QBox &q, const NodeF &nd)
{
    float gx = fmaxf(fmaxf(__fsub_rd(nd.lox, q.up[0]), __fsub_rd(q.dn[0], nd.hix)), 0.f);
    float gy = fmaxf(fmaxf(__fsub_rd(nd.loy, q.up[1]), __fsub_rd(q.dn[1], nd.hiy)), 0.f);
    float gz = fmaxf(fmaxf(__fsub_rd(nd.loz, q.up[2]), __fsub_rd(q.dn[2], nd.hiz)), 0.f);
    return __fadd_rd(__fadd_rd(__fmul_rd(gx, gx), __fmul_rd(gy, gy)), __fmul_rd(gz, gz));
}

__device__ __forceinline__ float box_upper(const QBox &q, const NodeF &nd)
{
    float fx = fmaxf(__fsub_ru(q.up[0], nd.lox), __fsub_ru(nd.hix, q.dn[0]));
    float fy = fmaxf(__fsub_ru(q.up[1], nd.loy), __fsub_ru(nd.hiy, q.dn[1]));
    float fz = fmaxf(__fsub_ru(q.up[2], nd.loz), __fsub_ru(nd.hiz, q.dn[2]));
    return __fadd_ru(__fadd_ru(__fmul_ru(fx, fx), __fmul_ru(fy, fy)), __fmul_ru(fz, fz));
}

// (K h)^2 rounded up, for a node's hmax (already rounded up) or the query radius
__device__ __forceinline__ float sq_up(float K, float h)
{
    float r = __fmul_ru(K, h);
    return __fmul_ru(r, r);
}

// LBVH_find_nearest_h (LinearBVHQueries.jl:118-140).  The reference walks the tree in DFS
// order with a shrinking radius and keeps the first strictly closer leaf, i.e. it returns
// the minimum squared distance and, among equal distances, the smallest sorted leaf index.
// This search visits the nearer child first (explicit stack) and applies exactly that
// rule, so it returns the same leaf while visiting far fewer nodes.  Boxes are the FP32
// outward-rounded ones (never farther than any leaf inside), and a subtree is skipped only
// when its box distance is strictly greater than the best distance.
constexpr int NN_STACK = 64;

__device__ __forceinline__ float child_dist(const DevTree &T, const QBox &q, int id, double px, double py,
                                            double pz, double &best, int64_t &bi)
{
    const int64_t n = T.n;
    if (id >= n) {
        int64_t b = id - n;
        double d2 = d2_point(px, py, pz, ldg4(T.leaf + b));
        if (d2 < best || (d2 == best && b < bi)) { best = d2; bi = b; }
        // a leaf needs no further visit: NaN compares false even when the best distance is beyond
        // FP32 and every finite or infinite bound would pass
        return __int_as_float(0x7fffffff);
    }
    return box_lower(q, load_node(T.node + (id - 1)));
}

// WITHIN: of the leaves with d2 <= within only (-1 if there is none).  The bound also ends the search
// early: a point far from all particles else visits the whole tree, as the FP32 boxes do not tell its
// distances apart (probes of radius 1 at 40,000 points some 1e9 from 2e5 particles: 332 ms, 0.29 ms with it).
template <bool WITHIN = false>
__device__ __forceinline__ int64_t nearest_leaf(const DevTree &T, double px, double py, double pz,
                                                double within = INFINITY)
{
    double best = INFINITY;
    int64_t bi = -1;
    if (WITHIN && within < INFINITY) {   // the index of a leaf at exactly that distance is below T.n
        best = within;
        bi = T.n;
    }
    if (WITHIN && !(within >= 0.0)) return -1;   // NaN
    if (T.root == 0) {
        double d2 = d2_point(px, py, pz, ldg4(T.leaf));
        return d2 < best || (WITHIN && d2 == best && bi > 0) ? 0 : -1;
    }
    const QBox q = make_qbox(px, py, pz);
    int sn[NN_STACK];
    float sd[NN_STACK];
    int sp = 0;
    int node = T.root;
    int64_t guard = 0, limit = 4 * T.n + 64;
    // a subtree is skipped only when its lower bound exceeds the best distance by the margin
    auto visit = [&](float d) { return d <= __fmul_ru(__double2float_ru(best), MARGIN_UP); };
    for (;;) {
        if (++guard > limit) { atomicOr(T.status, ST_TRAVERSAL); break; }
        int2 ch = __ldg(T.child + (node - 1));
        float dl = child_dist(T, q, ch.x, px, py, pz, best, bi);
        float dr = child_dist(T, q, ch.y, px, py, pz, best, bi);
        bool vl = visit(dl), vr = visit(dr);
        if (vl && vr) {
            bool lf = dl <= dr;
            int far = lf ? ch.y : ch.x;
            float fd = lf ? dr : dl;
            if (sp < NN_STACK) { sn[sp] = far; sd[sp] = fd; ++sp; }
            else { atomicOr(T.status, ST_TRAVERSAL); }
            node = lf ? ch.x : ch.y;
            continue;
        }
        if (vl) { node = ch.x; continue; }
        if (vr) { node = ch.y; continue; }
        node = 0;
        while (sp > 0) {
            --sp;
            if (visit(sd[sp])) { node = sn[sp]; break; }
        }
        if (node == 0) break;
    }
    return !WITHIN || bi < T.n ? bi : -1;
}

// --------------------------------------------------------------------------------------
// State of a stackless left/escape traversal (LinearBVHTraversalMacros.jl:135-371).  A subtree
// lying entirely inside the query's radius is turned into its contiguous sorted-leaf range,
// which is exactly the DFS order of its leaves, so the sequence of accepted leaves is the
// reference's.
struct Walk {
    int node;
    int64_t cur, end, guard, limit;
};

// The walk's pruning decision for internal node `node` (box `nd`): FP32 box distance with
// directed rounding against the node radius (query radius and/or K * hmax) with the 2^-20
// margin.  Shared by every walk of a query, so that all decide alike.
template <int STRAT>
__device__ __forceinline__ bool node_pruned(const DevTree &T, const NodeF &nd, int node, const QBox &q, float Kf,
                                            float r2a_up)
{
    float r2n;
    if (STRAT == GATHER) r2n = r2a_up;
    else {
        float rr = sq_up(Kf, __ldg(T.node_hmax + (node - 1)));
        r2n = STRAT == SCATTER ? rr : fmaxf(r2a_up, rr);
    }
    return box_lower(q, nd) > __fmul_ru(r2n, MARGIN_UP);
}

// Warp-uniform form of the same walk for the warp-per-query kernels: returns the next
// accepted item in DFS order, either a single leaf (lo == hi) or the whole contiguous leaf
// range of a subtree that lies inside the query radius.  With leaf_size > 1, a subtree of at
// most leaf_size leaves that is neither pruned nor accepted whole is scanned leaf by leaf in
// sorted order with the exact FP64 test instead of being descended: the accepted leaves and
// their order -- hence every sum -- are the same, only the node visits change.
template <int STRAT>
__device__ __forceinline__ bool next_item(const DevTree &T, Walk &w, double px, double py, double pz, double K,
                                          double r2a, int64_t &lo, int64_t &hi, int leaf_size = 1)
{
    const int64_t n = T.n;
    const QBox q = make_qbox(px, py, pz);
    const float Kf = (float)K;
    const float r2a_up = __double2float_ru(r2a);
    const float bulk_lim = __fmul_rd(__double2float_rd(r2a), MARGIN_DN);
    for (;;) {
        if (w.cur <= w.end) {   // linear scan of a small subtree's leaves
            if (++w.guard > w.limit) { flag(T.status, ST_TRAVERSAL); w.cur = 1; w.end = 0; w.node = 0; return false; }
            const int64_t b = w.cur++;
            const double4 L = ldg4(T.leaf + b);
            double r2;
            if (STRAT == GATHER) r2 = r2a;
            else {
                double r = __dmul_rn(K, L.w);
                double rr = __dmul_rn(r, r);
                r2 = STRAT == SCATTER ? rr : (r2a > rr ? r2a : rr);
            }
            if (d2_point(px, py, pz, L) <= r2) { lo = hi = b; return true; }
            continue;
        }
        if (w.node == 0) return false;
        if (++w.guard > w.limit) { flag(T.status, ST_TRAVERSAL); w.node = 0; return false; }
        const int node = w.node;
        if (node >= n) {
            int64_t b = node - n;
            double4 L = ldg4(T.leaf + b);
            w.node = __ldg(T.leaf_escape + b);
            double r2;
            if (STRAT == GATHER) r2 = r2a;
            else {
                double r = __dmul_rn(K, L.w);
                double rr = __dmul_rn(r, r);
                r2 = STRAT == SCATTER ? rr : (r2a > rr ? r2a : rr);
            }
            if (d2_point(px, py, pz, L) <= r2) { lo = hi = b; return true; }
            continue;
        }
        NodeF nd = load_node(T.node + (node - 1));
        if (node_pruned<STRAT>(T, nd, node, q, Kf, r2a_up)) { w.node = nd.escape; continue; }
        if (STRAT != SCATTER && box_upper(q, nd) <= bulk_lim) {
            int2 rg = __ldg(T.range + (node - 1));
            lo = rg.x;
            hi = rg.y;
            w.node = nd.escape;
            return true;
        }
        if (leaf_size > 1) {
            const int2 rg = __ldg(T.range + (node - 1));
            if (rg.y - rg.x < leaf_size) {   // scan this subtree's leaves, then continue after it
                w.cur = rg.x;
                w.end = rg.y;
                w.node = nd.escape;
                continue;
            }
        }
        w.node = nd.left;
    }
}

// Slot filler shared by the warp-per-query kernels: accepted leaves, in DFS order, are
// dealt to the 32 lanes (the k-th accepted leaf goes to lane k mod 32); PROC(fill) is
// called whenever 32 slots are full and once more for the remainder.
struct Slots {
    int fill;
    int64_t mine;   // this lane's leaf in the current batch (-1 if none)
};

template <typename PROC>
__device__ __forceinline__ void deal(Slots &S, int lane, int64_t lo, int64_t hi, PROC &proc)
{
    while (lo <= hi) {
        int64_t t = hi - lo + 1;
        int room = 32 - S.fill;
        if (t > room) t = room;
        if (lane >= S.fill && lane < S.fill + (int)t) S.mine = lo + (lane - S.fill);
        S.fill += (int)t;
        lo += t;
        if (S.fill == 32) {
            proc(32);
            S.fill = 0;
            S.mine = -1;
        }
    }
}

// Size class of a query of a accepted leaves, 0..124, ascending with a: the power of two and the next
// two bits.  The pair kernels take queries by descending class, and within a class in walk (Morton)
// order, so that queries running at the same time read the same particles.
__device__ __forceinline__ unsigned count_class(unsigned a)
{
    if (a == 0) return 0u;
    const unsigned e = 31u - (unsigned)__clz((int)a);
    return 4u * e + (e >= 2 ? (a >> (e - 2)) & 3u : (a << (2 - e)) & 3u) + 1u;
}

// query scheduling: warps take queries in the given order from a global counter
__device__ __forceinline__ int64_t next_query(unsigned long long *counter, int lane)
{
    unsigned long long q = 0;
    if (lane == 0) q = atomicAdd(counter, 1ULL);
    return (int64_t)__shfl_sync(0xffffffffu, q, 0);
}

// --------------------------------------------------------------------------------------
// One chunk of up to 32 runs of an item, one run per lane (lanes past the last run hold an
// empty one), with the inclusive prefix sums of the run lengths: leaf position t of the chunk,
// 0 <= t < tot, lies in the first run r with inc[r] > t.  Leaf indices and counts are 32-bit
// (n <= 2^30).
struct RunWindow {
    int lo, inc, ex, tot;          // this lane's run: first leaf, inclusive and exclusive prefix
    int r0 = -1, end0 = 0;         // run of the last position looked up, and where it ends
    int lo0 = 0, ex0 = 0;

    __device__ __forceinline__ RunWindow(const RunPool &P, int c, int cnt, int lane)
    {
        const uint2 rn = lane < cnt ? __ldg(P.runs + (int64_t)c * RUN_CHUNK + lane) : make_uint2(0u, 0u);
        lo = (int)rn.x;
        inc = (int)rn.y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        tot = __shfl_sync(0xffffffffu, inc, 31);
        ex = inc - (int)rn.y;
    }
    // makes r0 the run of position t (t >= the previous one); warp-uniform
    __device__ __forceinline__ void seek(int t)
    {
        if (end0 > t) return;
        r0 = __popc(__ballot_sync(0xffffffffu, inc <= t));   // prefix sums ascend: runs that end before t
        end0 = __shfl_sync(0xffffffffu, inc, r0);
        lo0 = __shfl_sync(0xffffffffu, lo, r0);
        ex0 = __shfl_sync(0xffffffffu, ex, r0);
    }
    // the leaf of position tb + lane into `mine`, on the lanes whose position lies in this chunk;
    // r0 is the run of position max(tb, 0)
    __device__ __forceinline__ void leaf_of(int tb, int lane, int &mine) const
    {
        const int tl = tb + lane;
        if (tb >= 0 && tb + 32 <= end0) {
            mine = lo0 + (tl - ex0);
            return;
        }
        // batch positions (after its first one in this chunk) at which a run starts: a lane's run
        // is r0 plus the starts up to its position
        const int first = tb < 0 ? -tb : 0, s = ex - tb;
        const unsigned starts = __reduce_or_sync(0xffffffffu, s > first && s < 32 && inc > ex ? 1u << s : 0u);
        const int r = r0 + __popc(starts & (0xffffffffu >> (31 - lane)));
        const int l = __shfl_sync(0xffffffffu, lo, r), e = __shfl_sync(0xffffffffu, ex, r);
        if (tl >= 0 && tl < tot) mine = l + (tl - e);
    }
};

// the chunk after chunk c of a list with `left` runs from c on
__device__ __forceinline__ int next_chunk(const RunPool &P, int c, int left)
{
    if (left <= RUN_CHUNK) return -1;
    return (c & (RUN_EXTENT - 1)) != RUN_EXTENT - 1 ? c + 1 : __ldg(P.next + c);
}

// Dealing of a walked query's accepted leaves (its runs, chunk by chunk) to the 32 lanes in DFS
// order: the k-th accepted leaf goes to lane k mod 32.  first(b) is called with the first leaf
// of a non-empty list; one(mine) for every full batch (every lane holds a leaf); two(m1) for
// two consecutive full batches inside one run (lane leaves m1 and m1 + 32) when cantwo()
// allows it, and four(m1) for four of them (m1, m1 + 32, m1 + 64, m1 + 96) when canfour()
// does.  Returns the fill of the last, partial batch, whose leaves are left in `mine` (-1 on
// empty lanes).
template <typename FIRST, typename ONE, typename TWO, typename CANTWO, typename FOUR, typename CANFOUR>
__device__ __forceinline__ int deal_runs(const RunPool &P, int64_t j, int lane, FIRST &first, ONE &one, TWO &two,
                                         CANTWO &cantwo, FOUR &four, CANFOUR &canfour, int &mine)
{
    const int2 itm = __ldg(P.items + j);
    int fill = 0, c = itm.x, left = itm.y;
    mine = -1;
    if (left > 0) first((int)__ldg(&P.runs[(int64_t)c * RUN_CHUNK].x));
    while (left > 0) {
        const int cnt = left < RUN_CHUNK ? left : RUN_CHUNK;
        const int nextc = next_chunk(P, c, left);
        RunWindow R(P, c, cnt, lane);
        int tb = -fill;
        for (;;) {
            // t0 < tot = inc[cnt - 1], so the cursor stops at a run of this chunk
            R.seek(tb <= 0 ? 0 : (tb < R.tot ? tb : R.tot - 1));
            if (tb >= 0 && tb + 64 <= R.end0) {
                const int m1 = R.lo0 + (tb - R.ex0) + lane;
                if (tb + 128 <= R.end0 && canfour()) {   // four full batches inside one run
                    four(m1);
                    tb += 128;
                    continue;
                }
                if (cantwo()) {   // two full batches inside one run
                    two(m1);
                    tb += 64;
                    continue;   // the next pass assigns or closes what is left of the chunk
                }
            }
            R.leaf_of(tb, lane, mine);
            if (tb + 31 < R.tot) {
                one(mine);   // full batch
                mine = -1;
                tb += 32;
            } else {
                fill = R.tot - tb;
                break;
            }
        }
        left -= cnt;
        c = nextc;
    }
    return fill;
}

// The same dealing for one of W warps that share a query: warp w gets the batches b with
// b mod W == w; one(mine) for every full one.  Returns the fill of the last, partial batch
// if it is this warp's (its leaves in `mine`), else 0.
template <int W, typename ONE>
__device__ __forceinline__ int deal_runs_part(const RunPool &P, int64_t j, int lane, int w, ONE &one, int &mine)
{
    const int2 itm = __ldg(P.items + j);
    int fill = 0, c = itm.x, left = itm.y, turn = 0;   // turn: the current batch's number mod W
    mine = -1;
    while (left > 0) {
        const int cnt = left < RUN_CHUNK ? left : RUN_CHUNK;
        const int nextc = next_chunk(P, c, left);
        RunWindow R(P, c, cnt, lane);
        int tb = -fill;
        for (;;) {
            if (turn == w && tb < R.tot) {
                R.seek(tb < 0 ? 0 : tb);
                R.leaf_of(tb, lane, mine);
            }
            if (tb + 31 >= R.tot) {
                fill = R.tot - tb;
                break;
            }
            if (turn == w) {
                one(mine);
                mine = -1;
            }
            tb += 32;
            turn = turn + 1 == W ? 0 : turn + 1;
        }
        left -= cnt;
        c = nextc;
    }
    return turn == w ? fill : 0;
}

// adds a row's first `fill` terms to acc in slot order
__device__ __forceinline__ double add_row(const double *row, int fill, double acc)
{
    const double2 *r2 = reinterpret_cast<const double2 *>(row);
    if (fill == 32) {
#pragma unroll
        for (int s = 0; s < 16; ++s) {
            const double2 v = r2[s];
            acc += v.x;
            acc += v.y;
        }
        return acc;
    }
    for (int s = 0; s < fill; ++s) acc += row[s];
    return acc;
}

// the n == 1 tree has no internal node: its single leaf is tested directly
template <int STRAT>
__device__ __forceinline__ bool single_leaf_accepted(const DevTree &T, double px, double py, double pz, double K,
                                                     double r2a, double4 &L, double &d2)
{
    L = ldg4(T.leaf);
    double r = __dmul_rn(K, L.w), rr = __dmul_rn(r, r);
    double r2 = STRAT == GATHER ? r2a : (STRAT == SCATTER ? rr : (r2a > rr ? r2a : rr));
    d2 = d2_point(px, py, pz, L);
    return d2 <= r2;
}

// --------------------------------------------------------------------------------------
// A query's FP64 sums and their finalisation (the reference's arithmetic)
struct Exact64 {
    double S1;
    double SA[MAXU];
    double Bq[3];
    double Fg[MAXG][3];
    double Bd[3], Sd;
    double D[MAXD];
    double Cc[MAXC][3];

    __device__ __forceinline__ void finalize(const DevCatalog &C, int64_t qi) const
    {
        int l = 0;
        if (S1 == 0.0) {
            for (int o = 0; o < C.L; ++o) C.out[o][qi] = __longlong_as_double(0x7ff8000000000000LL);
            return;
        }
        double inv = 1.0 / S1;
#pragma unroll
        for (int j = 0; j < MAXS; ++j) {
            if (j < C.n_scalar) {
                double s = pick<MAXU>(SA, C.s_u[j]);
                C.out[l++][qi] = C.s_shep[j] ? s * inv : s;
            }
        }
#pragma unroll
        for (int j = 0; j < MAXG; ++j) {
            if (j < C.n_grad) {
                int u = C.g_u[j];
                if (u < 0) {
                    double a = Sd * inv;
                    C.out[l++][qi] = Fg[j][0] - Bd[0] * a;
                    C.out[l++][qi] = Fg[j][1] - Bd[1] * a;
                    C.out[l++][qi] = Fg[j][2] - Bd[2] * a;
                } else {
                    double a = pick<MAXU>(SA, u) * inv;
                    C.out[l++][qi] = Fg[j][0] - Bq[0] * a;
                    C.out[l++][qi] = Fg[j][1] - Bq[1] * a;
                    C.out[l++][qi] = Fg[j][2] - Bq[2] * a;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < MAXD; ++j) {
            if (j < C.n_div) {
                double ax = pick<MAXU>(SA, C.d_u[j][0]) * inv;
                double ay = pick<MAXU>(SA, C.d_u[j][1]) * inv;
                double az = pick<MAXU>(SA, C.d_u[j][2]) * inv;
                double bb = ax * Bq[0] + ay * Bq[1] + az * Bq[2];
                C.out[l++][qi] = D[j] - bb;
            }
        }
#pragma unroll
        for (int j = 0; j < MAXC; ++j) {
            if (j < C.n_curl) {
                double ax = pick<MAXU>(SA, C.c_u[j][0]) * inv;
                double ay = pick<MAXU>(SA, C.c_u[j][1]) * inv;
                double az = pick<MAXU>(SA, C.c_u[j][2]) * inv;
                double bx = ay * Bq[2] - az * Bq[1];
                double by = az * Bq[0] - ax * Bq[2];
                double bz = ax * Bq[1] - ay * Bq[0];
                C.out[l++][qi] = -(Cc[j][0] - bx);
                C.out[l++][qi] = -(Cc[j][1] - by);
                C.out[l++][qi] = -(Cc[j][2] - bz);
            }
        }
    }
};

}  // namespace pb
