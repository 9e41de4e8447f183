// pb_fp64_impl.cuh -- the FP64 per-pair terms with the reference's expressions and the
// in-order column sums of the warp-per-query kernels, and the fused per-query body.  Shared by
// pb_interp64.cu and the batched kernel (pb_batch.cu); both are compiled with -fmad=false, so
// the values are the reference's FP64 results bit for bit in either.
//
// The FP64 pipe (64 lanes per SM: two issue cycles per warp instruction) bounds these kernels,
// so the terms are arranged to need fewer FP64 operations for the same bits: 1/h and 1/rho of a
// particle come from the tree (DevTree::aux), quotients by a number whose reciprocal is known
// take five operations (div_by), pieces and supports are selected by integer compares on the
// high word, the kernel family and the catalog's shape are compile-time, and a side (h_a or
// h_b) whose support the pair lies outside of is skipped: its terms are zeros.
#pragma once
#include "pb_interp_impl.cuh"

namespace pb {

// ------------------------------------------------------------------------------------
// x^N as jl_pow computes it for finite x >= 0, with the steps that only add zeros left out:
// (p, e) -> (p^2, its low part) is one squaring of the compensated pair.
__device__ __forceinline__ void jl_sq(double &p, double &e)
{
    const double err = p * 2.0 * e, s = p * p;
    e = fma(p, p, -s) + err;
    p = s;
}

template <int N>
__device__ __forceinline__ double jl_pow_n(double x)
{
    if (N == 2) return x * x;
    if (N == 3) return x * x * x;
    double p = x * x, e = fma(x, x, -p);   // x^2
    if (N == 4 || N == 5) {
        jl_sq(p, e);
        return N == 4 ? p + e : fma(p, x, x * e);
    }
    if (N == 6) {
        const double y = p, yl = e;
        jl_sq(p, e);
        return fma(p, y, fma(y, e, p * yl));
    }
    if (N == 7) {
        const double y = p * x, yl = fma(p, x, -y) + x * e;
        jl_sq(p, e);
        return fma(p, y, fma(y, e, p * yl));
    }
    jl_sq(p, e);
    jl_sq(p, e);
    return p + e;   // N == 8
}

// high words of the pieces' boundaries: for q >= 0, q < c  <=>  hi(q) < hi(c) (c has no low bits)
constexpr int HI_HALF = 0x3fe00000, HI_1 = 0x3ff00000, HI_3_2 = 0x3ff80000, HI_2 = 0x40000000, HI_5_2 = 0x40040000,
              HI_3 = 0x40080000;
template <int KT>
__device__ constexpr int hi_valid()
{
    return KT == 1 ? HI_5_2 : (KT == 2 ? HI_3 : HI_2);
}

// kshape<double>(KT, q) and kdshape<double>(KT, q) for q >= 0, same expressions and same bits
template <int KT>
__device__ __forceinline__ double shape64(double q)
{
    const int hq = __double2hiint(q);
    if (hq >= hi_valid<KT>()) return 0.0;
    if (KT == 0) {
        const double c = 0.25 * jl_pow_n<3>(2.0 - q);
        if (hq >= HI_1) return c;
        return c - jl_pow_n<3>(1.0 - q);
    }
    if (KT == 1) {
        double f = jl_pow_n<4>(2.5 - q);
        if (hq < HI_3_2) f = f - 5.0 * jl_pow_n<4>(1.5 - q);
        if (hq < HI_HALF) f = f + 10.0 * jl_pow_n<4>(0.5 - q);
        return f;
    }
    if (KT == 2) {
        double f = jl_pow_n<5>(3.0 - q);
        if (hq < HI_2) f = f - 6.0 * jl_pow_n<5>(2.0 - q);
        if (hq < HI_1) f = f + 15.0 * jl_pow_n<5>(1.0 - q);
        return f;
    }
    const double t = 1.0 - 0.5 * q;
    if (KT == 3) return jl_pow_n<4>(t) * (2.0 * q + 1.0);
    if (KT == 4) return jl_pow_n<6>(t) * ((35.0 / 12.0) * (q * q) + 3.0 * q + 1.0);
    return jl_pow_n<8>(t) * (4.0 * (q * q * q) + 6.25 * (q * q) + 4.0 * q + 1.0);
}

template <int KT>
__device__ __forceinline__ double dshape64(double q)
{
    const int hq = __double2hiint(q);
    if (hq >= hi_valid<KT>()) return 0.0;
    if (KT == 0) {
        const double c = -0.75 * jl_pow_n<2>(2.0 - q);
        if (hq >= HI_1) return c;
        return c + 3.0 * jl_pow_n<2>(1.0 - q);
    }
    if (KT == 1) {
        const double c = -4.0 * jl_pow_n<3>(2.5 - q);
        if (hq >= HI_3_2) return c;
        const double d = c + 20.0 * jl_pow_n<3>(1.5 - q);
        if (hq >= HI_HALF) return d;
        return d - 40.0 * jl_pow_n<3>(0.5 - q);
    }
    if (KT == 2) {
        const double c = -5.0 * jl_pow_n<4>(3.0 - q);
        if (hq >= HI_2) return c;
        const double d = c + 30.0 * jl_pow_n<4>(2.0 - q);
        if (hq >= HI_1) return d;
        return d - 75.0 * jl_pow_n<4>(1.0 - q);
    }
    const double t = 1.0 - 0.5 * q;
    if (KT == 3) return jl_pow_n<4>(t) * 2.0 - jl_pow_n<3>(t) * (4.0 * q + 2.0);
    if (KT == 4)
        return jl_pow_n<6>(t) * ((35.0 / 6.0) * q + 3.0) - jl_pow_n<5>(t) * ((35.0 / 4.0) * (q * q) + 9.0 * q + 3.0);
    return jl_pow_n<8>(t) * (12.0 * (q * q) + 12.5 * q + 4.0) -
           jl_pow_n<7>(t) * (16.0 * (q * q * q) + 25.0 * (q * q) + 16.0 * q + 4.0);
}

// One side of a pair's kernel (h = h_a or h_b with its correctly rounded reciprocal): W(r, h) and,
// with GRAD, the gradient's coefficient times the offset, in the operation order of kernel.jl:152-157 (W) and
// kernel.jl:284-296,371-376 (gradient).
// A pair outside the support of h (by more than the rounding of either quotient) is left out: its
// terms are zeros, which change no sum.  `regular` is false where some particle's h is negative,
// zero or extreme: then the reference's general expressions are evaluated.
template <int KT, bool GRAD>
__device__ __forceinline__ void side64(double r, double invr, bool rsafe, double dx, double dy, double dz, double h,
                                       double invh, bool regular, double &W, double &gx, double &gy, double &gz)
{
    W = gx = gy = gz = 0.0;
    const double qw = r * invh;
    if (regular && __double2hiint(qw) > hi_valid<KT>()) return;
    const double norm = knorm3<double>(KT);
    const double hD = invh * invh * invh;
    double f = shape64<KT>(qw);
    if (!regular) f = kshape<double>(KT, qw);
    W = hD * (norm * f);
    if (GRAD && invr != 0.0) {   // invr is 0 for a coincident pair
        const double q = div_by(r, h, invh, regular && rsafe);
        double d = dshape64<KT>(q);
        if (!regular) d = kdshape<double>(KT, q);
        const double coeff = d * norm * invr;
        const double hDp1 = hD * invh;
        gx = hDp1 * (dx * coeff);
        gy = hDp1 * (dy * coeff);
        gz = hDp1 * (dz * coeff);
    } else if (GRAD && !regular) {
        gx = gy = gz = hD * invh * 0.0;   // NaN where 1/h^4 overflows
    }
}

// ------------------------------------------------------------------------------------
// Warp-per-query FP64 kernel.  Accepted leaves are dealt to the 32 lanes in DFS order;
// each lane computes its pair's terms with the reference's expressions, the terms go to
// shared memory, and lane a then adds term a of every slot, in slot (= DFS) order, to its
// accumulator -- the reference's sequential sums, bit for bit, with the per-pair work
// spread over the warp.
constexpr int NT = 19;   // S1, SA[4], Bq[3], Fg[3], Bd[3], Sd, D, Cc[3]

// The terms a launch sums, by its catalog's shape: every one of the NT for CAT_ANY, else those that
// its outputs read (the others stay zero).  Term row k holds accumulator acc_of<CAT>(k).
template <int CAT>
__device__ constexpr int nterms64()
{
    return CAT == CAT_S1 ? 2 : (CAT == CAT_SG1 ? 8 : (CAT == CAT_C4 ? 11 : (CAT == CAT_GDC4 ? 15 : NT)));
}

template <int CAT>
__device__ constexpr int row_of(int a)   // term row of accumulator a, -1 if it is not summed
{
    if (CAT == CAT_S1) return a < 2 ? a : -1;
    if (CAT == CAT_SG1) return a < 2 ? a : (a >= 5 && a < 11 ? a - 3 : -1);
    if (CAT == CAT_C4) return a < 8 ? a : (a >= 16 ? a - 8 : -1);
    if (CAT == CAT_GDC4) return a < 11 ? a : (a >= 15 ? a - 4 : -1);
    return a;
}

// Blocks of 128 threads per SM of the pair kernels: they wait on loads and on the chain of
// dependent additions, so resident warps count against the registers (102 at 5 blocks, 85 at 6).
// 2.8e9 pairs, four columns with gradient, divergence and curl, M4 symmetric: 39.7 / 40.3 / 46.8 /
// 40.6 / 44.5 ms at 4 / 5 / 6 / 7 / 8 blocks; one scalar (1.2e9 pairs) 8.4 / 7.6 / 8.3 / 9.1 / 9.3; one side
// (gather, M6, 3.5e9 pairs) needs fewer registers: 50.1 / 43.0 / 38.9 / 39.6 / 40.2.
template <int STRAT, int CAT>
__host__ __device__ constexpr int minb64()
{
    return STRAT == SYMMETRIC || CAT == CAT_ANY ? 5 : 6;
}

// Term buffer of a warp: one row per term, one column per lane.  Lanes write their own column
// (consecutive doubles) and the summing lanes read their row two columns at a time; 34 doubles a
// row keep the 16-byte reads of eight neighbouring lanes on different banks.
constexpr int TROW = 34;
constexpr int TBUF = NT * TROW;   // doubles of a warp's buffer for any catalog

// per-query constants
struct Query64 {
    double px, py, pz, ha, invha;
    bool regular;   // every particle of the tree is (aux_regular)
};

template <int STRAT>
__device__ __forceinline__ Query64 make_query64(const DevTree &T, double px, double py, double pz, int64_t bnear)
{
    Query64 Q;
    Q.px = px; Q.py = py; Q.pz = pz;
    Q.ha = 0.0; Q.invha = 0.0;
    Q.regular = __ldg(T.odd) == 0;
    if (STRAT != SCATTER) {
        Q.ha = bnear < 0 ? __longlong_as_double(0x7ff8000000000000LL) : ldg4(T.leaf + bnear).w;
        Q.invha = 1.0 / Q.ha;
        Q.regular = Q.regular && bnear >= 0;
    }
    return Q;
}

// what a pair reads of its neighbour
struct Nb64 {
    double4 L, X;   // {x, y, z, h}, {1/h, 1/rho, m, rho}
    double A[MAXU];
};

template <int CAT>
__device__ __forceinline__ void load_nb64(const DevTree &T, const DevCatalog &C, int64_t b, Nb64 &N)
{
    N.L = ldg4(T.leaf + b);
    N.X = ldg4(T.aux + b);
#pragma unroll
    for (int u = 0; u < MAXU; ++u) N.A[u] = (u < CatShape<CAT>::nu(C)) ? __ldg(C.ucol[u] + b) : 0.0;
}

// the pair's terms, written to this lane's column of the warp's term buffer
template <int STRAT, int KT, int CAT>
__device__ __forceinline__ void terms64(const DevCatalog &C, const Query64 &Q, const Nb64 &N, double *col)
{
    constexpr bool any_cat = CAT == CAT_ANY;
    const bool grad = CatShape<CAT>::any(C);
    auto put = [&](int a, double v) { col[row_of<CAT>(a) * TROW] = v; };
    const double dx = Q.px - N.L.x, dy = Q.py - N.L.y, dz = Q.pz - N.L.z;
    const double d2 = dx * dx + dy * dy + dz * dz;
    const double r = sqrt(d2);
    const bool rsafe = exp_safe(r);
    const double invrb = N.X.y, mb = N.X.z, rb = N.X.w;
    // the gradient's 1/r; 0 stands for a coincident pair, which has no gradient terms
    const double invr = grad && d2 != 0.0 ? 1.0 / r : 0.0;
    double W, gx, gy, gz;
    auto side = [&](double h, double invh, double &w, double &x, double &y, double &z) {
        if (grad) side64<KT, true>(r, invr, rsafe, dx, dy, dz, h, invh, Q.regular, w, x, y, z);
        else side64<KT, false>(r, invr, rsafe, dx, dy, dz, h, invh, Q.regular, w, x, y, z);
    };
    if (STRAT == SYMMETRIC) {
        double Wa, ax, ay, az, Wb, bx, by, bz;
        side(Q.ha, Q.invha, Wa, ax, ay, az);
        side(N.L.w, N.X.x, Wb, bx, by, bz);
        W = 0.5 * (Wa + Wb);
        gx = 0.5 * (ax + bx); gy = 0.5 * (ay + by); gz = 0.5 * (az + bz);
    } else if (STRAT == GATHER) {
        side(Q.ha, Q.invha, W, gx, gy, gz);
    } else {
        side(N.L.w, N.X.x, W, gx, gy, gz);
    }
    const double mW = mb * W;
    const double w = div_by(mW, rb, invrb, Q.regular && exp_safe(mW));
    put(0, w);
#pragma unroll
    for (int u = 0; u < MAXU; ++u)
        if (row_of<CAT>(1 + u) >= 0) put(1 + u, N.A[u] * w);
    if (!grad) {
        if (any_cat)
            for (int a = 5; a < NT; ++a) put(a, 0.0);
        return;
    }
    const double ml = mb * invrb;
    const double qx = ml * gx, qy = ml * gy, qz = ml * gz;
    put(5, qx); put(6, qy); put(7, qz);
    if (any_cat && C.n_grad > 0 && C.g_u[0] < 0) {   // density gradient
        const double mx = mb * gx, my = mb * gy, mz = mb * gz;
        put(8, mx); put(9, my); put(10, mz);
        put(11, mx * invrb); put(12, my * invrb); put(13, mz * invrb);
        put(14, mW);
    } else {
        if (row_of<CAT>(8) >= 0) {
            const bool on = CatShape<CAT>::grad(C);   // the gradient's column is in slot 0
            put(8, on ? qx * N.A[0] : 0.0);
            put(9, on ? qy * N.A[0] : 0.0);
            put(10, on ? qz * N.A[0] : 0.0);
        }
        if (any_cat)
            for (int a = 11; a < 15; ++a) put(a, 0.0);
    }
    const double ax = N.A[1], ay = N.A[2], az = N.A[3];   // the divergence/curl vector
    if (row_of<CAT>(15) >= 0) put(15, CatShape<CAT>::div(C) ? qx * ax + qy * ay + qz * az : 0.0);
    if (row_of<CAT>(16) >= 0) {
        const bool on = CatShape<CAT>::curl(C);
        put(16, on ? ay * qz - az * qy : 0.0);
        put(17, on ? az * qx - ax * qz : 0.0);
        put(18, on ? ax * qy - ay * qx : 0.0);
    }
}

__device__ __forceinline__ void finalize64(const double *v, const DevCatalog &C, int64_t qi)
{
    Exact64 A;
    A.S1 = v[0];
#pragma unroll
    for (int u = 0; u < MAXU; ++u) A.SA[u] = v[1 + u];
    A.Bq[0] = v[5]; A.Bq[1] = v[6]; A.Bq[2] = v[7];
    A.Fg[0][0] = v[8]; A.Fg[0][1] = v[9]; A.Fg[0][2] = v[10];
    A.Bd[0] = v[11]; A.Bd[1] = v[12]; A.Bd[2] = v[13];
    A.Sd = v[14];
    A.D[0] = v[15];
    A.Cc[0][0] = v[16]; A.Cc[0][1] = v[17]; A.Cc[0][2] = v[18];
    A.finalize(C, qi);
}

// the warp's accumulators (lane k: term row k) to the query's outputs
template <int CAT>
__device__ __forceinline__ void store_sums64(double acc, const DevCatalog &C, int64_t qi, int lane)
{
    double v[NT];
#pragma unroll
    for (int a = 0; a < NT; ++a) {
        const int k = row_of<CAT>(a);
        v[a] = k >= 0 ? __shfl_sync(0xffffffffu, acc, k) : 0.0;
    }
    if (lane == 0) finalize64(v, C, qi);
}

// Sums of one query over batches of up to 32 accepted leaves.  A batch's neighbour records are
// loaded first, the previous batch's terms are added while the loads are in flight, and the
// new terms then take their place in the warp's buffer.
template <int STRAT, int KT, int CAT>
struct Sum64 {
    const DevTree &T;
    const DevCatalog &C;
    const Query64 &Q;
    double *buf;       // the warp's term buffer
    const double *row; // this lane's row of it
    int lane, pending = 0;
    double acc = 0.0;  // lane k < nterms64 owns the accumulator of term row k

    __device__ __forceinline__ Sum64(const DevTree &t, const DevCatalog &c, const Query64 &q, double *b, int l)
        : T(t), C(c), Q(q), buf(b), lane(l)
    {
        row = buf + lane * TROW;
    }
    __device__ __forceinline__ void batch(int fill, int64_t b)
    {
        Nb64 N;
        if (b >= 0) load_nb64<CAT>(T, C, b, N);
        // only the last batch of a query is partial; lanes without a row stay out of the loads
        // (each quarter-warp with an active lane costs a shared-memory wavefront)
        if (pending && lane < nterms64<CAT>()) acc = add_row(row, 32, acc);
        __syncwarp();
        if (b >= 0) terms64<STRAT, KT, CAT>(C, Q, N, buf + lane);
        __syncwarp();
        pending = fill;
    }
    __device__ __forceinline__ void finish(int64_t qi)
    {
        if (pending && lane < nterms64<CAT>()) acc = add_row(row, pending, acc);
        __syncwarp();
        store_sums64<CAT>(acc, C, qi, lane);
    }
};

// The fused FP64 sum of one query: the warp walks the tree (warp-uniform next_item), deals the
// accepted leaves to its lanes and sums them (Sum64).  sterm is the warp's buffer of TBUF doubles,
// bnear the nearest sorted leaf (-1 for itpScatter), leaf_size the walk's linear-scan cutoff.
template <int STRAT, int KT>
__device__ __forceinline__ void points64_query(const DevTree &T, const DevCatalog &C, double px, double py, double pz,
                                               int64_t bnear, int64_t qi, double *sterm, int lane, int leaf_size)
{
    const int64_t n = T.n;
    const double K = kernel_valid(KT);
    const Query64 Q = make_query64<STRAT>(T, px, py, pz, bnear);
    const double ra = __dmul_rn(K, Q.ha), r2a = __dmul_rn(ra, ra);
    Sum64<STRAT, KT, CAT_ANY> A(T, C, Q, sterm, lane);
    Slots S{0, -1};
    auto proc = [&](int fill) { A.batch(fill, S.mine); };
    if (T.root == 0) {
        double4 L;
        double d2;
        if (single_leaf_accepted<STRAT>(T, px, py, pz, K, r2a, L, d2)) deal(S, lane, 0, 0, proc);
    } else {
        Walk w{T.root, 1, 0, 0, 4 * n + 64};
        int64_t lo, hi;
        while (next_item<STRAT>(T, w, px, py, pz, K, r2a, lo, hi, leaf_size)) deal(S, lane, lo, hi, proc);
    }
    if (S.fill > 0) proc(S.fill);
    A.finish(qi);
}

// The two-phase FP64 sum of one walked query j (its runs in the pool P) at sample point qi:
// the accepted leaves dealt in DFS order, the terms and in-order sums of points64_query.
template <int STRAT, int KT, int CAT>
__device__ __forceinline__ void pairs64_query(const DevTree &T, const DevCatalog &C, const RunPool &P, int64_t j,
                                              int64_t qi, double px, double py, double pz, int64_t bnear,
                                              double *sterm, int lane)
{
    const Query64 Q = make_query64<STRAT>(T, px, py, pz, bnear);
    Sum64<STRAT, KT, CAT> A(T, C, Q, sterm, lane);
    auto first = [&](int64_t) {};
    auto one = [&](int64_t b) { A.batch(32, b); };
    auto cantwo = [&]() { return false; };
    // never called (cantwo and canfour are false)
    auto two = [&](int64_t) {};
    auto four = [&](int64_t) {};
    int mine = -1;
    const int fill = deal_runs(P, j, lane, first, one, two, cantwo, four, cantwo, mine);
    if (fill > 0) A.batch(fill, mine);
    A.finish(qi);
}

// The same sum by a block of four warps for a query with many neighbours: three warps compute
// the terms of every third batch each into a double-buffered set of term buffers, the fourth
// adds the three batches of the round before, in batch order.  A warp on its own needs the
// latency of a batch's loads and terms plus 32 dependent additions (9 cycles each) per batch;
// here only the additions remain in the chain, so the few heaviest queries of an uneven set do
// not decide when the launch ends (153,600 points with 5.7e8 pairs, up to 4e5 in one query:
// 18.8 -> 10.0 ms).  With enough such queries to fill the chip the warps' own form has the
// higher rate (2.8e9 pairs even out: 37 ms against 49 ms), hence the rule on an even share.  Every warp passes `rounds` barriers whatever it is dealt.  cnt is the query's
// number of accepted leaves; buf holds BLOCK64_BUFS term buffers.
constexpr int BLOCK64_PROD = 3;
constexpr int BLOCK64_BUFS = 2 * BLOCK64_PROD;

template <int STRAT, int KT, int CAT>
__device__ __forceinline__ void pairs64_block(const DevTree &T, const DevCatalog &C, const RunPool &P, int64_t j,
                                              int64_t qi, double px, double py, double pz, int64_t bnear, int cnt,
                                              double *buf, int warp, int lane)
{
    constexpr int NR = nterms64<CAT>(), SZ = NR * TROW;
    const int nb = (cnt + 31) >> 5, rounds = (nb + BLOCK64_PROD - 1) / BLOCK64_PROD;
    if (warp < BLOCK64_PROD) {
        const Query64 Q = make_query64<STRAT>(T, px, py, pz, bnear);
        int r = 0;
        auto batch = [&](int64_t b) {
            if (r >= rounds) return;
            if (b >= 0) {
                Nb64 N;
                load_nb64<CAT>(T, C, b, N);
                terms64<STRAT, KT, CAT>(C, Q, N, buf + ((r & 1) * BLOCK64_PROD + warp) * SZ + lane);
            }
            __syncwarp();
            __syncthreads();
            ++r;
        };
        int mine = -1;
        const int fill = deal_runs_part<BLOCK64_PROD>(P, j, lane, warp, batch, mine);
        if (fill > 0) batch(mine);
        while (r < rounds) {   // no batch of this warp in the last round
            __syncthreads();
            ++r;
        }
    } else {
        double acc = 0.0;   // lane k < NR owns the accumulator of term row k
        for (int r = 0; r < rounds; ++r) {
            __syncthreads();   // the round's terms are in place
            if (lane < NR)
                for (int w = 0; w < BLOCK64_PROD; ++w) {
                    const int left = cnt - 32 * (r * BLOCK64_PROD + w);
                    if (left <= 0) break;
                    acc = add_row(buf + ((r & 1) * BLOCK64_PROD + w) * SZ + lane * TROW, left < 32 ? left : 32, acc);
                }
            __syncwarp();
        }
        store_sums64<CAT>(acc, C, qi, lane);
    }
}

}  // namespace pb
