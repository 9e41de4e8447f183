// pb_lines.cu -- line-integrated (column) interpolation, itpScatter (both precision modes).
// One thread per line walking the tree with an FP64 node bound was bound by that bound (six
// divisions, two square roots a node) and by latency (5 % of the warp slots for a small image):
// 1.5e6 particles on 1024^2 lines 54.6 ms, 20,011 particles on 97 x 61 oblique lines 3.18 ms.  Now
// 9.3 ms (FP64 pipe 32 % active; the sums of 6e8 accepted pairs are most of it) and 0.20 ms.
// Compiled with -fmad=false: every expression is the IEEE result of the reference's operation
// order.
#include "line_tables.h"
#include "pb_internal.h"
#include "pb_interp_impl.cuh"

namespace pb {

__device__ const double g_line_inorm64[6][PB_LINE_NTAB] = PB_LINE_INORM_INIT;

// --------------------------------------------------------------------------------------
// Node bound of a line.  The box is projected on the plane normal to the line: with u, v
// orthonormal and normal to the unit direction, every point of the box is at least
// max(|u.(c - o)| - |u|.e, 0) along u (c the box's centre, e its half extents) and likewise along v
// from the line.  FP32, with the origin moved along the line next to the particles' box so that the
// offsets stay small; `eu0` and `ev0` bound the rounding of the projections and `slack` the cancellation
// in d2_line's difference (measured from the caller's origin), so a node is pruned only if
// d2_line exceeds the radius of every leaf in it.  29 FP32 operations a node; the FP64 slab and
// sphere bound (d2_line_box_lower) took six divisions and two square roots.  Directions
// that are not unit vectors to 1e-12 keep that one, as d2_line is not their distance, and so do trees with
// a negative h, where a leaf's radius may exceed its nodes' and the bound decides which leaves are reached.
struct LineBound {
    float ox, oy, oz, ux, uy, uz, vx, vy, vz, eu0, ev0, slack;   // eu0, ev0: added to the half extents
    bool plane;   // the FP32 bound holds; else d2_line_box_lower is taken
};

__device__ __forceinline__ LineBound make_line_bound(const DevTree &T, const double o[3], const double m[3])
{
    LineBound B;
    const double m2 = m[0] * m[0] + m[1] * m[1] + m[2] * m[2];
    B.plane = fabs(m2 - 1.0) <= 1e-12 && !(__ldg(T.odd) & ODD_NEGATIVE_H);
    const NodeF nd = load_node(T.node + (T.root - 1));
    const double lo[3] = {(double)nd.lox, (double)nd.loy, (double)nd.loz}, hi[3] = {(double)nd.hix, (double)nd.hiy, (double)nd.hiz};
    double c[3], t = 0.0, far2 = 0.0, rad2 = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        c[d] = 0.5 * (lo[d] + hi[d]);
        const double h = 0.5 * (hi[d] - lo[d]), q = c[d] - o[d];
        t += q * m[d];
        far2 += q * q;
        rad2 += h * h;
    }
    // u: the direction crossed with the axis it is least along (the image's own axis for a line
    // along an axis), v = m x u
    const double a0 = fabs(m[0]), a1 = fabs(m[1]), a2 = fabs(m[2]);
    double u[3];
    if (a0 <= a1 && a0 <= a2) { u[0] = 0.0; u[1] = m[2]; u[2] = -m[1]; }
    else if (a1 <= a2) { u[0] = -m[2]; u[1] = 0.0; u[2] = m[0]; }
    else { u[0] = m[1]; u[1] = -m[0]; u[2] = 0.0; }
    const double inv = 1.0 / sqrt(u[0] * u[0] + u[1] * u[1] + u[2] * u[2]);
    u[0] *= inv; u[1] *= inv; u[2] *= inv;
    const double v[3] = {m[1] * u[2] - m[2] * u[1], m[2] * u[0] - m[0] * u[2], m[0] * u[1] - m[1] * u[0]};
    double p[3], size = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        p[d] = o[d] + t * m[d];
        size += fabs(p[d]) + fmax(fabs(lo[d]), fabs(hi[d]));
    }
    B.ox = (float)p[0]; B.oy = (float)p[1]; B.oz = (float)p[2];
    B.ux = (float)u[0]; B.uy = (float)u[1]; B.uz = (float)u[2];
    B.vx = (float)v[0]; B.vy = (float)v[1]; B.vz = (float)v[2];
    // at most 16 roundings of values up to `size` in a projection, and the origin's move along the
    // line, whose rounding grows with the distance moved
    const double far = sqrt(far2) + sqrt(rad2);
    B.eu0 = B.ev0 = (float)(9.6e-7 * size + 1e-14 * far);
    B.slack = (float)(1.1e-12 * far * far + 1e-37);
    return B;
}

__device__ __forceinline__ bool line_pruned(const LineBound &B, const NodeF &nd, float K, float hmax)
{
    const float cx = fmaf(0.5f, nd.lox + nd.hix, -B.ox), cy = fmaf(0.5f, nd.loy + nd.hiy, -B.oy),
                cz = fmaf(0.5f, nd.loz + nd.hiz, -B.oz);
    const float ex = 0.5f * (nd.hix - nd.lox), ey = 0.5f * (nd.hiy - nd.loy), ez = 0.5f * (nd.hiz - nd.loz);
    const float pu = fmaf(B.uz, cz, fmaf(B.uy, cy, B.ux * cx)), pv = fmaf(B.vz, cz, fmaf(B.vy, cy, B.vx * cx));
    const float eu = fmaf(fabsf(B.uz), ez, fmaf(fabsf(B.uy), ey, fmaf(fabsf(B.ux), ex, B.eu0)));
    const float ev = fmaf(fabsf(B.vz), ez, fmaf(fabsf(B.vy), ey, fmaf(fabsf(B.vx), ex, B.ev0)));
    const float gu = fmaxf(fabsf(pu) - eu, 0.f), gv = fmaxf(fabsf(pv) - ev, 0.f);
    const float r = K * hmax;
    return fmaf(gv, gv, gu * gu) > fmaf(r * r, 1.000002f, B.slack);
}

// the line-integrated kernel's table of this launch: values, support radius, step and 1/step
struct LineTable {
    const double *I;
    double K, dq, inv_dq;
};

__device__ __forceinline__ LineTable make_line_table(const double *table, int kernel)
{
    const double K = kernel_valid(kernel), dq = K / double(PB_LINE_NTAB_DEV - 1);
    return LineTable{table + (int64_t)kernel * PB_LINE_NTAB_DEV, K, dq, 1.0 / dq};
}

// m W / rho of an accepted leaf with aux record X (line_integrated_kernel.jl:132-137); q / dq and
// m W / rho are taken in the short correctly rounded form (div_by)
__device__ __forceinline__ double line_weight(const double4 &X, const LineTable &lt, bool regular, double d2)
{
    const double dr = sqrt(d2 > 0.0 ? d2 : 0.0);
    const double q = dr * X.x;
    double Iq = 0.0;
    if (!(q >= lt.K)) {
        const double idxf = div_by(q, lt.dq, lt.inv_dq, exp_safe(q)) + 1.0;
        int i = (int)idxf;
        i = i < 1 ? 1 : (i > PB_LINE_NTAB_DEV - 1 ? PB_LINE_NTAB_DEV - 1 : i);
        const double t = idxf - double(i);
        Iq = __ldg(lt.I + i - 1) * (1.0 - t) + __ldg(lt.I + i) * t;
    }
    const double mW = X.z * (X.x * Iq);
    return div_by(mW, X.w, X.y, regular && exp_safe(mW));
}

__device__ __forceinline__ double leaf_radius2(double K, double h)
{
    const double r = __dmul_rn(K, h);
    return __dmul_rn(r, r);
}

// Stack of tree entries of a warp that walks the tree for a line or a tile of lines.  Its top is the
// next entry in DFS order: a node or leaf id, or an accepted leaf (negative).  A round takes the
// top 32 entries (visit decides what becomes of each: 0, itself, or its two children) and moves the
// accepted leaves before the first node still open to `next`, in DFS order.
constexpr int LSTACK = 512;   // entries; taken one at a time above LSTACK - 160, where a round adds at most one

struct LineWalk {
    int *stack, *next;   // LSTACK and 64 ints of shared memory
    int lane, size, fill;
    int64_t guard, limit;

    __device__ __forceinline__ void start(const DevTree &T)
    {
        size = 1;
        fill = 0;
        guard = 0;
        limit = 4 * T.n + 64;
        if (lane == 0) stack[0] = T.root;
        __syncwarp();
    }
    // visit(e, e0, e1): number of entries (0, 1, 2) that replace entry e >= 0; an accepted leaf b is
    // returned as one entry, b | 0x80000000
    template <typename VISIT>
    __device__ __forceinline__ bool round(const DevTree &T, VISIT &visit)
    {
        if (size <= 0) return false;
        if (++guard > limit || size > LSTACK - 2) {
            flag(T.status, ST_TRAVERSAL);
            return false;
        }
        const int k = size > LSTACK - 160 ? 1 : (size < 32 ? size : 32);
        const unsigned below = (1u << lane) - 1u;
        int c = 0, e0 = 0, e1 = 0;
        if (lane < k) {
            const int e = stack[size - 1 - lane];
            if (e < 0) {
                c = 1;
                e0 = e;
            } else {
                c = visit(e, e0, e1);
            }
        }
        __syncwarp();
        const unsigned open = __ballot_sync(0xffffffffu, c == 2);
        const int first = open ? __ffs(open) - 1 : 32;
        const unsigned done = __ballot_sync(0xffffffffu, c == 1 && lane < first);
        if (c == 1 && lane < first) next[fill + __popc(done & below)] = e0 & 0x7fffffff;
        fill += __popc(done);
        const unsigned kept = __ballot_sync(0xffffffffu, c >= 1 && lane >= first);
        size += __popc(kept) + __popc(open) - k;
        if (c >= 1 && lane >= first) {
            const int at = size - 1 - __popc(kept & below) - __popc(open & below);
            stack[at] = e0;
            if (c == 2) stack[at - 1] = e1;
        }
        __syncwarp();
        return true;
    }
    // the first 32 leaves of next[] have been used
    __device__ __forceinline__ void advance()
    {
        fill -= 32;
        const int v = next[32 + lane];
        __syncwarp();
        next[lane] = v;
        __syncwarp();
    }
};

// One line by a warp: its lanes walk (LineWalk), compute the terms of 32 accepted leaves at once, and
// lane k adds term k of each in DFS order -- the sums of one thread walking the tree.
constexpr int LROWS = 1 + MAXS;
constexpr int LROW = 34;   // doubles per term row (16-byte reads of eight lanes on different banks)

__device__ __forceinline__ void line_by_warp(const DevTree &T, const DevCatalog &C, const LineTable &lt, bool regular,
                                             const double o[3], const double m[3], int64_t li, LineWalk &Wk,
                                             double *term)
{
    const int lane = Wk.lane, n = (int)T.n;
    const float Kf = (float)lt.K;
    double acc = 0.0;   // lane k < LROWS: sum of term row k
    auto sum = [&](int f) {   // the first f leaves of next[]
        if (lane < f) {
            const int64_t b = Wk.next[lane];
            const double4 L = ldg4(T.leaf + b);
            const double w = line_weight(ldg4(T.aux + b), lt, regular, d2_line(L.x, L.y, L.z, o, m));
            term[lane] = w;
#pragma unroll
            for (int s = 0; s < MAXS; ++s)
                if (s < C.n_scalar) term[(1 + s) * LROW + lane] = __ldg(C.ucol[C.s_u[s]] + b) * w;
        }
        __syncwarp();
        if (lane <= C.n_scalar) acc = add_row(term + lane * LROW, f, acc);
        __syncwarp();
    };
    if (T.root == 0) {
        const double4 L = ldg4(T.leaf);
        if (d2_line(L.x, L.y, L.z, o, m) <= leaf_radius2(lt.K, L.w)) {
            Wk.next[0] = 0;
            __syncwarp();
            sum(1);
        }
    } else {
        const LineBound B = make_line_bound(T, o, m);
        auto visit = [&](int e, int &e0, int &e1) {
            if (e >= n) {
                const double4 L = ldg4(T.leaf + (e - n));
                e0 = (int)((unsigned)(e - n) | 0x80000000u);
                return d2_line(L.x, L.y, L.z, o, m) <= leaf_radius2(lt.K, L.w) ? 1 : 0;
            }
            const NodeF nd = load_node(T.node + (e - 1));
            const float hm = __ldg(T.node_hmax + (e - 1));
            const int2 ch = __ldg(T.child + (e - 1));
            e0 = ch.x;
            e1 = ch.y;
            const bool prune = B.plane ? line_pruned(B, nd, Kf, hm) : d2_line_box_lower(o, m, nd) > leaf_radius2(lt.K, (double)hm);
            return prune ? 0 : 2;
        };
        Wk.start(T);
        while (Wk.round(T, visit))
            if (Wk.fill >= 32) {
                sum(32);
                Wk.advance();
            }
        if (Wk.fill > 0) sum(Wk.fill);
    }
    const double S1 = __shfl_sync(0xffffffffu, acc, 0);
    if (lane >= 1 && lane <= C.n_scalar) {
        double v = acc;
        if (S1 == 0.0) v = __longlong_as_double(0x7ff8000000000000LL);
        else if (C.s_shep[lane - 1]) v = acc * (1.0 / S1);
        C.out[lane - 1][li] = v;
    }
}

// rest: the number of tiles and the tiles (of k_lines_tile) whose lines are taken; NULL: all lines
__global__ void __launch_bounds__(128) k_lines_warp(DevTree T, DevCatalog C, int64_t nl, const double *__restrict__ ox,
                                                    const double *__restrict__ oy, const double *__restrict__ oz,
                                                    const double *__restrict__ mx, const double *__restrict__ my,
                                                    const double *__restrict__ mz, const uint32_t *__restrict__ perm,
                                                    const double *__restrict__ table, unsigned long long *counter,
                                                    const uint32_t *__restrict__ rest)
{
    __shared__ int s_stack[4][LSTACK], s_next[4][64];
    __shared__ __align__(16) double s_term[4][LROWS * LROW];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    LineWalk Wk{s_stack[wib], s_next[wib], lane};
    const LineTable lt = make_line_table(table, T.kernel);
    const bool regular = __ldg(T.odd) == 0;
    const int64_t todo = rest ? 32 * (int64_t)__ldg(rest) : nl;
    unsigned long long nxt = 0;
    if (lane == 0) nxt = atomicAdd(counter, 1ULL);
    for (;;) {
        int64_t j = (int64_t)__shfl_sync(0xffffffffu, nxt, 0);
        if (j >= todo) break;
        if (lane == 0) nxt = atomicAdd(counter, 1ULL);
        if (rest) {
            j = (int64_t)__ldg(rest + 1 + (j >> 5)) * 32 + (j & 31);
            if (j >= nl) continue;   // past the last line of the last tile
        }
        const int64_t li = perm ? (int64_t)__ldg(perm + j) : j;
        if (li >= nl) continue;   // unreachable for a valid permutation
        const double o[3] = {__ldg(ox + li), __ldg(oy + li), __ldg(oz + li)};
        const double m[3] = {__ldg(mx + li), __ldg(my + li), __ldg(mz + li)};
        line_by_warp(T, C, lt, regular, o, m, li, Wk, s_term[wib]);
    }
}

// A tile of 32 lines of one direction by a warp: it walks the tree once for the rectangle the lines
// pierce in the plane normal to them and stages 32 of the leaves so found at a time.  Every lane marks
// the staged leaves near its own line (an FP32 test in the plane that errs on the safe side), then
// takes its marked ones in DFS order: the exact test, the term, the sums.  Two leaves are in flight
// per lane: a term is a chain of a square root, two table loads and two quotients.  Lines of different
// directions, and tiles whose lines share few of their leaves (fewer than 1 in LTILE_SHARE tests passed after
// LTILE_PROBE leaves, and after twice as many, and so on: a tile that lies across a jump of the Morton
// order, or lines in no order at all), are left to k_lines_warp, tile by tile in `rest`.  Taking them here,
// 32 lines one after the other, made one warp the end of the launch: 363^2 lines of 1.5e6 particles (M5) 36.3 ms,
// now 6.7; 400^2 with origins at scattered depths 50.2, now 13.1.  Shares of 4 / 8 / 12 / 16 / 32: 363^2 6.9 / 6.3 /
// 6.7 / 7.3 / 8.2, 400^2 at depths 12.9 / 12.6 / 13.1 / 14.3 / 18.3, 1024^2 17.3 / 16.6 / 16.7 / 16.6 / 16.6 ms; with M4
// 1024^2 11.88 / 11.85 / 11.81 at 8 / 12 / 16, 400^2 at depths 8.8 / 9.5 / 10.4.
// 3 / 4 / 5 / 6 blocks of 128 per SM (M4, 1.5e6 particles): 1024^2 lines 14.4 / 11.8 / 11.0 / 11.4 ms, 400^2 lines
// 4.7 / 5.0 at 4 / 5; 20,011 particles, 400^2 0.58 / 0.65: four are the best where the chip is not full.
constexpr int LTILE_PROBE = 512, LTILE_SHARE = 12;
constexpr int LREC = 14;   // doubles per staged leaf: x, y, z, (K h)^2, the aux record, four columns; two of padding

// WEIGH estimates the tiles' work instead, for the order they are taken in: the leaves of the subtrees of
// at most `cut` leaves that the tile's rectangle reaches (keys: 8 bits, heaviest first; vals: the tile).
template <bool WEIGH>
__global__ void __launch_bounds__(128, 4) k_lines_tile(DevTree T, DevCatalog C, int64_t nl, const double *__restrict__ ox,
                                                    const double *__restrict__ oy, const double *__restrict__ oz,
                                                    const double *__restrict__ mx, const double *__restrict__ my,
                                                    const double *__restrict__ mz, const uint32_t *__restrict__ perm,
                                                    const double *__restrict__ table, unsigned long long *counter,
                                                    const uint32_t *__restrict__ order, int cut, uint32_t *keys,
                                                    uint32_t *vals, uint32_t *rest)
{
    __shared__ int s_stack[4][LSTACK], s_next[4][64];
    __shared__ __align__(16) double s_rec[4][32 * LREC];
    __shared__ __align__(16) float4 s_pos[4][32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, n = (int)T.n;
    LineWalk Wk{s_stack[wib], s_next[wib], lane};
    double *rec = s_rec[wib];
    float4 *pos = s_pos[wib];
    const LineTable lt = make_line_table(table, T.kernel);
    const float Kf = (float)lt.K;
    const bool regular = __ldg(T.odd) == 0;
    const int64_t ntile = (nl + 31) / 32;
    unsigned long long nxt = 0;
    if (lane == 0) nxt = atomicAdd(counter, 1ULL);
    for (;;) {
        const int64_t k = (int64_t)__shfl_sync(0xffffffffu, nxt, 0);
        if (k >= ntile) break;
        if (lane == 0) nxt = atomicAdd(counter, 1ULL);
        const int64_t t = !WEIGH && order ? (int64_t)__ldg(order + k) : k;
        // lanes past the last line repeat it and store nothing
        const bool live = t * 32 + lane < nl;
        const int64_t j = live ? t * 32 + lane : nl - 1;
        int64_t li = perm ? (int64_t)__ldg(perm + j) : j;
        if (li >= nl) li = 0;   // unreachable for a valid permutation
        const double o[3] = {__ldg(ox + li), __ldg(oy + li), __ldg(oz + li)};
        const double m[3] = {__ldg(mx + li), __ldg(my + li), __ldg(mz + li)};
        bool same = T.root != 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double m0 = __shfl_sync(0xffffffffu, m[d], 0);   // every lane takes part
            same = same && m[d] == m0;
        }
        bool tiled = __all_sync(0xffffffffu, same);
        unsigned weight = 0;
        if (tiled) {
            LineBound B = make_line_bound(T, o, m);   // u, v are the same in every lane
            tiled = __all_sync(0xffffffffu, B.plane);
            // the lines' positions in the plane, relative to the first one's, and their rectangle
            const float px = __shfl_sync(0xffffffffu, B.ox, 0), py = __shfl_sync(0xffffffffu, B.oy, 0),
                        pz = __shfl_sync(0xffffffffu, B.oz, 0);
            const float dx = B.ox - px, dy = B.oy - py, dz = B.oz - pz;
            const float a = fmaf(B.uz, dz, fmaf(B.uy, dy, B.ux * dx)), b = fmaf(B.vz, dz, fmaf(B.vy, dy, B.vx * dx));
            float amin = a, amax = a, bmin = b, bmax = b, eps = B.eu0, slack = B.slack;
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                amin = fminf(amin, __shfl_xor_sync(0xffffffffu, amin, s));
                amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, s));
                bmin = fminf(bmin, __shfl_xor_sync(0xffffffffu, bmin, s));
                bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, s));
                eps = fmaxf(eps, __shfl_xor_sync(0xffffffffu, eps, s));
                slack = fmaxf(slack, __shfl_xor_sync(0xffffffffu, slack, s));
            }
            const float ac = 0.5f * (amin + amax), bc = 0.5f * (bmin + bmax);
            B.ox = fmaf(bc, B.vx, fmaf(ac, B.ux, px));
            B.oy = fmaf(bc, B.vy, fmaf(ac, B.uy, py));
            B.oz = fmaf(bc, B.vz, fmaf(ac, B.uz, pz));
            // three more roundings of the lines' positions, each below eps
            B.eu0 = fmaf(0.5f, amax - amin, 4.f * eps);
            B.ev0 = fmaf(0.5f, bmax - bmin, 4.f * eps);
            B.slack = slack;
            if (WEIGH) {
                auto weigh = [&](int e, int &e0, int &e1) {
                    if (e >= n) {
                        weight += 1u;
                        return 0;
                    }
                    if (line_pruned(B, load_node(T.node + (e - 1)), Kf, __ldg(T.node_hmax + (e - 1)))) return 0;
                    const int2 r = __ldg(T.range + (e - 1)), ch = __ldg(T.child + (e - 1));
                    if (r.y - r.x < cut) {
                        weight += (unsigned)(r.y - r.x + 1);
                        return 0;
                    }
                    e0 = ch.x;
                    e1 = ch.y;
                    return 2;
                };
                if (tiled) {
                    Wk.start(T);
                    while (Wk.round(T, weigh)) {}
                }
                weight = __reduce_add_sync(0xffffffffu, weight);
            } else {
                double S1 = 0.0, acc[MAXS];
#pragma unroll
                for (int s = 0; s < MAXS; ++s) acc[s] = 0.0;
                int tested = 0, passed = 0;
                // this line's position relative to the rectangle's centre
                const float al = a - ac, bl = b - bc;
                auto sum = [&](int f) {   // the first f leaves of next[]
                    if (lane < f) {
                        const int64_t b = Wk.next[lane];
                        const double4 L = ldg4(T.leaf + b), X = ldg4(T.aux + b);
                        double *r = rec + lane * LREC;
                        r[0] = L.x; r[1] = L.y; r[2] = L.z; r[3] = leaf_radius2(lt.K, L.w);
                        r[4] = X.x; r[5] = X.y; r[6] = X.z; r[7] = X.w;
#pragma unroll
                        for (int s = 0; s < MAXS; ++s) r[8 + s] = s < C.n_scalar ? __ldg(C.ucol[C.s_u[s]] + b) : 0.0;
                        const float cx = (float)L.x - B.ox, cy = (float)L.y - B.oy, cz = (float)L.z - B.oz;
                        const float rr = fmaf(Kf, __double2float_ru(fabs(L.w)), 8.f * eps);
                        pos[lane] = make_float4(fmaf(B.uz, cz, fmaf(B.uy, cy, B.ux * cx)),
                                                fmaf(B.vz, cz, fmaf(B.vy, cy, B.vx * cx)), fmaf(rr * rr, 1.000002f, slack), 0.f);
                    }
                    __syncwarp();
                    unsigned near = 0;
                    for (int i = 0; i < f; ++i) {
                        const float4 p = pos[i];
                        const float da = p.x - al, db = p.y - bl;
                        near |= (!(fmaf(db, db, da * da) > p.z) ? 1u : 0u) << i;
                    }
                    passed += __popc(near);
                    auto term = [&](int i, double *A) {   // w (0 if the exact test fails) and the columns
                        const double2 *r = reinterpret_cast<const double2 *>(rec + i * LREC);
                        const double2 xy = r[0], zr = r[1], p = r[2], q = r[3];
                        const double d2 = d2_line(xy.x, xy.y, zr.x, o, m);
                        const bool in = d2 <= zr.y;
                        const double w = line_weight(make_double4(p.x, p.y, q.x, q.y), lt, regular, d2);
#pragma unroll
                        for (int s = 0; s < MAXS; ++s) A[s] = in && s < C.n_scalar ? rec[i * LREC + 8 + s] * w : 0.0;
                        return in ? w : 0.0;   // adding zero leaves a sum as it is
                    };
                    while (near) {
                        const int i0 = __ffs(near) - 1;
                        near &= near - 1;
                        const int i1 = near ? __ffs(near) - 1 : -1;
                        near &= near - 1;
                        double A0[MAXS], A1[MAXS];
                        const double w0 = term(i0, A0), w1 = term(i1 >= 0 ? i1 : i0, A1);
                        S1 += w0;
                        if (i1 >= 0) S1 += w1;
#pragma unroll
                        for (int s = 0; s < MAXS; ++s) {
                            acc[s] += A0[s];
                            if (i1 >= 0) acc[s] += A1[s];
                        }
                    }
                    tested += f;
                    __syncwarp();
                };
                auto visit = [&](int e, int &e0, int &e1) {
                    if (e >= n) {
                        const double4 L = ldg4(T.leaf + (e - n));
                        e0 = (int)((unsigned)(e - n) | 0x80000000u);
                        NodeF nd;   // the leaf's position as an empty box (its rounding is within eu0, ev0)
                        nd.lox = nd.hix = (float)L.x;
                        nd.loy = nd.hiy = (float)L.y;
                        nd.loz = nd.hiz = (float)L.z;
                        return line_pruned(B, nd, Kf, __double2float_ru(fabs(L.w))) ? 0 : 1;
                    }
                    const NodeF nd = load_node(T.node + (e - 1));
                    const float hm = __ldg(T.node_hmax + (e - 1));
                    const int2 ch = __ldg(T.child + (e - 1));
                    e0 = ch.x;
                    e1 = ch.y;
                    return line_pruned(B, nd, Kf, hm) ? 0 : 2;
                };
                if (tiled) {
                    Wk.start(T);
                    while (Wk.round(T, visit))
                        if (Wk.fill >= 32) {
                            sum(32);
                            Wk.advance();
                            if (tested >= LTILE_PROBE && (tested & (tested - 1)) == 0 &&
                                (int64_t)__reduce_add_sync(0xffffffffu, (unsigned)passed) * LTILE_SHARE < (int64_t)tested * 32) {
                                tiled = false;
                                break;
                            }
                        }
                }
                if (tiled) {
                    if (Wk.fill > 0) sum(Wk.fill);
                    if (live) {
#pragma unroll
                        for (int s = 0; s < MAXS; ++s)
                            if (s < C.n_scalar)
                                C.out[s][li] = S1 == 0.0 ? __longlong_as_double(0x7ff8000000000000LL)
                                                         : (C.s_shep[s] ? acc[s] * (1.0 / S1) : acc[s]);
                    }
                }
            }
        }
        if (WEIGH) {
            if (lane == 0) {
                keys[t] = 255u - count_class(tiled ? weight : 0x7fffffffu);   // line by line: the most work
                vals[t] = (uint32_t)t;
            }
            continue;
        }
        if (!tiled && lane == 0) rest[1 + atomicAdd(rest, 1u)] = (uint32_t)t;
    }
}

// Lines from which on the tiles of 32 (in Morton order) fill the chip's warps twice; below, a warp per
// line has more in flight.  Tiles / a warp per line (M5), 256^2, 300^2, 363^2 (131,769) and 512^2 lines: 1.5e6
// particles 6.3 / 4.2, 6.6 / 5.7, 6.3 / 8.3, 6.7 / 16.2 ms; 2e5 2.0 / 2.2, 2.1 / 3.0, 2.2 / 4.4, 2.9 / 8.5;
// 20,011 0.69 / 1.10, 0.76 / 1.47, 0.79 / 2.07, 1.03 / 3.93: one line for all sets, where none is slower by tiles.
constexpr int64_t LINE_TILES_MIN = 131072;
// Particles from which on the tiles are taken by descending estimated work: in Morton order the tiles of
// the densest part, met late, run on alone (SMs active 70 % of the time).  Subtrees of at most
// n / 2^13 leaves are counted whole; n / 2^9 .. n / 2^15 are within 6 %.  Morton order / by work (M4), 1.5e6
// particles: 1024^2 lines face-on 12.1 / 11.8 ms, oblique 12.8 / 12.2, 700^2 oblique 8.2 / 7.3; 2e5 particles: 512^2
// 2.04 / 1.82, but 400^2 1.74 / 1.88; 20,011: 400^2 0.65 / 0.75 (the estimate costs more than it gives).
constexpr int64_t LINE_ORDER_MIN = 262144;
constexpr int LINE_CUT_SHIFT = 13;

cudaError_t launch_lines_fp64(Handle *H, const DevTree &T, const DevCatalog &C, int64_t nl, const double *ox,
                              const double *oy, const double *oz, const double *dx, const double *dy,
                              const double *dz, const uint32_t *perm)
{
    const double *tab = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void **)&tab, g_line_inorm64);
    if (e) return e;
    if ((e = H->counter.reserve(2 * sizeof(unsigned long long)))) return e;
    unsigned long long *ctr = H->counter.as<unsigned long long>();
    if ((e = cudaMemsetAsync(ctr, 0, 2 * sizeof(unsigned long long), H->stream))) return e;
    const bool tiles = nl >= LINE_TILES_MIN && perm;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, H->device);
    auto grid_of = [&](const void *kern, int64_t warps) {
        int per = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, 128, 0);
        return grid_for(warps, 4, sms * (per > 0 ? per : 1));
    };
    const int wgrid = grid_of((const void *)k_lines_warp, nl);
    if (tiles) {
        uint32_t *order = nullptr;
        const int64_t nt = (nl + 31) / 32;
        const int grid = grid_of((const void *)k_lines_tile<false>, nt);
        if ((e = H->line_rest.reserve(4 * (nt + 1)))) return e;
        uint32_t *rest = H->line_rest.as<uint32_t>();
        if ((e = cudaMemsetAsync(rest, 0, 4, H->stream))) return e;
        if (T.n >= LINE_ORDER_MIN) {
            if ((e = H->lpt_k.reserve(4 * nt)) || (e = H->lpt_v.reserve(4 * nt)) || (e = H->lpt_ka.reserve(4 * nt)) ||
                (e = H->lpt_va.reserve(4 * nt)))
                return e;
            uint32_t *k = H->lpt_k.as<uint32_t>(), *v = H->lpt_v.as<uint32_t>();
            k_lines_tile<true><<<grid, 128, 0, H->stream>>>(T, C, nl, ox, oy, oz, dx, dy, dz, perm, tab, ctr, nullptr,
                                                            (int)(T.n >> LINE_CUT_SHIFT), k, v, nullptr);
            if ((e = cudaGetLastError())) return e;
            if ((e = sort_pairs_u32(H, k, v, H->lpt_ka.as<uint32_t>(), H->lpt_va.as<uint32_t>(), nt, 8, &order))) return e;
            if ((e = cudaMemsetAsync(ctr, 0, sizeof(unsigned long long), H->stream))) return e;
            H->launches += 1;
        }
        k_lines_tile<false><<<grid, 128, 0, H->stream>>>(T, C, nl, ox, oy, oz, dx, dy, dz, perm, tab, ctr, order, 0, nullptr,
                                                         nullptr, rest);
        k_lines_warp<<<wgrid, 128, 0, H->stream>>>(T, C, nl, ox, oy, oz, dx, dy, dz, perm, tab, ctr + 1, rest);
        H->launches += 1;
    } else k_lines_warp<<<wgrid, 128, 0, H->stream>>>(T, C, nl, ox, oy, oz, dx, dy, dz, perm, tab, ctr, nullptr);
    H->launches += 1;
    return cudaGetLastError();
}

}  // namespace pb
