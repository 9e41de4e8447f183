// pb_build.cu -- LBVH build on the device, bit-exact against the reference.
//
//   bbox      per-axis min/max (exact in any order)           MortonCode.jl:443-456
//   encode    FP64 (v-vmin)*inv(dv), floor(2097151*f), interleave   MortonCode.jl:209-217,275-305,473-498
//   sort      stable LSD radix sort of (code, index)          == sortperm's index-tie order, MortonCode.jl:182
//   dedupe    c'[i] = i + max_{j<=i}(c[j]-j)                  == the sequential bump, MortonCode.jl:189-193
//   gather    permuted leaves and particle columns            InterpolationInput.jl:211-219, LinearBVH.jl:89-96
//   topology  Karras range/split + internal escapes           BinaryRadixTree.jl:140-260
//   refit     leaf escapes + bottom-up AABB/hmax refit         BinaryRadixTree.jl:262-281, LinearBVH.jl:98-156
//
// Compiled with -fmad=false: the quantisation must be the IEEE result of the reference's
// operation order.
#include <utility>

#include "pb_internal.h"

namespace pb {

// ------------------------------------------------------------------------------------
// bounding box
__global__ void k_bbox_partial(int64_t n, const double *__restrict__ x, const double *__restrict__ y,
                               const double *__restrict__ z, const double *__restrict__ h, double *part,
                               int *status)
{
    double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    int bad = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double v[3] = {x[i], y[i], z[i]};
        if (!isfinite(h[i])) bad = 1;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            if (!isfinite(v[d])) bad = 1;
            if (v[d] < mn[d]) mn[d] = v[d];
            if (v[d] > mx[d]) mx[d] = v[d];
        }
    }
    if (bad) atomicOr(status, ST_NONFINITE);
    __shared__ double s[6][32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        for (int o = 16; o > 0; o >>= 1) {
            double a = __shfl_down_sync(0xffffffffu, mn[d], o);
            double b = __shfl_down_sync(0xffffffffu, mx[d], o);
            if (a < mn[d]) mn[d] = a;
            if (b > mx[d]) mx[d] = b;
        }
    }
    if (lane == 0)
        for (int d = 0; d < 3; ++d) { s[d][w] = mn[d]; s[3 + d][w] = mx[d]; }
    __syncthreads();
    if (threadIdx.x < 6) {
        int d = threadIdx.x;
        double r = s[d][0];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
            double v = s[d][k];
            if (d < 3 ? (v < r) : (v > r)) r = v;
        }
        part[blockIdx.x * 6 + d] = r;
    }
}

// one block of six warps, one per bound
__global__ void __launch_bounds__(192) k_bbox_final(int nparts, const double *part, QuantParams *qp)
{
    __shared__ double s[6];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double r = w < 3 ? INFINITY : -INFINITY;
    for (int b = lane; b < nparts; b += 32) {
        const double v = part[b * 6 + w];
        if (w < 3 ? v < r : v > r) r = v;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double v = __shfl_down_sync(0xffffffffu, r, o);
        if (w < 3 ? v < r : v > r) r = v;
    }
    if (lane == 0) s[w] = r;
    __syncthreads();
    if (threadIdx.x < 3) {
        const int d = threadIdx.x;
        const double mn = s[d], dv = s[3 + d] - mn;
        qp->vmin[d] = mn;
        qp->flat[d] = (dv == 0.0);
        qp->inv[d] = (dv == 0.0) ? 0.0 : 1.0 / dv;
    }
}

cudaError_t launch_bbox(Handle *H, int64_t n, const double *x, const double *y, const double *z, const double *h)
{
    int grid = grid_for(n, 256, 148 * 4);
    cudaError_t e = H->bbox_part.reserve(sizeof(double) * 6 * grid);
    if (e) return e;
    k_bbox_partial<<<grid, 256, 0, H->stream>>>(n, x, y, z, h, H->bbox_part.as<double>(), H->status.as<int>());
    k_bbox_final<<<1, 192, 0, H->stream>>>(grid, H->bbox_part.as<double>(), H->qparams.as<QuantParams>());
    H->launches += 2;
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// quantise + Morton encode
__device__ __forceinline__ uint64_t quantize21(double v, double vmin, double inv, int flat)
{
    const double scale = 2097151.0;   // exp2(21) - 1 (MortonCode.jl:426-434)
    double f = flat ? 0.5 : __dmul_rn(__dsub_rn(v, vmin), inv);
    return (uint64_t)floor(__dmul_rn(scale, f));
}

__global__ void k_encode(int64_t n, const double *__restrict__ x, const double *__restrict__ y,
                         const double *__restrict__ z, const QuantParams *__restrict__ qp, uint64_t *codes,
                         uint32_t *idx)
{
    QuantParams q = *qp;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint64_t ix = quantize21(x[i], q.vmin[0], q.inv[0], q.flat[0]);
        uint64_t iy = quantize21(y[i], q.vmin[1], q.inv[1], q.flat[1]);
        uint64_t iz = quantize21(z[i], q.vmin[2], q.inv[2], q.flat[2]);
        codes[i] = (expand_bits3(ix) << 2) | (expand_bits3(iy) << 1) | expand_bits3(iz);
        idx[i] = (uint32_t)i;
    }
}

cudaError_t launch_encode(Handle *H, int64_t n, const double *x, const double *y, const double *z)
{
    k_encode<<<grid_for(n, 256), 256, 0, H->stream>>>(n, x, y, z, H->qparams.as<QuantParams>(),
                                                       H->codes.as<uint64_t>(), H->idx.as<uint32_t>());
    H->launches += 1;
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Stable LSD radix sort of (key, value) pairs, 8-bit digits, one launch per digit: the digit counts
// of every pass are taken in one read of the keys (they do not depend on the order), and a pass's
// tiles learn how many keys of each digit lie before them by decoupled look-back (D. Merrill, M.
// Garland, "Single-pass parallel prefix scan with decoupled look-back", 2016; A. Adinets, D. Merrill,
// "Onesweep", 2022).  Ranks inside a warp come from eight ballots an item; the tile is put in digit
// order in shared memory first, so that the writes of a digit are contiguous.  It replaces five
// launches a pass (count, three of scan, scatter) whose scatter was bound by the latency of its
// ranking: 4.2e6 keys of 63 bits 0.85 ms, 6,000 keys 0.25 ms; now 0.58 and 0.08 ms.
constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_PASSES = 8;

template <typename K>
__host__ __device__ constexpr int rs_items()   // items per thread: the tile and its counters fit 48 KB of shared memory
{
    return sizeof(K) == 8 ? 12 : 16;
}
template <typename K>
__host__ __device__ constexpr int rs_tile()
{
    return RS_THREADS * rs_items<K>();
}

// digit counts of every pass; a warp whose keys share a digit adds them at once
template <typename K>
__global__ void __launch_bounds__(RS_THREADS) k_rs_hist(int64_t n, const K *__restrict__ keys, int passes, uint32_t *hist)
{
    __shared__ uint32_t sh[RS_PASSES * 256];
    for (int k = threadIdx.x; k < passes * 256; k += RS_THREADS) sh[k] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t nw = (n + 31) & ~int64_t(31);   // whole warps
    for (int64_t i = blockIdx.x * (int64_t)RS_THREADS + threadIdx.x; i < nw; i += (int64_t)gridDim.x * RS_THREADS) {
        const bool valid = i < n;
        const unsigned mask = __ballot_sync(0xffffffffu, valid);
        const K key = valid ? keys[i] : K(0);
        for (int p = 0; p < passes; ++p) {
            const unsigned d = (unsigned)(key >> (8 * p)) & 255u;
            const unsigned d0 = __shfl_sync(0xffffffffu, d, 0);
            if (__all_sync(0xffffffffu, !valid || d == d0)) {
                if (lane == 0) atomicAdd(&sh[p * 256 + d0], (uint32_t)__popc(mask));
            } else if (valid) {
                atomicAdd(&sh[p * 256 + d], 1u);
            }
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < passes * 256; k += RS_THREADS)
        if (sh[k]) atomicAdd(&hist[k], sh[k]);
}

// look-back words: state in the upper half (0 nothing yet, 1 the tile's count, 2 the count up to and
// with the tile), count in the lower
__device__ __forceinline__ unsigned long long rs_word(unsigned state, uint32_t count)
{
    return ((unsigned long long)state << 32) | count;
}

template <typename K>
__global__ void __launch_bounds__(RS_THREADS) k_rs_pass(int64_t n, const K *__restrict__ kin,
                                                        const uint32_t *__restrict__ vin, K *kout, uint32_t *vout,
                                                        int shift, const uint32_t *__restrict__ hist, unsigned *ticket,
                                                        unsigned long long *look, unsigned long long *look_next,
                                                        unsigned wait)
{
    constexpr int ITEMS = rs_items<K>(), TILE = rs_tile<K>();
    __shared__ K s_key[TILE];
    __shared__ uint32_t s_val[TILE];
    __shared__ uint32_t wcnt[RS_WARPS][256];
    __shared__ uint32_t s_base[256];
    __shared__ unsigned long long s_warp[RS_WARPS];
    __shared__ unsigned s_tile;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, d = threadIdx.x;
    // tiles are numbered in the order their blocks start, so the tiles before one are running
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    for (int k = threadIdx.x; k < RS_WARPS * 256; k += RS_THREADS) (&wcnt[0][0])[k] = 0;
    __syncthreads();
    const int64_t tile = s_tile, t0 = tile * TILE;
    const int count = (int)(n - t0 < TILE ? n - t0 : TILE);
    if (count <= 0) return;   // unreachable: one block per tile
    look_next[tile * 256 + d] = 0;   // the next pass's words
    const unsigned below = (1u << lane) - 1u;
    K key[ITEMS];
    uint32_t val[ITEMS], rank[ITEMS];
    const int first = w * (32 * ITEMS) + lane;
#pragma unroll
    for (int c = 0; c < ITEMS; ++c) {
        const bool valid = first + c * 32 < count;
        key[c] = valid ? kin[t0 + first + c * 32] : K(0);
        val[c] = valid ? vin[t0 + first + c * 32] : 0u;
    }
    // rank of every key among the warp's earlier keys of its digit: the lanes with the same digit, then
    // the warp's running count
    unsigned peers[ITEMS];
#pragma unroll
    for (int c = 0; c < ITEMS; ++c) {
        const unsigned dg = (unsigned)(key[c] >> shift) & 255u;
        unsigned p = __ballot_sync(0xffffffffu, first + c * 32 < count);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const unsigned v = __ballot_sync(0xffffffffu, (dg >> b) & 1u);
            p &= (dg >> b) & 1u ? v : ~v;
        }
        peers[c] = p;
    }
#pragma unroll
    for (int c = 0; c < ITEMS; ++c) {
        const unsigned dg = (unsigned)(key[c] >> shift) & 255u;
        const bool valid = first + c * 32 < count;
        const int leader = valid ? __ffs(peers[c]) - 1 : lane;
        uint32_t old = 0;
        if (valid && lane == leader) {
            old = wcnt[w][dg];
            wcnt[w][dg] = old + __popc(peers[c]);
        }
        rank[c] = __shfl_sync(0xffffffffu, old, leader) + __popc(peers[c] & below);
        __syncwarp();
    }
    __syncthreads();
    uint32_t cnt = 0;   // this tile's keys of digit d
#pragma unroll
    for (int k = 0; k < RS_WARPS; ++k) {
        const uint32_t t = wcnt[k][d];
        wcnt[k][d] = cnt;
        cnt += t;
    }
    volatile unsigned long long *words = look;
    words[tile * 256 + d] = rs_word(tile == 0 ? 2 : 1, cnt);
    // exclusive prefix over the digits of the whole input's counts and of this tile's
    const uint32_t tot = hist[d];
    unsigned long long inc = ((unsigned long long)tot << 32) | cnt;   // the lower sum stays below 2^13
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) s_warp[w] = inc;
    __syncthreads();
    for (int k = 0; k < w; ++k) inc += s_warp[k];
    const uint32_t local = (uint32_t)inc - cnt, global = (uint32_t)(inc >> 32) - tot;
    // keys of digit d in the tiles before this one
    uint32_t before = 0;
    for (int64_t t = tile - 1; t >= 0;) {
        unsigned long long v = words[t * 256 + d];
        for (unsigned spin = 0; v >> 32 == 0 && spin < wait; ++spin) v = words[t * 256 + d];
        if (v >> 32 == 0) {
            // hardly ever: that tile is running and waits for nothing before it publishes.  This one then
            // waits no longer and counts the keys of that tile and of those before it itself.
            uint32_t c = 0;
            for (int64_t i = 0; i < (t + 1) * TILE; ++i) c += ((unsigned)(kin[i] >> shift) & 255u) == (unsigned)d;
            v = rs_word(2, c);
        }
        before += (uint32_t)v;
        if (v >> 32 == 2) break;
        --t;
    }
    if (tile > 0) words[tile * 256 + d] = rs_word(2, before + cnt);
    s_base[d] = global + before - local;
    // tile in digit order: position = first of the digit + the warps before + rank
#pragma unroll
    for (int c = 0; c < ITEMS; ++c) {
        const unsigned dg = (unsigned)(key[c] >> shift) & 255u;
        rank[c] += wcnt[w][dg];
    }
    __syncthreads();   // s_warp and wcnt have been read; reuse wcnt[0] for the digits' first positions
    wcnt[0][d] = local;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < ITEMS; ++c) {
        if (first + c * 32 < count) {
            const uint32_t p = wcnt[0][(unsigned)(key[c] >> shift) & 255u] + rank[c];
            if (p < (uint32_t)TILE) {   // always; never write out of bounds
                s_key[p] = key[c];
                s_val[p] = val[c];
            }
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < count; k += RS_THREADS) {
        const K kk = s_key[k];
        const uint32_t pos = s_base[(unsigned)(kk >> shift) & 255u] + (uint32_t)k;
        if (pos < (uint64_t)n) {   // always true for consistent counts
            kout[pos] = kk;
            vout[pos] = s_val[k];
        }
    }
}

// Sorts by the lowest `bits` bits.  The result is in (keys, vals) unless the number of passes is odd and
// `vals_at` is given: then *vals_at says where the values are and the keys are not moved back.
template <typename K>
static cudaError_t sort_pairs(Handle *H, K *keys, uint32_t *vals, K *kalt, uint32_t *valt, int64_t n, int bits,
                              uint32_t **vals_at)
{
    if (vals_at) *vals_at = vals;
    if (n <= 1) return cudaSuccess;
    const int64_t tiles = (n + rs_tile<K>() - 1) / rs_tile<K>();
    const int passes = (bits + 7) / 8;
    // [two sets of look-back words | counts | tickets]; a pass clears the other set for the next one
    const size_t set = sizeof(unsigned long long) * 256 * tiles, head = sizeof(uint32_t) * (256 + 1) * RS_PASSES;
    cudaError_t e = H->hist.reserve(2 * set + head);
    if (e) return e;
    unsigned long long *look[2] = {H->hist.as<unsigned long long>(), H->hist.as<unsigned long long>() + 256 * tiles};
    uint32_t *hist = reinterpret_cast<uint32_t *>(look[1] + 256 * tiles);
    unsigned *ticket = hist + 256 * RS_PASSES;
    // the second set is cleared by the first pass; the counts and tickets lie behind it
    if ((e = cudaMemsetAsync(look[0], 0, set, H->stream))) return e;
    if ((e = cudaMemsetAsync(hist, 0, head, H->stream))) return e;
    k_rs_hist<K><<<grid_for(n, RS_THREADS * 8, 148 * 4), RS_THREADS, 0, H->stream>>>(n, keys, passes, hist);
    K *src = keys, *dst = kalt;
    uint32_t *vs = vals, *vd = valt;
    for (int p = 0; p < passes; ++p) {
        k_rs_pass<K><<<(unsigned)tiles, RS_THREADS, 0, H->stream>>>(n, src, vs, dst, vd, 8 * p, hist + 256 * p, ticket + p,
                                                                   look[p & 1], look[(p + 1) & 1], (unsigned)H->sort_wait);
        std::swap(src, dst);
        std::swap(vs, vd);
    }
    H->launches += 1 + passes;
    if (vals_at) {
        *vals_at = vs;
    } else if (src != keys) {
        cudaMemcpyAsync(keys, src, sizeof(K) * n, cudaMemcpyDeviceToDevice, H->stream);
        cudaMemcpyAsync(vals, vs, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, H->stream);
    }
    return cudaGetLastError();
}

cudaError_t sort_pairs_u64(Handle *H, uint64_t *keys, uint32_t *vals, uint64_t *kalt, uint32_t *valt, int64_t n,
                           int bits, uint32_t **vals_at)
{
    return sort_pairs<uint64_t>(H, keys, vals, kalt, valt, n, bits, vals_at);
}

cudaError_t sort_pairs_u32(Handle *H, uint32_t *keys, uint32_t *vals, uint32_t *kalt, uint32_t *valt, int64_t n,
                           int bits, uint32_t **vals_at)
{
    return sort_pairs<uint32_t>(H, keys, vals, kalt, valt, n, bits, vals_at);
}

// ------------------------------------------------------------------------------------
// duplicate bump as an inclusive max-scan of d[i] = c[i] - i
constexpr int DD_THREADS = 1024, DD_ITEMS = 8, DD_CHUNK = DD_THREADS * DD_ITEMS;

__device__ __forceinline__ int64_t block_inclusive_max(int64_t v, int64_t *total)
{
    __shared__ int64_t ws[32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int64_t inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        int64_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o && t > inc) inc = t;
    }
    if (lane == 31) ws[w] = inc;
    __syncthreads();
    if (w == 0) {
        int64_t s = lane < nw ? ws[lane] : INT64_MIN;
        for (int o = 1; o < 32; o <<= 1) {
            int64_t t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o && t > s) s = t;
        }
        ws[lane] = s;
    }
    __syncthreads();
    int64_t r = inc;
    if (w > 0 && ws[w - 1] > r) r = ws[w - 1];
    if (total) *total = ws[nw - 1];
    __syncthreads();
    return r;
}

__global__ void k_dd_partial(int64_t n, const uint64_t *__restrict__ c, int64_t *part)
{
    int64_t base = (int64_t)blockIdx.x * DD_CHUNK;
    int64_t mx = INT64_MIN;
    for (int k = 0; k < DD_ITEMS; ++k) {
        int64_t i = base + k * DD_THREADS + threadIdx.x;
        if (i < n) {
            int64_t d = (int64_t)c[i] - i;
            if (d > mx) mx = d;
        }
    }
    int64_t tot;
    block_inclusive_max(mx, &tot);
    if (threadIdx.x == 0) part[blockIdx.x] = tot;
}

__global__ void k_dd_scan(int np, int64_t *part)
{
    // exclusive max-scan over chunk maxima (carry into each chunk)
    int64_t carry = INT64_MIN;
    for (int base = 0; base < np; base += DD_THREADS) {
        int i = base + threadIdx.x;
        int64_t v = i < np ? part[i] : INT64_MIN;
        int64_t tot;
        int64_t inc = block_inclusive_max(v, &tot);
        int64_t prev = __shfl_up_sync(0xffffffffu, inc, 1);
        __shared__ int64_t wlast[32];
        int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        if (lane == 31) wlast[w] = inc;
        __syncthreads();
        int64_t ex = (lane > 0) ? prev : (w > 0 ? wlast[w - 1] : INT64_MIN);
        if (carry > ex) ex = carry;
        __syncthreads();
        if (i < np) part[i] = ex;
        if (tot > carry) carry = tot;
    }
}

__global__ void k_dd_apply(int64_t n, uint64_t *c, const int64_t *__restrict__ carry)
{
    int64_t base = (int64_t)blockIdx.x * DD_CHUNK + (int64_t)threadIdx.x * DD_ITEMS;
    int64_t d[DD_ITEMS];
    int64_t run = INT64_MIN;
#pragma unroll
    for (int k = 0; k < DD_ITEMS; ++k) {
        int64_t i = base + k;
        d[k] = i < n ? (int64_t)c[i] - i : INT64_MIN;
        if (d[k] > run) run = d[k];
        d[k] = run;   // inclusive within the thread
    }
    // exclusive prefix of thread maxima
    int64_t inc = block_inclusive_max(run, nullptr);
    int64_t prev = __shfl_up_sync(0xffffffffu, inc, 1);
    __shared__ int64_t wl[32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 31) wl[w] = inc;
    __syncthreads();
    int64_t ex = (lane > 0) ? prev : (w > 0 ? wl[w - 1] : INT64_MIN);
    int64_t cin = carry[blockIdx.x];
    if (cin > ex) ex = cin;
#pragma unroll
    for (int k = 0; k < DD_ITEMS; ++k) {
        int64_t i = base + k;
        if (i < n) {
            int64_t v = d[k] > ex ? d[k] : ex;
            c[i] = (uint64_t)v + (uint64_t)i;
        }
    }
}

cudaError_t launch_dedupe(Handle *H, uint64_t *codes, int64_t n)
{
    if (n <= 1) return cudaSuccess;
    int nb = (int)((n + DD_CHUNK - 1) / DD_CHUNK);
    cudaError_t e = H->scan_tmp.reserve(sizeof(int64_t) * (nb + 1));
    if (e) return e;
    int64_t *part = H->scan_tmp.as<int64_t>();
    k_dd_partial<<<nb, DD_THREADS, 0, H->stream>>>(n, codes, part);
    k_dd_scan<<<1, DD_THREADS, 0, H->stream>>>(nb, part);
    k_dd_apply<<<nb, DD_THREADS, 0, H->stream>>>(n, codes, part);
    H->launches += 3;
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// permuted leaves and particle columns (up to GATHER_COLS of the quantity columns in one launch)
constexpr int GATHER_COLS = 8;

struct GatherCols {
    int n;
    const double *src[GATHER_COLS];
    double *dst[GATHER_COLS];
};

__global__ void k_gather(int64_t n, const uint32_t *__restrict__ idx, const double *__restrict__ x,
                         const double *__restrict__ y, const double *__restrict__ z, const double *__restrict__ h,
                         const double *__restrict__ m, const double *__restrict__ rho, double4 *leaf, double4 *aux,
                         double *rhos, int *odd, GatherCols cols)
{
    int bits = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t o = idx[i];
        if (o >= (uint64_t)n) o = 0;   // unreachable for a valid permutation; keeps reads in bounds
        const double ho = h[o], ro = rho[o];
        leaf[i] = make_double4(x[o], y[o], z[o], ho);
        aux[i] = make_double4(1.0 / ho, 1.0 / ro, m[o], ro);
        rhos[i] = ro;
        for (int c = 0; c < cols.n; ++c) cols.dst[c][i] = cols.src[c][o];
        if (!aux_regular(ho, ro)) bits |= ho < 0.0 ? ODD_RANGE | ODD_NEGATIVE_H : ODD_RANGE;
    }
    if (bits) atomicOr(odd, bits);
}

__global__ void k_gather_cols(int64_t n, const uint32_t *__restrict__ idx, GatherCols cols)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t o = idx[i];
        if (o >= (uint64_t)n) o = 0;
        for (int c = 0; c < cols.n; ++c) cols.dst[c][i] = cols.src[c][o];
    }
}

cudaError_t launch_gather(Handle *H, int64_t n, const double *x, const double *y, const double *z, const double *h,
                          const double *m, const double *rho, const std::vector<const double *> &cols)
{
    const uint32_t *idx = H->idx.as<uint32_t>();
    for (size_t c0 = 0; c0 == 0 || c0 < cols.size(); c0 += GATHER_COLS) {
        GatherCols G{};
        for (size_t c = c0; c < cols.size() && G.n < GATHER_COLS; ++c, ++G.n) {
            G.src[G.n] = cols[c];
            G.dst[G.n] = H->cols_s[c].as<double>();
        }
        if (c0 == 0)
            k_gather<<<grid_for(n, 256), 256, 0, H->stream>>>(n, idx, x, y, z, h, m, rho, H->leaf.as<double4>(),
                                                               H->leaf_aux.as<double4>(), H->rho_s.as<double>(),
                                                               H->odd.as<int>(), G);
        else k_gather_cols<<<grid_for(n, 256), 256, 0, H->stream>>>(n, idx, G);
        H->launches += 1;
    }
    return cudaGetLastError();
}

// the sorted x, y, z, m, h, rho as six columns, and the sorted quantity columns (the caller's arrays are
// put into Morton order)
__global__ void k_sorted_columns(int64_t n, const double4 *__restrict__ leaf, const double4 *__restrict__ aux, double *x,
                                 double *y, double *z, double *m, double *h, double *rho, GatherCols cols)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double4 L = ldg4(leaf + i), X = ldg4(aux + i);
        x[i] = L.x;
        y[i] = L.y;
        z[i] = L.z;
        m[i] = X.z;
        h[i] = L.w;
        rho[i] = X.w;
        for (int c = 0; c < cols.n; ++c) cols.dst[c][i] = cols.src[c][i];
    }
}

cudaError_t launch_sorted_columns(Handle *H, int64_t n, double *const dst[6], const std::vector<double *> &cols)
{
    GatherCols G{};
    for (size_t c = 0; c < cols.size(); ++c) {
        if (c >= GATHER_COLS) {
            cudaError_t e = cudaMemcpyAsync(cols[c], H->cols_s[c].p, sizeof(double) * n, cudaMemcpyDeviceToDevice, H->stream);
            if (e) return e;
            continue;
        }
        G.src[c] = H->cols_s[c].as<double>();
        G.dst[c] = cols[c];
        G.n = (int)c + 1;
    }
    k_sorted_columns<<<grid_for(n, 256), 256, 0, H->stream>>>(n, H->leaf.as<double4>(), H->leaf_aux.as<double4>(), dst[0],
                                                              dst[1], dst[2], dst[3], dst[4], dst[5], G);
    H->launches += 1;
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Karras topology (1-based, unified ids) with internal escapes
__device__ __forceinline__ int lcp(const uint64_t *__restrict__ c1, int64_t i, int64_t j)
{
    uint64_t a = c1[i], b = c1[j];
    uint64_t x = (a == b) ? ((uint64_t)i ^ (uint64_t)j) : (a ^ b);
    return x == 0 ? 64 : __clzll((long long)x);
}

__global__ void k_karras(int64_t n, const uint64_t *__restrict__ codes, int *left, int *right, int *parent,
                         int *escape, int2 *child, int2 *range)
{
    const uint64_t *c1 = codes - 1;
    const int64_t off = n - 1;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n - 1; t += (int64_t)gridDim.x * blockDim.x) {
        int64_t i = t + 1;
        // _range_direction / _find_range (BinaryRadixTree.jl:140-179)
        int dL = (i > 1) ? lcp(c1, i, i - 1) : -1;
        int dR = (i < n) ? lcp(c1, i, i + 1) : -1;
        int64_t d = (dR - dL >= 0) ? 1 : -1;
        int dmin = (1 <= i - d && i - d <= n) ? lcp(c1, i, i - d) : -1;
        int64_t lmax = 2;
        for (;;) {
            int64_t j = i + lmax * d;
            if (j < 1 || j > n) break;
            if (lcp(c1, i, j) <= dmin) break;
            lmax *= 2;
        }
        int64_t l = 0;
        for (int64_t s = lmax >> 1; s > 0; s >>= 1) {
            int64_t j = i + (l + s) * d;
            if (j >= 1 && j <= n && lcp(c1, i, j) > dmin) l += s;
        }
        int64_t j = i + l * d;
        int64_t lo = i < j ? i : j, hi = i < j ? j : i;
        // _split_position (BinaryRadixTree.jl:181-202)
        int64_t split;
        if (c1[lo] == c1[hi]) {
            split = (lo + hi) >> 1;
            if (split < lo) split = lo;
            if (split > hi - 1) split = hi - 1;
        } else {
            int pfl = lcp(c1, lo, hi);
            split = lo;
            int64_t step = hi - lo;
            while (step > 1) {
                step = (step + 1) >> 1;
                int64_t ns = split + step;
                if (ns < hi && lcp(c1, lo, ns) > pfl) split = ns;
            }
        }
        int64_t li = (split == lo) ? lo + off : split;
        int64_t ri = (split + 1 == hi) ? hi + off : split + 1;
        left[i - 1] = (int)li;
        right[i - 1] = (int)ri;
        child[i - 1] = make_int2((int)li, (int)ri);
        range[i - 1] = make_int2((int)(lo - 1), (int)(hi - 1));   // 0-based sorted leaf range of the subtree
        parent[li - 1] = (int)i;
        parent[ri - 1] = (int)i;
        // internal escape (BinaryRadixTree.jl:245-260); adj[k] = lcp(k, k+1), adj[n] = +inf
        int e;
        if (hi == n) e = 0;
        else if (hi == n - 1) e = (int)(off + n);
        else {
            int64_t nx = hi + 1;
            int anx = (nx < n) ? lcp(c1, nx, nx + 1) : 0x7fffffff;
            int apv = lcp(c1, nx - 1, nx);
            e = (anx < apv) ? (int)(off + nx) : (int)nx;
        }
        escape[i - 1] = e;
    }
}

// Leaf escapes (BinaryRadixTree.jl:262-281) and the Karras bottom-up refit with atomic
// second arrival (LinearBVH.jl:98-156).  Min/max are order independent, so the FP64
// boxes and hmax are bit-identical to a sequential refit.
//
// A block takes RF_LEAVES consecutive leaves.  The nodes whose leaf range lies inside them are
// combined in shared memory (a Karras node's id is one end of its range, so ids index the block's
// slots) and written together; then the few climbs that reach past the block's leaves go on through
// global counters, with fences around the children's boxes, which are read through L2 (__ldcg).
// The climb through global memory alone waited on a fence and four dependent loads per node and wrote
// every box by itself: 4.2e6 leaves 884 us, 1e6 leaves 269, 6,000 leaves 50; now 520, 182 and 38 us (64 to 512 leaves a block are within 15 %).
constexpr int RF_LEAVES = 256;

struct RefitBox {
    double mn[3], mx[3], h;
};

__device__ __forceinline__ void refit_merge(RefitBox &a, const RefitBox &b)
{
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        a.mn[d] = (a.mn[d] < b.mn[d]) ? a.mn[d] : b.mn[d];
        a.mx[d] = (a.mx[d] > b.mx[d]) ? a.mx[d] : b.mx[d];
    }
    a.h = (a.h > b.h) ? a.h : b.h;
}

__global__ void __launch_bounds__(RF_LEAVES) k_refit(int64_t n, const int *__restrict__ parent,
                                                     const int *__restrict__ left, const int *__restrict__ right,
                                                     const int2 *__restrict__ range, int *escape,
                                                     const double4 *__restrict__ leaf, NodeF *node, float *node_hmax,
                                                     double *bmin, double *bmax, double *hmax, unsigned *counters,
                                                     int *leaf_escape, int *status)
{
    __shared__ RefitBox s_box[RF_LEAVES];
    __shared__ unsigned s_count[RF_LEAVES];
    __shared__ int s_left[RF_LEAVES], s_right[RF_LEAVES], s_parent[RF_LEAVES], s_escape[RF_LEAVES];
    __shared__ int2 s_range[RF_LEAVES];
    const int64_t nin = n - 1, k0 = (int64_t)blockIdx.x * RF_LEAVES, k = k0 + threadIdx.x;
    const int64_t k1 = k0 + RF_LEAVES < n ? k0 + RF_LEAVES : n;   // the block's leaves: [k0, k1)
    // the topology of the nodes with the block's ids, so that a climb inside waits for no global load
    s_count[threadIdx.x] = 0;
    if (k < nin) {
        s_left[threadIdx.x] = left[k];
        s_right[threadIdx.x] = right[k];
        s_parent[threadIdx.x] = parent[k];
        s_escape[threadIdx.x] = escape[k];
        s_range[threadIdx.x] = range[k];
    }
    __syncthreads();
    const int64_t id = n + k;
    const bool live = k < n;
    int p = live ? parent[id - 1] : 0, from = (int)id;
    RefitBox B{};   // of the node climbed from
    if (live) {
        int e = 0;
        if (p != 0) e = (left[p - 1] == (int)id) ? right[p - 1] : escape[p - 1];
        leaf_escape[k] = e;
        escape[id - 1] = e;
        const double4 L = leaf[k];
        B = RefitBox{{L.x, L.y, L.z}, {L.x, L.y, L.z}, L.w};
    }
    auto valid = [&](int q, int l, int r) { return q >= 0 && q <= nin && l >= 1 && l < 2 * n && r >= 1 && r < 2 * n; };
    // min and max do not depend on the order of the children, but the choice between -0 and 0 does:
    // left child first
    auto combine = [&](bool from_left, RefitBox &S) {
        if (from_left) refit_merge(B, S);
        else {
            refit_merge(S, B);
            B = S;
        }
    };
    bool climbing = live && p != 0;
    while (climbing && p - 1 >= k0 && p - 1 < k1) {   // at most RF_LEAVES steps: every one has its own slot
        const int at = (int)(p - 1 - k0);
        if (!(s_range[at].x >= k0 && s_range[at].y < k1)) break;
        const int l = s_left[at], r = s_right[at], sib = l == from ? r : l;
        if (!valid(p, l, r)) { atomicOr(status, ST_REFIT); climbing = false; break; }
        __threadfence_block();   // this child's box (below) before its arrival
        const unsigned old = atomicAdd(&s_count[at], 1u);
        if (old != 1) {   // the second arrival combines
            if (old > 1) atomicOr(status, ST_REFIT);
            climbing = false;
            break;
        }
        __threadfence_block();
        RefitBox S;
        if (sib >= n) {
            const double4 M = leaf[sib - n];
            S = RefitBox{{M.x, M.y, M.z}, {M.x, M.y, M.z}, M.w};
        } else {
            const volatile double *v = reinterpret_cast<const volatile double *>(&s_box[sib - 1 - k0]);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                S.mn[d] = v[d];
                S.mx[d] = v[3 + d];
            }
            S.h = v[6];
        }
        combine(l == from, S);
        s_box[at] = B;
        from = p;
        p = s_parent[at];
        climbing = p != 0;
    }
    __syncthreads();
    auto put = [&](int64_t i, const RefitBox &X, int l, int esc) {
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            bmin[d * nin + i] = X.mn[d];
            bmax[d * nin + i] = X.mx[d];
        }
        hmax[i] = X.h;
        NodeF nd;
        nd.lox = __double2float_rd(X.mn[0]); nd.loy = __double2float_rd(X.mn[1]); nd.loz = __double2float_rd(X.mn[2]);
        nd.hix = __double2float_ru(X.mx[0]); nd.hiy = __double2float_ru(X.mx[1]); nd.hiz = __double2float_ru(X.mx[2]);
        nd.left = l;
        nd.escape = esc;
        node[i] = nd;
        node_hmax[i] = __double2float_ru(X.h);
    };
    if (k < nin && s_count[threadIdx.x] == 2u) {
        put(k, s_box[threadIdx.x], s_left[threadIdx.x], s_escape[threadIdx.x]);
        counters[k] = 2u;
    }
    __syncthreads();   // the boxes of the block's top nodes are written
    int64_t depth = 0;
    while (climbing) {
        const int l = left[p - 1], r = right[p - 1], sib = l == from ? r : l;
        // a valid tree has depth < n and ids in range; anything else is reported, not followed
        if (++depth > n || !valid(p, l, r)) { atomicOr(status, ST_REFIT); break; }
        const int esc = escape[p - 1], up = parent[p - 1];
        __threadfence();
        if (atomicAdd(&counters[p - 1], 1u) == 0) break;
        __threadfence();
        RefitBox S;
        if (sib >= n) {
            const double4 M = leaf[sib - n];
            S = RefitBox{{M.x, M.y, M.z}, {M.x, M.y, M.z}, M.w};
        } else {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                S.mn[d] = __ldcg(&bmin[d * nin + sib - 1]);
                S.mx[d] = __ldcg(&bmax[d * nin + sib - 1]);
            }
            S.h = __ldcg(&hmax[sib - 1]);
        }
        combine(l == from, S);
        put(p - 1, B, l, esc);
        from = p;
        p = up;
        climbing = p != 0;
    }
}

__global__ void k_check_counters(int64_t nin, const unsigned *__restrict__ counters, int *status)
{
    int bad = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nin; i += (int64_t)gridDim.x * blockDim.x)
        if (counters[i] != 2u) bad = 1;
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(status, ST_REFIT);
}

cudaError_t launch_topology(Handle *H, int64_t n)
{
    if (n < 2) {
        cudaMemsetAsync(H->escape.p, 0, sizeof(int), H->stream);
        cudaMemsetAsync(H->parent.p, 0, sizeof(int), H->stream);
        cudaMemsetAsync(H->leaf_escape.p, 0, sizeof(int), H->stream);
        return cudaGetLastError();
    }
    int64_t ntot = 2 * n - 1;
    cudaMemsetAsync(H->parent.p, 0, sizeof(int) * ntot, H->stream);
    cudaMemsetAsync(H->counters.p, 0, sizeof(unsigned) * (n - 1), H->stream);
    k_karras<<<grid_for(n - 1, 256), 256, 0, H->stream>>>(n, H->codes.as<uint64_t>(), H->left.as<int>(),
                                                          H->right.as<int>(), H->parent.as<int>(), H->escape.as<int>(),
                                                          H->node_child.as<int2>(), H->node_range.as<int2>());
    k_refit<<<(unsigned)((n + RF_LEAVES - 1) / RF_LEAVES), RF_LEAVES, 0, H->stream>>>(
        n, H->parent.as<int>(), H->left.as<int>(), H->right.as<int>(), H->node_range.as<int2>(), H->escape.as<int>(),
        H->leaf.as<double4>(),
        H->node.as<NodeF>(), H->node_hmax.as<float>(), H->bmin64.as<double>(), H->bmax64.as<double>(),
        H->hmax64.as<double>(), H->counters.as<unsigned>(), H->leaf_escape.as<int>(), H->status.as<int>());
    k_check_counters<<<grid_for(n - 1, 256), 256, 0, H->stream>>>(n - 1, H->counters.as<unsigned>(),
                                                                  H->status.as<int>());
    H->launches += 3;
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Morton order of query points (schedule only: outputs are written back to their own slot)
// 30-bit Morton code of a sample point in a tree's quantisation frame (10 bits per axis,
// clamped to the particles' box): only an ordering key, not the build's codes
__device__ __forceinline__ uint32_t query_code30(const QuantParams &q, double x, double y, double z)
{
    const double p[3] = {x, y, z};
    uint32_t c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double f = q.flat[d] ? 0.5 : (p[d] - q.vmin[d]) * q.inv[d];
        f = fmin(fmax(f, 0.0), 1.0);
        if (!(f == f)) f = 0.0;
        c[d] = (uint32_t)(f * 1023.0);
    }
    return ((uint32_t)expand_bits3(c[0]) << 2) | ((uint32_t)expand_bits3(c[1]) << 1) | (uint32_t)expand_bits3(c[2]);
}

__global__ void k_query_codes(int64_t nq, const double *__restrict__ qx, const double *__restrict__ qy,
                              const double *__restrict__ qz, const QuantParams *__restrict__ qp, int drop,
                              uint32_t *keys, uint32_t *perm)
{
    const QuantParams q = *qp;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nq; i += (int64_t)gridDim.x * blockDim.x) {
        keys[i] = query_code30(q, qx[i], qy[i], qz[i]) >> drop;
        perm[i] = (uint32_t)i;
    }
}

__global__ void k_batch_query_codes(int64_t m, const BatchDisc *__restrict__ discs, const int64_t *__restrict__ starts,
                                    const uint32_t *__restrict__ slot_disc, const int *__restrict__ slot_of,
                                    int64_t s0, int bits, uint64_t *keys, uint32_t *vals)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x) {
        const int lo = slot_of[t];
        const BatchDisc &D = discs[slot_disc[lo]];
        const int64_t qi = s0 + t - starts[lo];
        keys[t] = ((uint64_t)(uint32_t)lo << bits) | (query_code30(*D.qp, D.qx[qi], D.qy[qi], D.qz[qi]) >> (30 - bits));
        vals[t] = (uint32_t)t;
    }
}

cudaError_t launch_batch_query_codes(Handle *H, int64_t m, const BatchDisc *discs, const int64_t *starts,
                                     const uint32_t *slot_disc, const int *slot_of, int64_t s0, int bits,
                                     uint64_t *keys, uint32_t *vals)
{
    k_batch_query_codes<<<grid_for(m, 256), 256, 0, H->stream>>>(m, discs, starts, slot_disc, slot_of, s0, bits, keys, vals);
    H->launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_query_codes(Handle *H, int64_t nq, const double *qx, const double *qy, const double *qz,
                               int drop, uint32_t *keys, uint32_t *perm)
{
    k_query_codes<<<grid_for(nq, 256), 256, 0, H->stream>>>(nq, qx, qy, qz, H->qparams.as<QuantParams>(), drop, keys,
                                                            perm);
    H->launches += 1;
    return cudaGetLastError();
}

}  // namespace pb
