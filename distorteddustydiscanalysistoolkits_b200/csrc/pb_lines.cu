// pb_lines.cu -- line-integrated (column) interpolation, itpScatter (both precision modes).
// Compiled with -fmad=false: every expression is the IEEE result of the reference's operation
// order.
#include "line_tables.h"
#include "pb_internal.h"
#include "pb_interp_impl.cuh"

namespace pb {

__device__ const double g_line_inorm64[6][PB_LINE_NTAB] = PB_LINE_INORM_INIT;

// --------------------------------------------------------------------------------------
// line-sample kernel (itpScatter): one thread per line
__device__ __forceinline__ double line_lut(const double *__restrict__ I, double qmax, double q)
{
    const double dq = qmax / double(PB_LINE_NTAB_DEV - 1);
    double idxf = q / dq + 1.0;
    int i = (int)idxf;
    i = i < 1 ? 1 : (i > PB_LINE_NTAB_DEV - 1 ? PB_LINE_NTAB_DEV - 1 : i);
    double t = idxf - double(i);
    return __ldg(I + i - 1) * (1.0 - t) + __ldg(I + i) * t;
}

__global__ void __launch_bounds__(128) k_lines(DevTree T, DevCatalog C, int64_t nl, const double *__restrict__ ox,
                                               const double *__restrict__ oy, const double *__restrict__ oz,
                                               const double *__restrict__ mx, const double *__restrict__ my,
                                               const double *__restrict__ mz, const uint32_t *__restrict__ perm,
                                               const double *__restrict__ table)
{
    const int64_t n = T.n;
    const int k = T.kernel;
    const double K = kernel_valid(k);
    const double *I = table + (int64_t)k * PB_LINE_NTAB_DEV;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nl; j += (int64_t)gridDim.x * blockDim.x) {
        int64_t li = perm ? (int64_t)__ldg(perm + j) : j;
        if (li >= nl) continue;
        double o[3] = {__ldg(ox + li), __ldg(oy + li), __ldg(oz + li)};
        double m[3] = {__ldg(mx + li), __ldg(my + li), __ldg(mz + li)};
        double S1 = 0.0, acc[MAXS];   // plain sums in the reference order
#pragma unroll
        for (int s = 0; s < MAXS; ++s) acc[s] = 0.0;
        int node = T.root;
        int64_t bi = 0, guard = 0, limit = 4 * n + 64;
        bool brute = (node == 0);
        while (brute ? (bi < n) : (node != 0)) {
            if (++guard > limit) { flag(T.status, ST_TRAVERSAL); break; }
            bool leafnode = brute || node >= n;
            if (leafnode) {
                int64_t b = brute ? bi++ : (int64_t)(node - n);
                double4 L = ldg4(T.leaf + b);
                int esc = brute ? 0 : __ldg(T.leaf_escape + b);
                double r = __dmul_rn(K, L.w);
                double r2 = __dmul_rn(r, r);
                double d2 = d2_line(L.x, L.y, L.z, o, m);
                if (d2 <= r2) {
                    const double4 X = ldg4(T.aux + b);
                    // line_integrated_kernel_function (line_integrated_kernel.jl:132-137)
                    double dr = sqrt(d2 > 0.0 ? d2 : 0.0);
                    double invh = X.x;
                    double q = dr * invh;
                    double Iq = (q >= K) ? 0.0 : line_lut(I, K, q);
                    double W = invh * Iq;
                    double w = X.z * W / X.w;
                    S1 += w;
#pragma unroll
                    for (int s = 0; s < MAXS; ++s)
                        if (s < C.n_scalar) acc[s] += __ldg(C.ucol[C.s_u[s]] + b) * w;
                }
                if (!brute) node = esc;
            } else {
                NodeF nd = load_node(T.node + (node - 1));
                double r = __dmul_rn(K, (double)__ldg(T.node_hmax + (node - 1)));
                double r2 = __dmul_rn(r, r);
                node = (d2_line_box_lower(o, m, nd) > r2) ? nd.escape : nd.left;
            }
        }
        int l = 0;
#pragma unroll
        for (int s = 0; s < MAXS; ++s) {
            if (s < C.n_scalar) {
                double v;
                if (S1 == 0.0) v = __longlong_as_double(0x7ff8000000000000LL);
                else v = C.s_shep[s] ? acc[s] * (1.0 / S1) : acc[s];
                C.out[l++][li] = v;
            }
        }
    }
}

cudaError_t launch_lines_fp64(Handle *H, const DevTree &T, const DevCatalog &C, int64_t nl, const double *ox,
                              const double *oy, const double *oz, const double *dx, const double *dy,
                              const double *dz, const uint32_t *perm)
{
    const double *tab = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void **)&tab, g_line_inorm64);
    if (e) return e;
    int bs = 128;
    k_lines<<<grid_for(nl, bs, 1 << 30), bs, 0, H->stream>>>(T, C, nl, ox, oy, oz, dx, dy, dz, perm, tab);
    H->launches += 1;
    return cudaGetLastError();
}

}  // namespace pb
