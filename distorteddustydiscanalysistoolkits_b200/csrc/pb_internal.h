// pb_internal.h -- host-side handle and the launchers shared between translation units.
#pragma once
#include <cstdint>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "pb_device.cuh"

namespace pb {

// One disc of a batched launch (pb_batch.cu): its tree, the FP32C and FP64 catalogs of its
// columns and outputs, its FP32C payload, and its sample points.
struct BatchDisc {
    DevTree T;
    DevCatalog C32, C64;
    const float4 *pay;
    const double *qx, *qy, *qz;
    const QuantParams *qp;   // the disc's quantisation frame (Morton order of its sample points)
    int64_t nq;
    int stride;
    int pad;
};
static_assert(sizeof(BatchDisc) % 8 == 0, "batch descriptors are copied in 8-byte words");

// grow-only device buffer
struct DBuf {
    void *p = nullptr;
    size_t bytes = 0;
    cudaError_t reserve(size_t b)
    {
        if (b <= bytes) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
        cudaError_t e = cudaMalloc(&p, b < 256 ? 256 : b);
        if (e == cudaSuccess) bytes = b < 256 ? 256 : b;
        return e;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    template <typename T> T *as() const { return static_cast<T *>(p); }
};

// learned schedule: MLP of SCHED_F features -> SCHED_H -> SCHED_H -> 1
constexpr int SCHED_F = 16;
constexpr int SCHED_H = 64;
constexpr int SCHED_NPARAM = SCHED_H * SCHED_F + SCHED_H + SCHED_H * SCHED_H + SCHED_H + SCHED_H + 1;

struct Handle {
    int device = 0;
    cudaStream_t stream = nullptr;       // where launches go
    cudaStream_t own_stream = nullptr;   // created by pb_create
    std::string err;
    int64_t launches = 0;

    // built particle set
    bool built = false;
    int64_t n = 0;
    int ncol = 0;
    int kernel = 0;

    DBuf in_x, in_y, in_z, in_h, in_m, in_rho;    // staging for host inputs
    std::vector<DBuf> in_cols;
    DBuf codes, codes_alt, idx, idx_alt, scan_tmp, hist;
    DBuf bbox_part, qparams, status;
    DBuf leaf, leaf_aux, odd, leaf_escape, node, node_hmax, node_child, node_range;
    DBuf payload;       // per-call FP32 particle payload of the FP32-compensated path
    DBuf counter;       // work-queue counter of the warp-per-query kernels
    DBuf left, right, escape, parent;
    DBuf bmin64, bmax64, hmax64, counters;
    DBuf rho_s;
    std::vector<DBuf> cols_s;
    DBuf col_ptrs;      // device array of sorted column pointers

    // run lists of the two-phase point path (walk kernel -> pair kernels)
    DBuf grid_ax, grid_out;   // axes / points of pb_grid_points
    DBuf pool_runs, pool_next, pool_ctr, items, wbnear, qacc, qflag, defer_a, defer_b, lpt_k, lpt_v, lpt_ka,
        lpt_va, iota, long_list, long_count, line_rest;
    int walk_split = 64;   // accepted and kept; the walk is not split any more
    int sched = 1;         // 0 plain (input order, one walk per query, no ordering), 1 tuned, 2 learned
    int64_t light_max = 4096;   // FP32C: queries with at most this many neighbours are summed in FP64
    int64_t slice = int64_t(1) << 22;   // queries per two-phase slice
    double pool_cpq = 0.0;   // largest pool chunks per completed query seen by the last call (0: none)
    // learned work prediction (pb_sched.cu)
    DBuf mlp_w, mlp_m, mlp_v, mlp_g, mlp_norm, mlp_scr, mlp_idx, mlp_x, mlp_y, mlp_loss, sched_feat, sched_pred,
        sched_ql, sched_tmp;
    bool mlp_ready = false;
    float sched_width = 1.f;
    int sched_nclass = 16;
    unsigned long long pool_cap = 0;
    int64_t walk_rounds = 0, deferred_total = 0;
    // queries and accepted pairs of the last point call summed by the FP32C (heavy) and the
    // FP64 (light) pair kernels
    int64_t split_hq = 0, split_lq = 0, split_hp = 0, split_lp = 0;

    // batched launch (pb_batch_points): descriptors, processing-order starts, pinned staging
    DBuf batch_desc, batch_starts, batch_slots, batch_ctr;
    void *batch_host = nullptr;
    size_t batch_host_bytes = 0;
    int leaf_size = 1;       // warp-uniform walk: subtrees of at most this many leaves are scanned
    int batch_order = 0;     // 0: discs in the given order, 1: discs with the most work first
    int batch_blocks = 0;    // blocks per SM of the batched pair kernel (0: as many as fit)
    int64_t batch_slice = 0; // sample points per slice the batch's run pool was sized for
    int batch_walk_split = 16;   // accepted and kept, as walk_split
    DBuf batch_slot_of;      // processing slot of every point of a slice
    DBuf batch_mk, batch_mka, batch_mv, batch_mva;         // Morton walk order of a slice

    // staging of small host arrays packed into one copy (ordinary memory, then page-locked) and of the words
    // the host reads back
    unsigned char *pack = nullptr, *pin = nullptr;
    size_t pack_bytes = 0;
    int64_t pin_after = 32, pin_uses = 0;   // 0: never page-locked
    bool pin_failed = false;
    DBuf in_pack, q_pack, out_pack;

    // query-side scratch
    DBuf q_x, q_y, q_z, q_keys, q_keys_alt, q_perm, q_perm_alt, q_out, q_aux, q_rest;
    std::vector<DBuf> q_outs;

    // timing (CUDA events around the build and the traversal launches)
    bool timing = false;
    cudaEvent_t ev[8] = {};
    float t_build_ms = 0.f, t_interp_ms = 0.f;
    float t_phase_ms[3] = {0.f, 0.f, 0.f};   // nearest search, walk (+ ordering), pairs; all slices and rounds
    int64_t interp_launches = 0;
    int sort_queries = 1;
    int64_t sort_wait = int64_t(1) << 22;   // reads of a look-back word before a sort tile counts for itself
    int block_size = 128;

    ~Handle();
};

// ---- launchers (pb_build.cu) ----
cudaError_t launch_bbox(Handle *H, int64_t n, const double *x, const double *y, const double *z, const double *h);
cudaError_t launch_encode(Handle *H, int64_t n, const double *x, const double *y, const double *z);
// stable sorts by the lowest bits; vals_at: where the sorted values are, instead of in vals (the keys
// are then left where the last pass put them)
cudaError_t sort_pairs_u64(Handle *H, uint64_t *keys, uint32_t *vals, uint64_t *kalt, uint32_t *valt, int64_t n,
                           int bits, uint32_t **vals_at = nullptr);
cudaError_t sort_pairs_u32(Handle *H, uint32_t *keys, uint32_t *vals, uint32_t *kalt, uint32_t *valt, int64_t n,
                           int bits, uint32_t **vals_at = nullptr);
// per point t of a batch slice: key (processing slot << bits) | the highest `bits` bits of the point's
// 30-bit Morton code in its disc's quantisation frame, value t
cudaError_t launch_batch_query_codes(Handle *H, int64_t m, const BatchDisc *discs, const int64_t *starts,
                                     const uint32_t *slot_disc, const int *slot_of, int64_t s0, int bits,
                                     uint64_t *keys, uint32_t *vals);
cudaError_t launch_dedupe(Handle *H, uint64_t *codes, int64_t n);
cudaError_t launch_gather(Handle *H, int64_t n, const double *x, const double *y, const double *z, const double *h,
                          const double *m, const double *rho, const std::vector<const double *> &cols);
cudaError_t launch_topology(Handle *H, int64_t n);
// 30-bit Morton codes of the sample points without their lowest `drop` bits
cudaError_t launch_query_codes(Handle *H, int64_t nq, const double *qx, const double *qy, const double *qz, int drop,
                               uint32_t *keys, uint32_t *perm);
// the sorted x, y, z, m, h, rho and quantity columns to device arrays
cudaError_t launch_sorted_columns(Handle *H, int64_t n, double *const dst[6], const std::vector<double *> &cols);

// ---- launchers (pb_walk.cu) ----
cudaError_t launch_nearest_list(Handle *H, const DevTree &T, int64_t m, const uint32_t *ql, const double *qx,
                                const double *qy, const double *qz, int *bnear, bool listed);
// listed: the nearest search of the same queries has listed those with the longest walks
cudaError_t launch_walk(Handle *H, const DevTree &T, int strategy, const RunPool &P, int64_t m, const uint32_t *ql,
                        const double *qx, const double *qy, const double *qz, bool listed, unsigned long long *counter);
cudaError_t launch_split_order(Handle *H, const RunPool &P, int64_t m, unsigned light_max, bool plain,
                               uint32_t **order, unsigned long long *pairs);
cudaError_t launch_iota(Handle *H, int64_t m, uint32_t *out);
cudaError_t launch_count_heavy(Handle *H, const RunPool &P, int64_t m, unsigned light_max, unsigned *count,
                               unsigned long long *pairs);
int batch_catalog_shape(const DevCatalog &C);

// ---- launchers (pb_sched.cu) ----
cudaError_t launch_sched_features(Handle *H, const DevTree &T, int64_t m, const uint32_t *ql, const double *qx,
                                  const double *qy, const double *qz, const int *bnear, float *feat);
cudaError_t launch_mlp_predict(Handle *H, int64_t n, const float *X, float *y);
cudaError_t launch_mlp_grad(Handle *H, int64_t nb, const float *X, const float *T, const int64_t *idx, float *loss);
const float *mlp_last_sq(Handle *H, int64_t nb);
cudaError_t launch_mlp_adam(Handle *H, float lr, int64_t step);
cudaError_t launch_draw(Handle *H, int64_t nb, int64_t n, unsigned long long seed, unsigned long long step,
                        int64_t *idx);
cudaError_t launch_sched_order(Handle *H, int64_t m, const float *pred, float width, int nclass, uint32_t *order);
cudaError_t launch_gather_u32(Handle *H, int64_t m, const uint32_t *order, const uint32_t *src, uint32_t *dst);
cudaError_t launch_gather_i32(Handle *H, int64_t m, const uint32_t *order, const int *src, int *dst);

// ---- launchers (pb_interp64.cu / pb_interp32.cu / pb_query.cu) ----
// classes: the order is by descending size class
cudaError_t launch_pairs_fp32(Handle *H, const DevTree &T, const DevCatalog &C, int strategy, const RunPool &P,
                              int64_t m, const uint32_t *ql, const uint32_t *order, const double *qx,
                              const double *qy, const double *qz, bool classes);
cudaError_t launch_points_fp64(Handle *H, const DevTree &T, const DevCatalog &C, int strategy, int64_t nq,
                               const double *qx, const double *qy, const double *qz, const uint32_t *perm,
                               int64_t npts);
// queries of a higher size class than block_min accepted leaves (the first of the order) are taken by
// whole blocks; 0xffffffff: none
cudaError_t launch_pairs_fp64(Handle *H, const DevTree &T, const DevCatalog &C, int strategy, const RunPool &P,
                              int64_t m, unsigned block_min, const uint32_t *ql, const uint32_t *order,
                              const double *qx, const double *qy, const double *qz);
cudaError_t launch_points_fp32(Handle *H, const DevTree &T, const DevCatalog &C, int strategy, int64_t nq,
                               const double *qx, const double *qy, const double *qz, const uint32_t *perm,
                               int64_t npts);
cudaError_t launch_lines_fp64(Handle *H, const DevTree &T, const DevCatalog &C, int64_t nl, const double *ox,
                              const double *oy, const double *oz, const double *dx, const double *dy,
                              const double *dz, const uint32_t *perm);
cudaError_t launch_nearest(Handle *H, const DevTree &T, int64_t nq, const double *qx, const double *qy,
                           const double *qz, double *h_out, int64_t *idx_out);
cudaError_t launch_query(Handle *H, const DevTree &T, int64_t nq, const double *qx, const double *qy,
                         const double *qz, const double *radius, const int64_t *offsets, int64_t *counts,
                         int64_t *pool, int64_t *nearest, double *nearest_d2);
cudaError_t launch_grid_points(Handle *H, int coord, const double *a0, int64_t n0, const double *a1, int64_t n1,
                               const double *a2, int64_t n2, double *x, double *y, double *z);
cudaError_t launch_stats(Handle *H, const DevTree &T, int strategy, int64_t nq, const double *qx, const double *qy,
                         const double *qz, int64_t *stats);
// image plane of pb_line_image: origin c, axes e1 and e2, line direction d
struct LineFrame {
    double c[3], e1[3], e2[3], d[3];
};
cudaError_t launch_batch_slice(Handle *H, int strategy, int kernel, int cat, int cat64, const BatchDisc *discs,
                               const int64_t *starts, const uint32_t *slot_disc, int ndisc, int64_t s0, int64_t m,
                               const RunPool &P, int fp64_only, unsigned light_max, int leaf_size, int blocks_per_sm,
                               int *slot_of, unsigned long long *ctr);
cudaError_t launch_batch_payload(Handle *H, const DevTree &T, const DevCatalog &C, float4 **pay, int *stride);
cudaError_t launch_line_image(Handle *H, const double *a0, int64_t n0, const double *a1, int64_t n1, const LineFrame &F,
                              double *ox, double *oy, double *oz, double *dx, double *dy, double *dz);

// Nearest searches of at most this many points go a warp each instead of a thread each
// (2,744 points 131 -> 20 us, 20,000 points 222 -> 95 us; 153,600 points would take 587 us, not 297: a
// warp reads more nodes than its lanes' own searches, but waits for a quarter of the steps).  In a tree of few
// particles the steps are few: thread / warp each 83 / 91 us (100 particles, 24,000 points), 74 / 75
// (16,000); 106 / 119 (1,000 particles, 32,000 points), 103 / 101 (24,000); 143 / 138 (8,000 particles, 32,000).
constexpr int64_t NEAREST_WARP_MAX = 32768;
inline int64_t nearest_warp_max(int64_t nparticles)
{
    return nparticles >= 4096 ? NEAREST_WARP_MAX : (nparticles >= 512 ? 24576 : 12288);
}

inline int grid_for(int64_t n, int block, int cap = 148 * 32)
{
    int64_t g = (n + block - 1) / block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

}  // namespace pb

// the opaque handle of the C ABI (include/partia_b200.h)
struct pb_handle {
    pb::Handle H;
};
