// Batched VCD: the types and device helpers shared by the batched stages (vcd_batched.cu) and the forward-
// projection stage kernels, which are compiled per geometry kind in their own translation units
// (b_fp_parallel.cu, b_fp_cone.cu, b_fp_translation.cu) for build parallelism.
#pragma once

#include <vector>

#include "back_project.cuh"
#include "bp_fast.cuh"
#include "direct_filter.cuh"
#include "fp_cb.cuh"
#include "mbx_common.cuh"
#include "mbx_host.hpp"
#include "mbx_reduce.cuh"
#include "qggmrf.cuh"

namespace mbx {

constexpr int BT_THREADS = 256;
constexpr int BT_ELEM_TILE = 2048;   // cylinder elements per tile (delta, apply)
constexpr int BT_SINO_TILE = 4096;   // sinogram / recon elements per tile (linquad, error, stats)
constexpr float BT_EPS_F32 = 1.1920928955078125e-07f;

struct VcdScan {
    float *recon;               // flat (Nr*Nc, S)
    float *err;                 // (V, R, C)
    const float *wts;           // (V, R, C) or NULL
    float *hess;                // flat (Nr*Nc, S)
    const int32_t *partition;   // (K, M)
    float *bp, *delta, *dsino;  // workspace slices
    const float *y;             // measured sinogram (set-up input) or NULL
    long long nsino, nrecon;
    int K, M, nr, nc, ns;
    float *tsino;               // transposed copy of the sinogram a back-projection stage reads, or NULL (bp_fast.cuh)
    int V, R, C, rp;
};

// Direct-recon filtering of one scan in the set-up: rows of y into err.
struct FiltScan {
    const float *in;
    float *out;
    long long rows;
    int R, C, fdk;
    double filter_scale, out_scale, D, ddc, ddr, dco, dro;
};

// A work list of projection tiles over the scans of a batch: per scan, its argument record(s) and tile count.
// Tiles are numbered over the scans in `order` (decreasing per-tile cost) and handed out dynamically.
struct ProjList {
    const BpArgs *bp;      // back-projection records (or NULL)
    const FpArgs *fp;      // forward-projection records (or NULL)
    const int *off;        // [num_scans + 1] tile prefix over the positions of `order`
    const int *dim;        // [num_scans] per scan: gx (back projection) or channel blocks (forward)
    const int *order;      // [num_scans] scan at each position
    const int *schedule;   // [num_steps][num_scans] record of each scan at each step, or NULL (record 0)
    int stride;            // records per scan
    int *counter;          // next tile (reset by a memset before each launch)
    const CbPlanned *planned;  // forward lists: stored record passes of each record, or NULL (walk every tile)
};

// Projection work lists of a batch.  PL_BUILD covers every (scan, subset, view, channel block) tile: the builds
// of the planned forward projections.
enum { PL_BP = 0, PL_FP, PL_INIT_BP, PL_INIT_FP, PL_HESS, PL_BUILD, PL_COUNT };

struct BatchedTables {
    VcdScan *scans;
    float *fm;          // [scan] 1 / sigma_y^2 (per call)
    QParams *qp;        // [scan] qGGMRF parameters (per call)
    BpArgs *bpargs;     // [scan][subset]
    FpArgs *fpargs;     // [scan][subset]
    BpArgs *init_bp;    // [scan]: filtered sinogram -> recon over the region of reconstruction
    FpArgs *init_fp;    // [scan]: recon -> dsino over the region of reconstruction
    BpArgs *hess_bp;    // [scan]: weights (or ones) -> Hessian over every pixel, squared coefficients
    FiltScan *filt;     // [scan]
    CbPlanned *planned; // [scan][subset] stored record passes of the subset forward projections (planned batches)
    int *pl_off;        // [PL_COUNT][num_scans + 1]
    int *pl_dim;        // [PL_COUNT][num_scans]
    int *pl_order;      // [PL_COUNT][num_scans]
    int *el_off, *sn_off, *rc_off, *flt_off, *tr_off;  // [num_scans + 1] tile prefix offsets (scan order)
    int *box_first;     // [num_scans * K + 1] chunk prefix over (scan, subset) records
    int *counters;      // [PL_COUNT]
    int *schedule;      // [num_steps][num_scans]
    double *p_prior, *p_fwd, *p_l1, *p_iter, *p_init;
    float *alpha;       // [num_scans]
    float *alpha_init;  // [num_scans]
    double *step_stats; // [num_steps][num_scans][4]
    double *iter_stats; // [num_iterations][num_scans][4]
};

struct BatchedPlanHost {
    BatchedTables t;
    int num_scans, kind, num_steps, num_iterations, ksum, has_setup;
    int planned_fp;                 // subset forward projections replay stored record passes
    int pl_grid_replay, pl_grid_build;  // grids of the replay and build kernels (variant fp_minb)
    void *plan_cursors;             // [ksum] bump cursors of the planned lists (one memset resets them)
    size_t plan_cursor_bytes;
    int pl_total[PL_COUNT], pl_grid[PL_COUNT];
    size_t pl_smem[PL_COUNT];
    int el_total, sn_total, rc_total, flt_total, box_total, tr_total;
    int el_grid, sn_grid, rc_grid, flt_grid, box_grid, tr_grid;
    int windows[3];       // by back projection (SW_SUBSET, SW_INIT, SW_HESS): reads windows of transposed copies
    size_t flt_smem;
    int init_minb;  // b_fp variant of the initial projection: cb_many for parallel beam, else 2
    int fp_minb;  // b_fp variant of the subset stage: 2 or cb_many resident CTAs per SM
    size_t fp_smem_replay;  // shared memory of the replay kernel (the replay layouts of the subset plans)
    int magic;
};
static_assert(sizeof(BatchedPlanHost) <= sizeof(mbx_batched_plan), "plan record too large");
constexpr int BT_MAGIC = 0x6d627863;

inline ProjList proj_list(const BatchedTables &T, int which, int num_scans) {
    ProjList L;
    L.bp = which == PL_BP ? T.bpargs : which == PL_INIT_BP ? T.init_bp : which == PL_HESS ? T.hess_bp : nullptr;
    L.fp = which == PL_FP ? T.fpargs : which == PL_INIT_FP ? T.init_fp : nullptr;
    L.off = T.pl_off + which * (num_scans + 1);
    L.dim = T.pl_dim + which * num_scans;
    L.order = T.pl_order + which * num_scans;
    const bool subsets = which == PL_BP || which == PL_FP;
    L.schedule = subsets ? T.schedule : nullptr;
    L.stride = 0;  // set by the caller (the number of subsets for the subset lists)
    L.counter = T.counters + which;
    L.planned = nullptr;
    return L;
}

__device__ __forceinline__ int find_scan(const int *__restrict__ off, int num_scans, int t) {
    int lo = 0, hi = num_scans;  // off[lo] <= t < off[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(off + mid) <= t) lo = mid; else hi = mid;
    }
    return lo;
}

// Sum of NV values over the block into slot[NV * t + i] (fixed order).
template <int NV>
__device__ __forceinline__ void tile_reduce(const double (&v)[NV], double *slot) {
    __shared__ double sh[32][NV];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const double a = warp_sum(v[i]);
        if (lane == 0) sh[warp][i] = a;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            double a = lane < BT_THREADS / 32 ? sh[lane][i] : 0.0;
            a = warp_sum(a);
            if (lane == 0) slot[i] = a;
        }
    }
    __syncthreads();
}

// Next tile of a dynamically scheduled work list (one atomic per CTA per tile).
__device__ __forceinline__ int fetch_tile(int *counter) {
    __shared__ int s_next;
    __syncthreads();  // every thread is done with the previous tile index
    if (threadIdx.x == 0) s_next = atomicAdd(counter, 1);
    __syncthreads();
    return s_next;
}

#ifndef MBX_BATCHED_FP_CAP
#define MBX_BATCHED_FP_CAP 2048  // most records per pass of the batched forward projections (and their stored passes)
#endif

// Record of scan s in a work list at a step.
template <class A>
__device__ __forceinline__ const A &list_record(const A *recs, const ProjList &L, int num_scans, int step, int s) {
    const int r = L.schedule ? __ldg(L.schedule + step * num_scans + s) : 0;
    return recs[s * L.stride + r];
}

// Sizes and plans of one scan of a batch (host side).
struct ScanSizes {
    long long ncyl, nsino, nrecon, npix;
    int el_tiles, sn_tiles, rc_tiles, flt_tiles;
    BpfPlan bpp;  // subset back projection
    CbPlan fpp;   // subset forward projection
    CbPlan ifp;   // initial forward projection, on the same channel blocks
    BpfPlan ibp;  // initial back projection over the region of reconstruction
    BpfPlan hbp;  // Hessian back projection over every pixel
    int hbp_slices;  // > 0: hbp is planned on one slice and broadcast to this many (unit-weight parallel beam)
    bool setup;   // the scan carries the set-up inputs
    int tr_tiles; // 32-channel blocks of the transposed copy over all views
};

// The back projections of a scan: of a subset, of the region of reconstruction (from the filtered sinogram), of every pixel
// (the Hessian).
enum { SW_SUBSET = 0, SW_INIT, SW_HESS, SW_COUNT };

// How a batch runs them, by list: whether they read windows of transposed copies, and the most slices of a tile.
struct BatchBp {
    bool windows[SW_COUNT];
    int most[SW_COUNT];
};

inline int scan_sizes(const mbx_scan &sc, ScanSizes &z, const BatchBp &B) {
    const mbx_geom &g = sc.geom;
    int rc = validate_geom(&g);
    if (rc != MBX_OK) return rc;
    if (!sc.flat_recon || !sc.error_sinogram || !sc.fm_hessian || !sc.partition) return MBX_ERR_INVALID_ARG;
    if (sc.num_subsets <= 0 || sc.subset_size <= 0) return MBX_ERR_INVALID_ARG;
    if (!(sc.qp.sigma_x > 0.0f) || !(sc.qp.T > 0.0f) || !(sc.qp.p > 0.0f)) return MBX_ERR_INVALID_ARG;
    z.bpp = plan_bp_fast(g, sc.subset_size, g.num_views, 0, B.most[SW_SUBSET]);
    // the channel blocks of either kernel variant (the tuner keeps the faster): the second's are the narrower
    z.fpp = plan_fp_cb(g, 0, 0, 2, cb_many(g.kind) >= 4 ? CB_MANY_CHANNELS : 128, 0, MBX_BATCHED_FP_CAP);
    z.ifp = z.fpp;
    if (!z.bpp.ok || !z.fpp.ok) return MBX_ERR_UNSUPPORTED;  // batched path needs the radius-1 kernels
    if ((long long)sc.subset_size * g.num_recon_slices >= (1LL << 31)) return MBX_ERR_UNSUPPORTED;
    if (sc.subset_size > (1 << 24)) return MBX_ERR_UNSUPPORTED;  // list positions share a word with the bin
    z.ncyl = (long long)sc.subset_size * g.num_recon_slices;
    z.nsino = (long long)g.num_views * g.num_det_rows * g.num_det_channels;
    z.npix = (long long)g.num_recon_rows * g.num_recon_cols;
    z.nrecon = z.npix * g.num_recon_slices;
    z.el_tiles = (int)((z.ncyl + BT_ELEM_TILE - 1) / BT_ELEM_TILE);
    z.sn_tiles = (int)((z.nsino + BT_SINO_TILE - 1) / BT_SINO_TILE);
    z.rc_tiles = (int)((z.nrecon + BT_SINO_TILE - 1) / BT_SINO_TILE);
    z.tr_tiles = g.num_views * ceil_div(g.num_det_channels + 2 * BPF_EDGE, 32);
    z.setup = sc.sinogram != nullptr || sc.full_indices != nullptr || sc.num_full_indices != 0;
    z.flt_tiles = 0;
    if (z.setup) {
        if (!sc.sinogram || !sc.full_indices || sc.num_full_indices <= 0 || sc.num_full_indices > z.npix)
            return MBX_ERR_INVALID_ARG;
        // the initial forward projection reads voxels by pixel index, which shares a word with the bin
        if (z.npix > (1 << 24) || z.nrecon >= (1LL << 31)) return MBX_ERR_UNSUPPORTED;
        z.hbp_slices = 0;
        if (bp_unit_broadcast(g, nullptr, sc.weights)) {  // unit-weight parallel Hessian: one slice, broadcast
            z.hbp = plan_bp_fast(one_slice_geometry(g), z.npix, g.num_views, 0, B.most[SW_HESS]);
            if (z.hbp.ok && z.hbp.splits == 1) z.hbp_slices = g.num_recon_slices;
        }
        if (z.hbp_slices == 0) z.hbp = plan_bp_fast(g, z.npix, g.num_views, 0, B.most[SW_HESS]);
        if (!z.hbp.ok) return MBX_ERR_UNSUPPORTED;
        if (g.kind != MBX_GEOM_TRANSLATION) {  // translation geometry starts from zeros (no direct recon)
            if (!filter_admits(g.num_det_channels, g.kind != MBX_GEOM_PARALLEL))
                return MBX_ERR_UNSUPPORTED;
            z.ibp = plan_bp_fast(g, sc.num_full_indices, g.num_views, 0, B.most[SW_INIT]);
            if (!z.ibp.ok) return MBX_ERR_UNSUPPORTED;
            z.flt_tiles = ceil_div((long long)g.num_views * g.num_det_rows, filter_shape(g.num_det_channels).rows);
        } else {
            z.ibp = z.hbp;  // unused
        }
    }
    return MBX_OK;
}

// Each back projection of a scan has a tensor map of its own, whose box holds the rows that its plan waits for: the height
// of its slice tiles, and so of its windows, follows its list.
inline const BpfPlan &scan_bp_plan(const ScanSizes &z, int which) {
    return which == SW_SUBSET ? z.bpp : which == SW_INIT ? z.ibp : z.hbp;
}
// Rows of the box of that map, in fours (0: no windows, or the scan has no such back projection).
inline int scan_window_box(const ScanSizes &z, int which, const BatchBp &B) {
    return B.windows[which] && (which == SW_SUBSET || z.setup) ? scan_bp_plan(z, which).boxq : 0;
}

// Sizes of every scan, and how the batch runs its back projections.  A unit's views follow one another, so a list whose
// units make less than about two waves of the chip's warps takes as long as one or two units: it reads its taps from the
// sinograms, in tiles as low (down to 8 slices) as still make one wave.  Stage of one step, us, gathering kernel of 16-slice
// tiles / windows / taps from the sinograms, 4 scans unless said: parallel 180 x 5 x 200 in 4 subsets (0.4 waves)
// 186 / 231 / 122, 360 x 64 x 300 in 8 (0.9) 1512 / 876 / 718, 16 scans of 360 x 28 x 300 in 8 (1.6) 2157 / 1336 / 1150,
// 360 x 28 x 437 in 4 (1.9) 2020 / 1123 / 1303, 16 scans of 180 x 40 x 200 in 4 (2.7) 884 / 630 / 768; cone 100 x 200 x 60
// in 8 (0.2) 510 / 798 / 189, 16 scans of 200 x 40 x 160 in 4 (1.6) 2540 / 1438 / 1397.  Translation geometry: as bp_windows.
constexpr double BATCH_WINDOW_WAVES = 1.75;
inline int batch_sizes(const mbx_scan *scans, int n, std::vector<ScanSizes> &zs, BatchBp &B) {
    const double slots = 8.0 * BPF_LAUNCH_WARPS * num_sms();
    for (int w = 0; w < SW_COUNT; ++w) {
        B.windows[w] = true;
        B.most[w] = BPF_ST;
    }
    zs.assign(n, ScanSizes{});
    auto plan = [&]() {
        for (int s = 0; s < n; ++s) {
            const int rc = scan_sizes(scans[s], zs[s], B);
            if (rc != MBX_OK) return rc;
        }
        return (int)MBX_OK;
    };
    auto waves = [&](int w) {
        double units = 0.0;
        for (int s = 0; s < n; ++s) {
            const BpfPlan &p = scan_bp_plan(zs[s], w);
            if (w != SW_SUBSET && !zs[s].setup) return 1e9;
            units += (double)p.gx * p.gy * BPF_WARPS;
        }
        return units / slots;
    };
    int rc = plan();
    for (int w = 0; w < SW_COUNT && rc == MBX_OK; ++w) {
        B.windows[w] = waves(w) >= BATCH_WINDOW_WAVES;
        for (int s = 0; s < n; ++s) {
            if (scans[s].geom.kind == MBX_GEOM_TRANSLATION && w == SW_SUBSET && 2 * scans[s].subset_size <= zs[s].npix)
                B.windows[w] = false;
            // every copy has to be addressable (32-bit offsets); the Hessian's needs weights to copy
            const mbx_geom &g = scans[s].geom;
            if ((long long)g.num_views * (g.num_det_channels + 2 * BPF_EDGE) * bpf_padded_rows(g) >= (1LL << 31) ||
                (w == SW_HESS && !scans[s].weights))
                B.windows[w] = false;
        }
        while (rc == MBX_OK && !B.windows[w] && B.most[w] > 8) {
            B.most[w] /= 2;
            rc = plan();
            if (rc != MBX_OK || waves(w) <= 1.1) continue;
            B.most[w] *= 2;  // too many for a wave
            rc = plan();
            break;
        }
    }
    return rc;
}

// The forward-projection stage kernels of one geometry kind: b_fp (walk), b_fp_replay (stored passes) and
// b_fp_build (store the passes), each compiled for 2 or cb_many resident CTAs per SM (minb).  fp_stage_kernel returns
// the kernel of (minb, mode) for occupancy queries and attributes; launch_fp_stage launches it over a work list.
const void *fp_stage_kernel(int kind, int minb, int mode);
void launch_fp_stage(int kind, int minb, int mode, int grid, size_t smem, cudaStream_t st, const ProjList &L, int n,
                     int step, int first, int total, int *err);

}  // namespace mbx
