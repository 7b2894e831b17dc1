// Sparse back projector for parallel-beam, cone-beam and translation geometry (sm_100a).
//
// Replaces Projectors.sparse_back_project (projectors.py:131-209) over the geometry plugins
// ParallelBeamModel.back_project_one_view_to_pixel_batch (parallel_beam.py:180-221),
// ConeBeamModel.back_project_one_view_to_pixel_batch (cone_beam.py:379-541) and
// TranslationModel.back_project_one_view_to_pixel_batch (translation_model.py:382-542); coeff_power = 2 gives
// the Hessian diagonal of TomographyModel.compute_hessian_diagonal (tomography_model.py:679-708).  Radius-1
// geometries run bp_fast.cuh when its plan fits (translation geometry when the caller gives a magnification
// bound); the other cases run the general kernel of back_project.cuh, described here.
//
// One thread owns one pixel and a tile of ST slices.  Its ST accumulators stay in registers across all
// views, so there are no global atomics and no per-view partial cylinders.  Lanes run along pixels, so the
// channel gathers of a warp fall in a narrow channel range of one detector row.  Per-view angle, cos and
// sin are staged in shared memory.  For cone beam each thread first gathers, for every detector row its
// slice tile touches in this view, the horizontal fan sum sum_k A_chan_k * sino[m, n_c + k] into its own
// column of a shared-memory buffer (row-major across threads, so conflict-free), then applies the
// voxel-centric vertical fan from that buffer; each detector row is therefore gathered once per view
// instead of once per vertical tap.  The optional weights are multiplied into every gathered value
// (a fused W * e).  Views may be split over CTAs with a fixed-order second-stage sum when there are too
// few pixels to fill the GPU (caller workspace).
#include <algorithm>

#include "back_project.cuh"
#include "bp_fast.cuh"
#include "bp_gather.cuh"

namespace mbx {

// Whether a call makes a transposed copy of its views (bp_fast.cuh): the copy's rows are addressed in 32 bits.
static bool bp_transposes(const mbx_geom &g, const BpfPlan &pl, long long num_pixels, int num_views_sel) {
    return bp_windows(g, pl, num_pixels, num_views_sel) &&
           (long long)g.num_views * (g.num_det_channels + 2 * BPF_EDGE) * bpf_padded_rows(g) < (1LL << 31);
}

bool bpf_window_map(CUtensorMap &map, const float *copy, const mbx_geom &g, int num_views_sel, int boxq) {
    using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = []() -> Encode {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000,
                                                               cudaEnableDefault, &found);
        return e == cudaSuccess && found == cudaDriverEntryPointSuccess ? reinterpret_cast<Encode>(fn) : nullptr;
    }();
    if (!encode || (reinterpret_cast<uintptr_t>(copy) & 15)) return false;
    const cuuint64_t rp = (cuuint64_t)bpf_padded_rows(g);
    const cuuint64_t dims[2] = {rp, (cuuint64_t)bpf_transposed_views(g, num_views_sel) *
                                        (cuuint64_t)(g.num_det_channels + 2 * BPF_EDGE)};
    const cuuint64_t strides[1] = {rp * 4};
    const cuuint32_t box[2] = {4u * (cuuint32_t)boxq, BPF_BOX}, elem[2] = {1, 1};
    return encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(copy), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Parallel-beam calls with values and no windows gather (bp_gather.cuh).
static bool bp_gathers(const mbx_geom &g, const BpfPlan &pl, long long num_pixels, int num_views_sel) {
    return g.kind == MBX_GEOM_PARALLEL && !bp_windows(g, pl, num_pixels, num_views_sel);
}

size_t bp_workspace_bytes(const mbx_geom &g, long long num_pixels, int num_views_sel) {
    const BpfPlan fp = plan_bp_fast(g, num_pixels, num_views_sel);
    if (!fp.ok) return plan_bp(g, num_pixels, num_views_sel).workspace;
    if (bp_gathers(g, fp, num_pixels, num_views_sel))  // (without values: the partial sums of the plan)
        return std::max(fp.workspace, plan_bp_gather(g, num_pixels, num_views_sel).workspace);
    return fp.workspace +
           (bp_transposes(g, fp, num_pixels, num_views_sel) ? bpf_transposed_bytes(g, num_views_sel) : 0);
}

size_t bp_noalloc_bytes(const mbx_geom &g, long long num_pixels, int num_views_sel) {
    const BpfPlan fp = plan_bp_fast(g, num_pixels, num_views_sel, 1);
    if (!fp.ok) return plan_bp(g, num_pixels, num_views_sel).workspace;
    return bp_gathers(g, fp, num_pixels, num_views_sel)
               ? std::max(fp.workspace, plan_bp_gather(g, num_pixels, num_views_sel).workspace)
               : fp.workspace;
}

static int back_project_gather(const mbx_geom &g, const float *sino, const float *w, const int32_t *pix,
                               long long num_pixels, const int32_t *views, int num_views_sel, int coeff_power,
                               float scale, float *out, void *ws, size_t ws_bytes, cudaStream_t st,
                               int splits_of = 0) {
    const BpgPlan pl = plan_bp_gather(g, num_pixels, num_views_sel, splits_of);
    if (pl.workspace > 0 && (ws == nullptr || ws_bytes < pl.workspace)) return MBX_ERR_WORKSPACE;
    const long long stride = num_pixels * (long long)g.num_recon_slices;
    const bool split = pl.splits > 1;
    float *dst = split ? static_cast<float *>(ws) : out;
    const BpgArgs A = {g,     sino, w,   pix, views, num_pixels, num_views_sel, coeff_power,
                       scale, dst,  split ? stride : 0, pl};
    bp_gather_kernel<<<dim3((unsigned)pl.gx, (unsigned)pl.gy, (unsigned)pl.splits), 256, 0, st>>>(A, device_error_ptr());
    note_launch();
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && split) {
        launch_split_sum(dst, stride, pl.splits, scale, out, stride, st);
        e = cudaGetLastError();
    }
    return e == cudaSuccess ? MBX_OK : set_cuda_error(e);
}

__global__ void __launch_bounds__(256) bp_transpose_kernel(const float *__restrict__ src, const float *__restrict__ wts,
                                                           const int32_t *__restrict__ views, int num_views,
                                                           int first, float *__restrict__ dst, int num_rows,
                                                           int num_channels, int rp) {
    const int j = first + blockIdx.y;
    const int vi = views ? views[j] : j;
    if (vi < 0 || vi >= num_views) return;  // flagged and skipped by the projection
    const int rows = 32 * ceil_div(ceil_div(rp, 32), (int)gridDim.z);  // per block: 32, in all but absurdly tall views
    bpf_transpose_block(src, wts, dst, (long long)vi * num_rows * num_channels,
                        (long long)j * (num_channels + 2 * BPF_EDGE) * rp, blockIdx.x * 32, blockIdx.z * rows,
                        min(rp, ((int)blockIdx.z + 1) * rows), num_rows, num_channels, rp);
}

template <int KIND, bool TR>
static cudaError_t launch_bp_fast_kind(const BpArgs &A, const CUtensorMap &map, cudaStream_t st) {
    auto kern = bp_fast_kernel<KIND, TR>;
    const cudaError_t ea = set_max_dynamic_smem(reinterpret_cast<const void *>(kern), 100 * 1024);
    if (ea != cudaSuccess) return ea;
    constexpr int W = bpf_launch_warps(TR);
    const dim3 grid((unsigned)(A.plan.gx * A.plan.gy * (BPF_WARPS / W)), A.plan.splits);
    kern<<<grid, 32 * W, bpf_smem_bytes(KIND, W, TR), st>>>(A, map, device_error_ptr());
    note_launch();
    return cudaGetLastError();
}

template <bool TR>
static cudaError_t launch_bp_fast(const BpArgs &A, const CUtensorMap &map, cudaStream_t st) {
    switch (A.g.kind) {
        case MBX_GEOM_PARALLEL: return launch_bp_fast_kind<MBX_GEOM_PARALLEL, TR>(A, map, st);
        case MBX_GEOM_CONE: return launch_bp_fast_kind<MBX_GEOM_CONE, TR>(A, map, st);
        default: return launch_bp_fast_kind<MBX_GEOM_TRANSLATION, TR>(A, map, st);
    }
}

int back_project(const mbx_geom &g, const float *sino, const float *w, const int32_t *pix, long long num_pixels,
                 const int32_t *views, int num_views_sel, int coeff_power, float scale, float *out, void *ws,
                 size_t ws_bytes, cudaStream_t st, bool noalloc) {
    if (num_pixels == 0) return MBX_OK;
    BpArgs A = {};
    A.g = g;
    A.sino = sino;
    A.wts = w;
    A.pix = pix;
    A.num_pixels = num_pixels;
    A.views = views;
    A.num_views_sel = num_views_sel;
    A.coeff_power = coeff_power;
    A.scale = scale;
    A.out = out;
    CUtensorMap map = {};
    if (bp_unit_broadcast(g, sino, w)) {  // unit-weight parallel Hessian: one slice, written to every slice
        A.g = one_slice_geometry(g);
        A.plan = plan_bp_fast(A.g, num_pixels, num_views_sel, noalloc);
        if (A.plan.ok && A.plan.splits == 1) {
            A.views_per_split = A.plan.views_per_split;
            A.out_slices = g.num_recon_slices;
            const cudaError_t e = launch_bp_fast<false>(A, map, st);
            return e == cudaSuccess ? MBX_OK : set_cuda_error(e);
        }
        A.g = g;
    }
    A.plan = plan_bp_fast(g, num_pixels, num_views_sel, noalloc);
    if (A.plan.ok && sino && bp_gathers(g, A.plan, num_pixels, num_views_sel))
        return back_project_gather(g, sino, w, pix, num_pixels, views, num_views_sel, coeff_power, scale, out, ws,
                                   ws_bytes, st);
    if (A.plan.ok) {
        bool tr = !noalloc && sino && bp_transposes(g, A.plan, num_pixels, num_views_sel);
        const size_t need = A.plan.workspace + (tr ? bpf_transposed_bytes(g, num_views_sel) : 0);
        if (need > 0 && (ws == nullptr || ws_bytes < need)) {
            if (noalloc || ws_bytes < bp_noalloc_bytes(g, num_pixels, num_views_sel)) return MBX_ERR_WORKSPACE;
            return back_project(g, sino, w, pix, num_pixels, views, num_views_sel, coeff_power, scale, out, ws, ws_bytes,
                                st, true);  // no room for a transposed copy: without one
        }
        float *copy = reinterpret_cast<float *>(static_cast<char *>(ws) + A.plan.workspace);
        tr = tr && bpf_window_map(map, copy, g, num_views_sel, A.plan.boxq);
        // parallel with windows by its size, but no room or no map for them: the gather in the windows' splits, so that the
        // sums are the same (720 x 64 x 512 subset of 4: the gather takes 2.26 ms, reading taps as bp_direct_unit does 4.5)
        if (g.kind == MBX_GEOM_PARALLEL && sino && !tr)
            return back_project_gather(g, sino, w, pix, num_pixels, views, num_views_sel, coeff_power, scale, out, ws,
                                       ws_bytes, st, A.plan.splits);
        const long long stride = num_pixels * (long long)g.num_recon_slices;
        A.views_per_split = A.plan.views_per_split;
        if (A.plan.splits > 1) {
            A.out = static_cast<float *>(ws);
            A.split_stride = stride;
        }
        cudaError_t e = cudaSuccess;
        if (tr) {
            A.tsino = copy;
            A.rp = bpf_padded_rows(g);
            const int nt = bpf_transposed_views(g, num_views_sel);
            A.tsino_all = num_views_sel > g.num_views || !views ? 1 : 0;
            const int32_t *tv = A.tsino_all ? nullptr : views;
            // views in grid.y, at most 65535 per launch
            for (int j0 = 0; j0 < nt && e == cudaSuccess; j0 += 65535) {
                bp_transpose_kernel<<<dim3((unsigned)ceil_div(g.num_det_channels + 2 * BPF_EDGE, 32), (unsigned)std::min(nt - j0, 65535),
                                           (unsigned)std::min((long long)ceil_div(A.rp, 32), 65535LL)),
                                      256, 0, st>>>(sino, w, tv, g.num_views, j0, copy, g.num_det_rows,
                                                    g.num_det_channels, A.rp);
                note_launch();
                e = cudaGetLastError();
            }
            if (e == cudaSuccess) e = launch_bp_fast<true>(A, map, st);
        } else {
            e = launch_bp_fast<false>(A, map, st);
        }
        if (e == cudaSuccess && A.plan.splits > 1) {
            launch_split_sum(A.out, stride, A.plan.splits, scale, out, stride, st);
            e = cudaGetLastError();
        }
        return e == cudaSuccess ? MBX_OK : set_cuda_error(e);
    }
    const BpPlan pl = plan_bp(g, num_pixels, num_views_sel);
    if (pl.workspace > 0 && (ws == nullptr || ws_bytes < pl.workspace)) return MBX_ERR_WORKSPACE;
    float *dst = pl.splits > 1 ? static_cast<float *>(ws) : out;
    const long long stride = num_pixels * (long long)g.num_recon_slices;
    const long long ss = pl.splits > 1 ? stride : 0;
    cudaError_t e;
    if (g.kind == MBX_GEOM_PARALLEL)
        e = launch_bp_parallel(g, pl, sino, w, pix, num_pixels, views, num_views_sel, coeff_power, scale, dst, ss, st);
    else if (g.kind == MBX_GEOM_CONE)
        e = launch_bp_cone(g, pl, sino, w, pix, num_pixels, views, num_views_sel, coeff_power, scale, dst, ss, st);
    else
        e = launch_bp_translation(g, pl, sino, w, pix, num_pixels, views, num_views_sel, coeff_power, scale, dst, ss,
                                  st);
    if (e != cudaSuccess) return set_cuda_error(e);
    if (pl.splits > 1) {
        launch_split_sum(dst, stride, pl.splits, scale, out, stride, st);
        e = cudaGetLastError();
        if (e != cudaSuccess) return set_cuda_error(e);
    }
    return MBX_OK;
}

}  // namespace mbx

extern "C" size_t mbx_back_project_workspace_bytes(const mbx_geom *g, int64_t num_pixels, int32_t num_views_sel) {
    if (mbx::validate_geom(g) != MBX_OK || num_pixels < 0 || num_views_sel <= 0) return 0;
    return mbx::bp_workspace_bytes(*g, num_pixels, num_views_sel);
}

extern "C" size_t mbx_back_project_least_workspace_bytes(const mbx_geom *g, int64_t num_pixels, int32_t num_views_sel) {
    if (mbx::validate_geom(g) != MBX_OK || num_pixels < 0 || num_views_sel <= 0) return 0;
    return std::min(mbx::bp_workspace_bytes(*g, num_pixels, num_views_sel),
                    mbx::bp_noalloc_bytes(*g, num_pixels, num_views_sel));
}

extern "C" int mbx_sparse_back_project(const mbx_geom *g, const float *sinogram, const float *weights,
                                       const int32_t *pixel_indices, int64_t num_pixels, const int32_t *view_indices,
                                       int32_t num_views_sel, int32_t coeff_power, float scale, float *out,
                                       void *workspace, size_t workspace_bytes, void *stream) {
    int rc = mbx::validate_geom(g);
    if (rc != MBX_OK) return rc;
    if (num_pixels < 0 || num_views_sel <= 0) return MBX_ERR_INVALID_ARG;
    if (num_pixels > 0 && (!pixel_indices || !out)) return MBX_ERR_INVALID_ARG;
    if (coeff_power != 1 && coeff_power != 2) return MBX_ERR_UNSUPPORTED;
    if (!view_indices && num_views_sel > g->num_views) return MBX_ERR_INVALID_ARG;
    if (!sinogram) {  // no sinogram: the values are the weights, or 1 everywhere when there are none either
        sinogram = weights;
        weights = nullptr;
    }
    return mbx::back_project(*g, sinogram, weights, pixel_indices, num_pixels, view_indices, num_views_sel,
                             coeff_power, scale, out, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}
