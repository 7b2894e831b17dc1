// FBP / FDK sinogram filtering (sm_100a).
//
// Replaces ParallelBeamModel.fbp_filter (parallel_beam.py:303-348) and ConeBeamModel.fdk_filter
// (cone_beam.py:779-846) with the ramp filter of generate_direct_recon_filter (tomography_utils.py:4-35):
//   h[d] = 1/2 sinc(d) - 1/4 sinc(d/2)^2, d in [-(C-1), C-1]  ->  h[0] = 1/4, h[odd d] = -1/(pi d)^2, h[even] = 0
// and the 'valid' part of fftconvolve(row, h): out[i] = sum_j row[j] h[i - j].
// The convolution is evaluated directly (only the C/2 odd taps and the centre tap are nonzero); direct_filter.cuh has the
// arithmetic and how a block is spread over rows and outputs.
// FDK: the pre-weight D / sqrt(D^2 + u^2 + v^2) (cone_beam.py:806-818, detector_mn_to_uv :709-738) is applied
// while staging; both geometries apply the final pi / num_views.  Samples, taps and sums are float64 (the float32 sums of
// a direct convolution are off by a few 1e-6 of the row's scale, which the VCD iterations that start from this recon can
// amplify).
#include "direct_filter.cuh"
#include "mbx_host.hpp"

namespace mbx {

// FEW: blocks of fewer rows than filter_shape's default, `groups` of them (1.59 ms with a group count that the compiler does
// not know where 1.50 is taken without, 360 x 256 x 512).
template <bool WHOLE, bool FEW>
__global__ void __launch_bounds__(FILT_THREADS, 2)
direct_filter_kernel(const float *__restrict__ sino, float *__restrict__ out, long long num_rows_total, int R, int C,
                     int rows, double filter_scale, double out_scale, int fdk, double D, double delta_det_channel,
                     double delta_det_row, double det_channel_offset, double det_row_offset, int groups) {
    extern __shared__ __align__(16) double sm[];
    direct_filter_rows<WHOLE>(sino, out, (long long)blockIdx.x * rows, num_rows_total, R, C, filter_scale, out_scale, fdk,
                              D, delta_det_channel, delta_det_row, det_channel_offset, det_row_offset, sm,
                              FEW ? groups : 0);
}

}  // namespace mbx

extern "C" int mbx_direct_filter(const mbx_geom *g, const float *sinogram, float *out, void *stream) {
    int rc = mbx::validate_geom(g);
    if (rc != MBX_OK) return rc;
    if (!sinogram || !out || sinogram == out) return MBX_ERR_INVALID_ARG;
    // translation geometry has no direct reconstruction (the base TomographyModel's zeros,
    // tomography_model.py:934-964)
    if (g->kind == MBX_GEOM_TRANSLATION) return MBX_ERR_UNSUPPORTED;
    const int C = g->num_det_channels, R = g->num_det_rows;
    if (!mbx::filter_admits(C, g->kind != MBX_GEOM_PARALLEL)) return MBX_ERR_UNSUPPORTED;
    const long long rows_total = (long long)g->num_views * R;
    // blocks of fewer rows when the default's would leave SMs idle: a block's staging and taps are what such a call waits
    // for (209 x 16 x 95, FDK: 23 us with 52 blocks of 64 rows, 15 with 209 of 16)
    int groups = mbx::filter_shape(C).groups;
    while (groups > 1 && mbx::ceil_div(rows_total, 16 * groups) < 2 * mbx::num_sms()) groups /= 2;
    const size_t smem = mbx::filter_smem_bytes(C, groups);
    const auto kern = groups < mbx::filter_shape(C).groups ? mbx::direct_filter_kernel<false, true>
                      : mbx::filter_whole(C)               ? mbx::direct_filter_kernel<true, false>
                                                           : mbx::direct_filter_kernel<false, false>;
    {
        cudaError_t e = mbx::set_max_dynamic_smem(reinterpret_cast<const void *>(kern), 200 * 1024);
        if (e != cudaSuccess) return mbx::set_cuda_error(e);
    }
    double filter_scale, out_scale;
    int fdk;
    mbx::direct_filter_scales(*g, filter_scale, out_scale, fdk);
    const int rows = mbx::filter_shape(C, groups).rows;
    const unsigned blocks = (unsigned)((rows_total + rows - 1) / rows);
    kern<<<blocks, mbx::FILT_THREADS, smem, static_cast<cudaStream_t>(stream)>>>(
        sinogram, out, rows_total, R, C, rows, filter_scale, out_scale, fdk, g->source_detector_dist, g->delta_det_channel,
        g->delta_det_row, g->det_channel_offset, g->det_row_offset, groups);
    mbx::note_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? MBX_OK : mbx::set_cuda_error(e);
}
