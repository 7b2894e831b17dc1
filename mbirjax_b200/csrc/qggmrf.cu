// qGGMRF prior kernels (sm_100a).
//
// mbx_qggmrf_grad_hess replaces qggmrf_gradient_and_hessian_at_indices (qggmrf.py:118-148): the
// per-cylinder pass (qggmrf.py:151-188, zero differences beyond both ends of the cylinder) and the
// per-slice pass over the four in-slice neighbours with clipped indices (qggmrf.py:191-247), both built on
// get_2_b_tilde (qggmrf.py:250-279).  One thread per (subset pixel, slice), lanes along the slice axis, so
// every read of the centre and of each neighbour cylinder is coalesced.
//
// mbx_qggmrf_loss_grad replaces qggmrf_loss (qggmrf.py:31-65) and adds its analytic gradient (the
// reference differentiates it with autodiff): rho(a) = a^p/(p sigma^p) u/(1+u), u = (a/(T sigma))^(q-p),
// a = max(|delta|, T sigma eps), and rho'(delta) = sign(delta) a^(p-1)/sigma^p u (q/p + u)/(1+u)^2 (0 where
// the clip is active).  A voxel's gradient is the sum over its up-to-six neighbour differences (no atomics); the loss is
// reduced in float64 with a fixed-order two-stage reduction.
#include <algorithm>

#include "mbx_common.cuh"
#include "mbx_host.hpp"
#include "mbx_reduce.cuh"
#include "qggmrf.cuh"

namespace mbx {

__global__ void qggmrf_grad_hess_kernel(const float *__restrict__ recon, int nr, int nc, int ns,
                                        const int32_t *__restrict__ pix, long long num_pixels, const QParams q,
                                        float *__restrict__ grad_out, float *__restrict__ hess_out, int *err) {
    const long long total = num_pixels * ns;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long p = i / ns;
        const int k = (int)(i - p * ns);
        const int idx = pix[p];
        float g = 0.0f, h = 0.0f;
        if (idx < 0 || idx >= nr * nc) {
            flag_error(err, MBX_ERRFLAG_PIXEL);
        } else {
            qggmrf_voxel(recon, nr, nc, ns, idx, k, q, g, h);
        }
        grad_out[i] = g;
        hess_out[i] = h;
    }
}

// rho and rho' of one difference (both need the same power u).  p = 2 (the default) needs no other power.
__device__ __forceinline__ void qrho(float delta, const QParams &q, float &rho, float &prime) {
    const float a0 = fabsf(delta), a = fmaxf(a0, q.a_min);
    const float u = powf(a / q.t_sigma, q.q_minus_p);
    const float ap = q.p == 2.0f ? a * a : powf(a, q.p);
    const float ap1 = q.p == 2.0f ? a : powf(a, q.p_minus_1);
    rho = ap * q.inv_p_sigma_p * u / (1.0f + u);
    const float d = ap1 * q.inv_sigma_p * u * (q.q_over_p + u) / ((1.0f + u) * (1.0f + u));
    prime = a0 < q.a_min ? 0.0f : (delta < 0.0f ? -d : d);
    if (a0 != a0) prime = a0;
}

// A block's LOSS_THREADS threads hold as many consecutive (column, slice) elements and walk rows [r0, r1): the derivative
// of a difference is evaluated once, by the thread of its lower voxel, and its upper voxel takes it from the walk's last
// step (rows) or from shared memory (columns, slices; evaluated again at the block's own edge).  The kernel is bound by the
// arithmetic of the powers, about 100 instructions each: this way a voxel has 3 to 4 of them (p = 2) where evaluating
// rho and rho' of its six differences separately took 18; 256 x 256 x 128: 577 -> 188 us.
constexpr int LOSS_THREADS = 512;

__global__ void __launch_bounds__(LOSS_THREADS)
qggmrf_loss_grad_kernel(const float *__restrict__ x, int nr, int nc, int ns, int qblocks, int rows, const QParams q,
                        float *__restrict__ grad_out, double *__restrict__ partials) {
    __shared__ float s_col[2][LOSS_THREADS], s_sl[2][LOSS_THREADS];  // derivatives, by parity of the row
    const long long sr = (long long)nc * ns;  // row stride
    const int tid = threadIdx.x;
    const int chunk = blockIdx.x / qblocks;
    const long long e = (long long)(blockIdx.x - chunk * qblocks) * LOSS_THREADS + tid;
    const bool on = e < sr;
    const int col = on ? (int)(e / ns) : 0, k = on ? (int)(e - (long long)col * ns) : 0;
    const int r0 = chunk * rows, r1 = min(nr, r0 + rows);
    const bool has_col = on && col + 1 < nc, has_sl = on && k + 1 < ns;
    const float *p = x + (long long)r0 * sr + e;
    double loss = 0.0;
    float x0 = on ? __ldg(p) : 0.0f, up = 0.0f, unused;
    if (on && r0 > 0) qrho(x0 - __ldg(p - sr), q, unused, up);  // of the difference with the row before
    for (int row = r0; row < r1; ++row, p += sr) {
        float g = q.b_axis[0] * up, l = 0.0f, rho, xn = 0.0f, dc = 0.0f, ds = 0.0f;
        up = 0.0f;
        if (on && row + 1 < nr) {
            xn = __ldg(p + sr);
            qrho(xn - x0, q, rho, up);
            l += q.b_axis[0] * rho;
        }
        g -= q.b_axis[0] * up;
        if (has_col) {
            qrho(__ldg(p + ns) - x0, q, rho, dc);
            l += q.b_axis[1] * rho;
        }
        if (has_sl) {
            qrho(__ldg(p + 1) - x0, q, rho, ds);
            l += q.b_axis[2] * rho;
        }
        const int b = row & 1;
        s_col[b][tid] = dc;
        s_sl[b][tid] = ds;
        __syncthreads();  // (the other buffer's readers passed this barrier of the row before)
        if (on) {
            float pc = 0.0f, ps = 0.0f;
            if (col > 0) {
                if (tid >= ns)
                    pc = s_col[b][tid - ns];
                else
                    qrho(x0 - __ldg(p - ns), q, unused, pc);
            }
            if (k > 0) {
                if (tid >= 1)
                    ps = s_sl[b][tid - 1];
                else
                    qrho(x0 - __ldg(p - 1), q, unused, ps);
            }
            g += q.b_axis[1] * (pc - dc) + q.b_axis[2] * (ps - ds);
            if (grad_out) grad_out[(long long)row * sr + e] = g;
        }
        loss += (double)l;
        x0 = xn;
    }
    block_reduce_store(loss, partials);
}

// Blocks of elements of a row, rows of a block and blocks in all: about three waves of blocks of at least 8 rows, since a
// block's first row costs an extra evaluation; volumes that cannot give that many take fewer rows, down to one, as long
// as the blocks fit the chip at once (102 x 45 x 13: 22 us in walks of 8 rows, 7.5 in walks of one).
static void loss_shape(int nr, int nc, int ns, int &qblocks, int &rows, unsigned &blocks) {
    qblocks = ceil_div((long long)nc * ns, LOSS_THREADS);
    long long chunks = (9LL * num_sms() + qblocks - 1) / qblocks;
    const long long fit = (4LL * num_sms() + qblocks - 1) / qblocks;
    const long long most = std::max((long long)nr / 8, std::min((long long)nr, fit));
    if (chunks > most) chunks = most;
    if (chunks < 1) chunks = 1;
    rows = ceil_div(nr, chunks);
    blocks = (unsigned)((long long)qblocks * ceil_div(nr, rows));
}

int qggmrf_grad_hess(const float *recon, int nr, int nc, int ns, const int32_t *pix, long long num_pixels,
                     const mbx_qggmrf_params &qp, float *grad, float *hess, cudaStream_t st) {
    if (num_pixels == 0) return MBX_OK;
    const QParams q = make_qparams(qp);
    const long long total = num_pixels * ns;
    qggmrf_grad_hess_kernel<<<grid_for(total, 256), 256, 0, st>>>(recon, nr, nc, ns, pix, num_pixels, q, grad, hess,
                                                                   device_error_ptr());
    mbx::note_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? MBX_OK : set_cuda_error(e);
}

}  // namespace mbx

extern "C" int mbx_qggmrf_grad_hess(const float *flat_recon, int32_t num_recon_rows, int32_t num_recon_cols,
                                    int32_t num_recon_slices, const int32_t *pixel_indices, int64_t num_pixels,
                                    const mbx_qggmrf_params *qp, float *grad_out, float *hess_out, void *stream) {
    if (!flat_recon || !qp || num_recon_rows <= 0 || num_recon_cols <= 0 || num_recon_slices <= 0 || num_pixels < 0)
        return MBX_ERR_INVALID_ARG;
    if (num_pixels > 0 && (!pixel_indices || !grad_out || !hess_out)) return MBX_ERR_INVALID_ARG;
    if (!(qp->sigma_x > 0.0f) || !(qp->T > 0.0f) || !(qp->p > 0.0f)) return MBX_ERR_INVALID_ARG;
    return mbx::qggmrf_grad_hess(flat_recon, num_recon_rows, num_recon_cols, num_recon_slices, pixel_indices,
                                 num_pixels, *qp, grad_out, hess_out, static_cast<cudaStream_t>(stream));
}

extern "C" size_t mbx_qggmrf_loss_grad_workspace_bytes(int32_t num_recon_rows, int32_t num_recon_cols,
                                                       int32_t num_recon_slices) {
    if (num_recon_rows <= 0 || num_recon_cols <= 0 || num_recon_slices <= 0) return 0;
    int qblocks, rows;
    unsigned blocks;
    mbx::loss_shape(num_recon_rows, num_recon_cols, num_recon_slices, qblocks, rows, blocks);
    return mbx::align256(blocks * sizeof(double));
}

extern "C" int mbx_qggmrf_loss_grad(const float *recon, int32_t num_recon_rows, int32_t num_recon_cols,
                                    int32_t num_recon_slices, const mbx_qggmrf_params *qp, double *loss_out,
                                    float *grad_out, void *workspace, size_t workspace_bytes, void *stream) {
    if (!recon || !qp || !loss_out || num_recon_rows <= 0 || num_recon_cols <= 0 || num_recon_slices <= 0)
        return MBX_ERR_INVALID_ARG;
    if (!(qp->sigma_x > 0.0f) || !(qp->T > 0.0f) || !(qp->p > 0.0f)) return MBX_ERR_INVALID_ARG;
    int qblocks, rows;
    unsigned blocks;
    mbx::loss_shape(num_recon_rows, num_recon_cols, num_recon_slices, qblocks, rows, blocks);
    if (!workspace || workspace_bytes < blocks * sizeof(double)) return MBX_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const mbx::QParams q = mbx::make_qparams(*qp);
    double *partials = static_cast<double *>(workspace);
    mbx::qggmrf_loss_grad_kernel<<<blocks, mbx::LOSS_THREADS, 0, st>>>(
        recon, num_recon_rows, num_recon_cols, num_recon_slices, qblocks, rows, q, grad_out, partials);
    mbx::note_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return mbx::set_cuda_error(e);
    mbx::launch_sum_partials(partials, (int)blocks, 1, loss_out, st);
    e = cudaGetLastError();
    return e == cudaSuccess ? MBX_OK : mbx::set_cuda_error(e);
}
