// Back projector specialised for psf_radius == 1 (the reference's default geometry: delta_voxel equal to the
// detector pitch at the magnification).  Same contract and arithmetic as the general bp_kernel (back_project.cuh);
// organised so that a (pixel, slice, view) costs few instructions and its detector samples come from shared memory:
//
//  * A warp owns 32 pixels (one per lane) x a tile of ts <= BPF_ST slices, with the accumulators of a lane's slices in
//    registers (as pairs, for the two-wide FMA) across all views.  Warps share nothing, so they run without barriers; a plan
//    counts them in tiles of eight, and a launch puts two (four without windows) in a CTA.
//  * Per view each lane computes the footprint of its pixel in registers: centre channel, three coefficients
//    (already raised to coeff_power, zero off the detector), and for the fan geometries the affine map slice ->
//    detector row m_p(k) = A0 + k*A1 and the vertical-angle factor c2 = (mag/D)^2, 1/cos(phi_k) = sqrt(1 + c2 z_k^2).
//    It is trig-free: cos/sin(theta - theta_p) and 1/cos(theta_p) come from the per-view cos/sin and
//    rsqrt(D^2 + u^2) instead of atan2/cos/sin per pixel.
//  * The channels and rows that the warp's footprints touch (their exact range, by warp min/max) are a small window
//    of the view, about 20 to 36 channels wide for a compact pixel list.  Calls that bp_windows() names first make a
//    transposed copy of their sinogram (view, channel, row; weights multiplied in, zeros off the detector), whose windows
//    the TMA unit copies into the warp's own shared memory, channels outermost (boxes of 8 channels; no load or store
//    instruction, and no share of the load/store pipe, which bounds the kernel), so that a lane reads four rows of a
//    channel with one 16-byte load at a constant offset; the channel pitch is an odd number of 16-byte units, so lanes on
//    neighbouring channels hit different banks.  The other calls read their taps from the sinogram itself
//    (bp_direct_unit, bp_gather.cuh).
//  * Fan geometries: a lane first forms the horizontal sum of each window row in its own column of a row buffer
//    ([row][lane], conflict-free), then the vertical fan reads three of its rows per slice with no bounds tests.
//    plan_bp_fast admits a geometry only when the rows of a slice tile (ts * max |dm/dk| + 4) fit that buffer.
//    Measured (B200, one subset of 4 unless said): parallel 652 x 57 x 437 1724 -> 885 us a call against the kernel that
//    gathered each tap from global memory (21 instructions per slice and view there, 12 here), cone 360 x 256 x 512
//    (subset of 8) 11.98 -> 6.34 ms, translation 49 x 128 x 128 (all pixels) 197 -> 107 us, weighted squared cone
//    180 x 61 x 203 2.41 -> 1.29 ms; with windows copied by 16-byte cp.async instead of the TMA the parallel call took
//    975 us.
//  * Pixels without locality, which would need many windows, are handled some lanes at a time, each with private
//    columns of its own taps in the place of the window.
#pragma once

#include <cuda.h>  // CUtensorMap

#include <algorithm>
#include <type_traits>

#include "back_project.cuh"

namespace mbx {

constexpr int BPF_THREADS = 256;
constexpr int BPF_WARPS = BPF_THREADS / 32;
#ifndef MBX_BPF_ST
#define MBX_BPF_ST 32
#endif
constexpr int BPF_ST = MBX_BPF_ST;  // most slices per thread (a multiple of 4)
constexpr int BPF_CACHE_ROWS = 48;  // row-buffer depth (fan geometries): ts * max|dm/dk| + 4 must fit
constexpr int BPF_BOX = 8;          // channels per TMA box
constexpr int BPF_EDGE = 2;         // channels of zeros on either side of a view of the transposed copy
constexpr int BPF_FAN_QUADS = 13;   // most rows of a fan window and of the row buffer, in fours: BPF_CACHE_ROWS and the
                                    // rounding of the first row down to a multiple of 4
// A warp whose pixels need several windows of a view copies them one by one while their channels fall in at most
// BPF_WINDOWS stretches of BPF_SPLIT channels.
constexpr int BPF_SPLIT = 32;
constexpr int BPF_WINDOWS = 4;
// Window floats: 32 channels of 36 rows (parallel, two buffers), 32 channels of 52 rows (fan geometries).
constexpr int BPF_WIN_PARALLEL = 32 * 36;
constexpr int BPF_WIN_FAN = 32 * 4 * BPF_FAN_QUADS;

struct BpfPlan {
    int nsl;      // slice tiles per CTA (warps per pixel group)
    int npg;      // pixel groups of 32 per CTA
    int lg_pcta;  // log2(32 * npg)
    int chunk;    // footprints staged ahead of their use: 0, a lane computes its own pixel's when it needs them
    int vc;       // views whose constants a warp holds at a time
    int inline_fp;  // 1 (see chunk)
    int ts;       // slices per tile (<= BPF_ST)
    int boxq;     // rows of a window in fours, an odd number
    int tiles;    // ceil(S / ts)
    int gx, gy, splits, views_per_split;
    size_t smem, workspace;  // of a launched CTA; the partial sums of the splits
    bool ok;
};

// Pairs of floats in one 64-bit register, for the two-wide FMA / add / multiply (each half rounded on its own).
using bpf2 = unsigned long long;
__device__ __forceinline__ bpf2 bpf_pair(float a, float b) {
    bpf2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void bpf_unpair(bpf2 v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ bpf2 bpf_fma(bpf2 a, bpf2 b, bpf2 c) {
    bpf2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ bpf2 bpf_mul(bpf2 a, bpf2 b) {
    bpf2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ bpf2 bpf_add(bpf2 a, bpf2 b) {
    bpf2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// Shared memory at byte address a + OFS: one float, or four as two pairs.
template <int OFS>
__device__ __forceinline__ float bpf_lds(unsigned a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFS));
    return v;
}
template <int OFS>
__device__ __forceinline__ void bpf_lds4(unsigned a, bpf2 &x, bpf2 &y) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2+%3];" : "=l"(x), "=l"(y) : "r"(a), "n"(OFS));
}
// A loop over I = 0 .. N-1 with I a constant (for immediate offsets).
template <int I, int N, class F>
__device__ __forceinline__ void bpf_for(F f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        bpf_for<I + 1, N>(f);
    }
}

// Footprint of one (pixel, view): first of the channels that can hold a nonzero tap (nc - 1, or with two taps nc - 1
// or nc) and the coefficients of the channels from there (0 off the detector); fan geometries: row map A0 + k*A1,
// c2 = (mag/D)^2 and the slice-height offset (translation).
struct BpfFoot {
    int ch;
    float a[3];
    float A0, A1, c2, zv;
};

// vw, one view's constants: x, y = cos, sin of the angle (translation: tx, ty); z = tz (translation) or delta_voxel /
// cos_alpha (parallel); w = element offset of the view in the sinogram (int bits; -1: invalid view).
template <int KIND>
__device__ __forceinline__ void bpf_footprint(const mbx_geom &g, const float4 &vw, float x_tilde, float y_tilde,
                                              int coeff_power, bool two, BpfFoot &f) {
    const float cs = vw.x, sn = vw.y;
    const float inv_dc = 1.0f / g.delta_det_channel;
    const int num_channels = g.num_det_channels;
    const float det_center_channel = 0.5f * (float)(num_channels - 1);
    float n_p, w, scale;  // scale = delta_voxel / cos_alpha
    if (KIND == MBX_GEOM_TRANSLATION) {
        // no rotation (translation_model.py:595-656).  Coefficient L / cos(theta_p), no delta_voxel factor; the
        // vertical fan is the cone's with slice heights delta_voxel k + zv, zv = -tz - delta_voxel (S-1)/2.
        const float x_p = x_tilde - cs;
        const float y_p = y_tilde - sn;
        const float inv_d = 1.0f / g.source_detector_dist;
        const float mag = 1.0f / (1.0f / g.magnification - y_p * inv_d);
        const float u = mag * x_p;
        n_p = (u + g.det_channel_offset) * inv_dc + det_center_channel;
        const float t = u * inv_d;
        const float cos_tp = rsqrtf(fmaf(t, t, 1.0f));
        w = mag * (g.delta_voxel * inv_dc);
        scale = 1.0f / cos_tp;
        const float inv_dr = 1.0f / g.delta_det_row;
        const float z0v = -vw.z - g.delta_voxel * (0.5f * (float)(g.num_recon_slices - 1));
        const float mr = mag * inv_d;
        f.A0 = (mag * z0v + g.det_row_offset) * inv_dr + 0.5f * (float)(g.num_det_rows - 1);
        f.A1 = mag * g.delta_voxel * inv_dr;
        f.c2 = mr * mr;
        f.zv = z0v;
    } else if (KIND == MBX_GEOM_PARALLEL) {
        const float x = cs * x_tilde - sn * y_tilde;
        n_p = (x + g.det_channel_offset) * inv_dc + det_center_channel;
        const float cos_alpha = fmaxf(fabsf(cs), fabsf(sn));
        w = (g.delta_voxel * inv_dc) * cos_alpha;
        scale = vw.z;
    } else {
        const float x_p = cs * x_tilde - sn * y_tilde;
        const float y_p = sn * x_tilde + cs * y_tilde;
        const float inv_d = isinf(g.source_detector_dist) ? 0.0f : 1.0f / g.source_detector_dist;
        const float mag = 1.0f / (1.0f / g.magnification - y_p * inv_d);
        const float u = mag * x_p;
        n_p = (u + g.det_channel_offset) * inv_dc + det_center_channel;
        // theta_p = atan2(u, D): cos = D / h, sin = u / h with h = sqrt(D^2 + u^2)  (D = inf: cos 1, sin 0)
        const float t = u * inv_d;
        const float inv_h = rsqrtf(fmaf(t, t, 1.0f));                    // cos(theta_p)
        const float cos_tp = inv_h, sin_tp = t * inv_h;
        const float cd = cs * cos_tp + sn * sin_tp;                       // cos(theta - theta_p)
        const float sd = sn * cos_tp - cs * sin_tp;                       // sin(theta - theta_p)
        const float cos_alpha = fmaxf(fabsf(cd), fabsf(sd));
        w = mag * (g.delta_voxel * inv_dc) * (cos_alpha / cos_tp);
        scale = g.delta_voxel / cos_alpha;
        const float inv_dr = 1.0f / g.delta_det_row;
        const float center_slice = 0.5f * (float)(g.num_recon_slices - 1);
        const float z0 = g.recon_slice_offset - g.delta_voxel * center_slice;
        const float mr = mag * inv_d;
        f.A0 = (mag * z0 + g.det_row_offset) * inv_dr + 0.5f * (float)(g.num_det_rows - 1);
        f.A1 = mag * g.delta_voxel * inv_dr;
        f.c2 = mr * mr;
        f.zv = z0;
    }
    const int nc = (int)rintf(n_p);
    const float half_w = (w + 1.0f) * 0.5f;
    const float l_max = fminf(1.0f, w);
    const float d = n_p - (float)nc;
    if (KIND == MBX_GEOM_PARALLEL && two) {
        // w <= 1: the voxel reaches at most one of the two neighbours, the one on its side of the centre channel
        const bool up = d > 0.0f;
        f.ch = up ? nc : nc - 1;
        const float c = scale * fminf(fmaxf(half_w - fabsf(d), 0.0f), l_max);
        const float e = scale * fminf(fmaxf(half_w - fabsf(d - (up ? 1.0f : -1.0f)), 0.0f), l_max);
        f.a[0] = up ? c : e;
        f.a[1] = up ? e : c;
        f.a[2] = 0.0f;
    } else {
        f.ch = nc - 1;
#pragma unroll
        for (int k = 0; k < 3; ++k)
            f.a[k] = scale * fminf(fmaxf(half_w - fabsf(d - (float)(k - 1)), 0.0f), l_max);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if ((unsigned)(f.ch + k) >= (unsigned)num_channels) f.a[k] = 0.0f;
        if (coeff_power == 2) f.a[k] *= f.a[k];
    }
}

// Pixel position relative to the recon centre (ALU): x from the column, y from the row (translation geometry
// spaces rows by delta_recon_row).
template <int KIND>
__device__ __forceinline__ void bpf_pixel(const mbx_geom &g, int idx, float &x_tilde, float &y_tilde) {
    if (KIND == MBX_GEOM_TRANSLATION) {
        const int row = idx / g.num_recon_cols;
        const int col = idx - row * g.num_recon_cols;
        x_tilde = g.delta_voxel * ((float)col - 0.5f * (float)(g.num_recon_cols - 1));
        y_tilde = g.delta_recon_row * ((float)row - 0.5f * (float)(g.num_recon_rows - 1));
    } else {
        pixel_tilde(g, idx, x_tilde, y_tilde);
    }
}

// Arguments of one back projection (one scan).
struct BpArgs {
    mbx_geom g;
    const float *sino;         // full sinogram (num_views, R, C)
    const float *wts;          // optional weights, same shape (NULL: ones)
    const float *tsino;        // weights x sinogram of the call's views as (view, channel, rp rows), or NULL
    int rp;                    // rows of tsino, a multiple of 4 (0 past num_det_rows)
    const CUtensorMap *tmap;   // its tensor map (batched lists; a plain launch passes the map as a parameter)
    int tsino_all;             // tsino holds every view of the geometry (else the selected views in their order)
    const int32_t *pix;        // (num_pixels,) flat pixel indices
    long long num_pixels;
    const int32_t *order;      // optional permutation of [0, num_pixels): processing order (locality)
    const int32_t *views;      // (num_views_sel,) or NULL
    int num_views_sel, views_per_split, coeff_power;
    float scale;
    float *out;                // (num_pixels, S) in list order, or a flat recon when out_by_index
    long long split_stride;    // 0: final output; else partial-sum workspace stride
    int out_by_index;
    int out_slices;            // > 0: g has one slice and its value is written to all out_slices slices of the
                               // output cylinder (the unit-weight Hessian of parallel beam, equal in every slice)
    BpfPlan plan;
};

// Parallel beam with neither sinogram nor weights (the unit-weight Hessian diagonal): every detector row holds the
// same ones and every slice the same footprints, so all slices of a pixel receive the same sum of the same terms
// in the same order.  The back projection is then planned on one slice (one_slice_geometry) and that value is
// written to every slice.
inline bool bp_unit_broadcast(const mbx_geom &g, const float *sino, const float *wts) {
    return g.kind == MBX_GEOM_PARALLEL && !sino && !wts && g.num_recon_slices > 1;
}

inline mbx_geom one_slice_geometry(const mbx_geom &g) {
    mbx_geom g1 = g;
    g1.num_recon_slices = 1;
    return g1;
}

// Read-only load of *p when ok, else 0 (a predicated load: no branch, so several stay in flight).
__device__ __forceinline__ float bpf_ldg(const float *p, bool ok) {
    float v = 0.0f;
    asm("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q ld.global.nc.f32 %0, [%1];\n\t}" : "+f"(v) : "l"(p), "r"((int)ok));
    return v;
}

// One warp's TMA barriers (one per window buffer; byte addresses in shared memory) and their phase parities.
struct BpfPipe {
    unsigned bar;
    unsigned parity;  // bit b: parity that buffer b waits for next
    bool failed;      // a copy did not complete: the warp's work ends
};

__device__ __forceinline__ BpfPipe bpf_pipe_init(float *at) {
    BpfPipe p;
    p.bar = (unsigned)__cvta_generic_to_shared(at);
    p.parity = 0;
    p.failed = false;
    if ((threadIdx.x & 31) == 0) {
        asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(p.bar) : "memory");
        asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(p.bar + 8) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    return p;
}

__device__ __forceinline__ bool bpf_try_wait(unsigned bar, unsigned parity) {
    unsigned done;
    asm volatile("{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.shared.b64 q, [%1], %2;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done != 0;
}

__device__ __forceinline__ unsigned long long bpf_now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Waits for buffer b's copy; the same answer in every lane.  A copy takes some microseconds; one that has not completed
// after BPF_WAIT_NS (BPF_WAIT_AGAIN_NS once the device error word says that another failed, so that a launch of many warps
// ends soon) never will: the error is flagged, and the caller ends its unit.
constexpr unsigned long long BPF_WAIT_NS = 250000000, BPF_WAIT_AGAIN_NS = 2000000;
__device__ __forceinline__ bool bpf_pipe_wait(BpfPipe &p, int b, int *err) {
    const unsigned bar = p.bar + 8u * (unsigned)b, par = (p.parity >> b) & 1u;
    p.parity ^= 1u << b;
    bool done = bpf_try_wait(bar, par);
    if (__all_sync(0xffffffffu, done)) return true;
    const unsigned long long t0 = bpf_now_ns();
    for (;;) {
        for (int i = 0; i < 64 && !done; ++i) done = bpf_try_wait(bar, par);
        if (__all_sync(0xffffffffu, done)) return true;
        const bool again = err && (*reinterpret_cast<volatile int *>(err) & MBX_ERRFLAG_CACHE);
        if (__any_sync(0xffffffffu, bpf_now_ns() - t0 > (again ? BPF_WAIT_AGAIN_NS : BPF_WAIT_NS))) break;
    }
    flag_error(err, MBX_ERRFLAG_CACHE);
    p.failed = true;
    return false;
}

// True in one lane of the (converged) warp, by elect.sync, which the compiler knows to leave a single thread: it then
// issues the TMA instructions without a loop over the threads that might execute them.
__device__ __forceinline__ bool bpf_elect() {
    unsigned one;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(one));
    return one != 0;
}

// Before a warp's first copies through a tensor map in global memory: the map was written by a copy to the device, and
// the TMA unit reads maps through a cache of its own, which may hold what stood there before.
__device__ __forceinline__ void bpf_acquire_map(const CUtensorMap *tmap) {
    asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(tmap) : "memory");
    __syncwarp();
}

// Starts the TMA copy of channels c .. c + nch - 1 (rows of the transposed copy, counted over views and edge channels)
// and rows r0 .. (a multiple of 4) into buffer b at win; rows outside the copy arrive as zeros.  c, nch, r0 and b are the
// warp's.
__device__ __forceinline__ void bpf_stage_tma(float *win, const BpArgs &A, const CUtensorMap *tmap, const BpfPipe &p,
                                              int b, int r0, int c, int nch) {
    const unsigned box = 16u * BPF_BOX * (unsigned)A.plan.boxq;
    const int n = (nch + BPF_BOX - 1) / BPF_BOX;
    c = __shfl_sync(0xffffffffu, c, 0);
    r0 = __shfl_sync(0xffffffffu, r0, 0);
    unsigned dst = __shfl_sync(0xffffffffu, (unsigned)__cvta_generic_to_shared(win), 0);
    const unsigned bar = __shfl_sync(0xffffffffu, p.bar + 8u * (unsigned)b, 0);
    if (bpf_elect()) {
        asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(bar), "r"(box * (unsigned)n) : "memory");
        for (int i = 0; i < n; ++i, dst += box, c += BPF_BOX)
            asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                         ::"r"(dst), "l"(tmap), "r"(r0), "r"(c), "r"(bar)
                         : "memory");
    }
}

// A lane's own channels ch .. ch + taps - 1 (on the view or its edge channels), rows r0 .. r0 + 4 nq - 1, into its private
// columns at win.
__device__ __forceinline__ void bpf_stage_private(float *win, const BpArgs &A, int voff, int r0, int nq, int pitch,
                                                  int ch, int taps) {
    for (int k = 0; k < taps; ++k) {
        float *dst = win + k * pitch;
        const float *src = A.tsino + (long long)(voff + ch + k + BPF_EDGE) * A.rp;
        for (int q = 0, r = r0; q < nq; ++q, r += 4) {
            const bool ok = r >= 0 && r < A.rp;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;"
                         ::"r"((unsigned)__cvta_generic_to_shared(dst + 4 * q)), "l"(ok ? src + r : A.tsino), "r"(ok ? 16 : 0)
                         : "memory");
        }
    }
}

// Waits for this warp's private columns.
__device__ __forceinline__ void bpf_private_wait() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // before the next TMA copy into the buffer
}

// The constants of view v of a call, see bpf_footprint.
template <int KIND, bool TR>
__device__ __forceinline__ float4 bpf_view(const BpArgs &A, int v) {
    const mbx_geom &g = A.g;
    const int vi = A.views ? A.views[v] : v;
    const bool ok = vi >= 0 && vi < g.num_views;
    float4 vw;
    if (KIND == MBX_GEOM_TRANSLATION) {
        vw.x = ok ? g.translations[3 * vi] : 0.0f;
        vw.y = ok ? g.translations[3 * vi + 1] : 0.0f;
        vw.z = ok ? g.translations[3 * vi + 2] : 0.0f;
    } else {
        const float ang = ok ? g.angles[vi] : 0.0f;
        vw.x = cosf(ang);
        vw.y = sinf(ang);
        vw.z = KIND == MBX_GEOM_PARALLEL ? g.delta_voxel / fmaxf(fabsf(vw.x), fabsf(vw.y)) : 0.0f;
    }
    // TR: first channel of the view in the transposed copy; otherwise the element offset of the view
    vw.w = __int_as_float(!ok ? -1
                          : TR ? (A.tsino_all ? vi : v) * (g.num_det_channels + 2 * BPF_EDGE)
                               : vi * (g.num_det_rows * g.num_det_channels));
    return vw;
}

// Channels that a window of 4 boxq rows holds, in whole boxes.
__host__ __device__ constexpr int bpf_window_channels(int kind, int boxq) {
    return (kind == MBX_GEOM_PARALLEL ? BPF_WIN_PARALLEL : BPF_WIN_FAN) / (4 * boxq) & ~(BPF_BOX - 1);
}

// Parallel beam: the window of one view for every pixel of a box of grid rows and columns (x, y and z, w of box), as first
// channel and channels (0: the view misses the box).  The channel is linear in the position, so the corners bound it; the
// slack covers the rounding of either side.
struct BpfBounds {
    int c_lo, nch;
    bool wide;  // larger than a window (or not a number)
};

// The same in one word (of a window that is not wide).
constexpr int BPF_NCH_BITS = 9;
static_assert(BPF_WIN_PARALLEL / 4 < (1 << BPF_NCH_BITS), "the widest window's channels do not fit their bits");
__host__ __device__ constexpr int bpf_pack_window(int c_lo, int nch) { return (c_lo + BPF_EDGE) << BPF_NCH_BITS | nch; }
__host__ __device__ constexpr int bpf_packed_first(int w) { return (w >> BPF_NCH_BITS) - BPF_EDGE; }
__host__ __device__ constexpr int bpf_packed_channels(int w) { return w & ((1 << BPF_NCH_BITS) - 1); }

// cs, sn: the view's angle; ok: it is a view of the sinogram.
__host__ __device__ __forceinline__ BpfBounds bpf_bounds(const mbx_geom &g, float cs, float sn, bool ok, int4 box,
                                                         int cap) {
    const float inv_dc = 1.0f / g.delta_det_channel;
    const float det_center_channel = 0.5f * (float)(g.num_det_channels - 1);
    float n_lo = 3.0e38f, n_hi = -3.0e38f, sum = 0.0f, size = 0.0f;
    for (int corner = 0; corner < 4; ++corner) {
        const float yt = g.delta_voxel * ((float)((corner & 1) ? box.y : box.x) - 0.5f * (float)(g.num_recon_rows - 1));
        const float xt = g.delta_voxel * ((float)((corner & 2) ? box.w : box.z) - 0.5f * (float)(g.num_recon_cols - 1));
        const float n = ((cs * xt - sn * yt) + g.det_channel_offset) * inv_dc + det_center_channel;
        n_lo = fminf(n_lo, n);
        n_hi = fmaxf(n_hi, n);
        sum += n;
        size = fmaxf(size, (fabsf(cs * xt) + fabsf(sn * yt) + fabsf(g.det_channel_offset)) * inv_dc + det_center_channel);
    }
    BpfBounds b;
    b.wide = !(fabsf(sum) < 4.0e6f) || !(n_hi - n_lo < 1.0e6f);
    if (b.wide) n_lo = n_hi = 0.0f;
    const float slack = fmaxf(0.02f, 8.0e-7f * size);  // six roundings on either side, of terms up to `size` channels
    b.c_lo = max((int)rintf(n_lo - slack) - 1, -BPF_EDGE);
    b.nch = max(min((int)rintf(n_hi + slack) + 1, g.num_det_channels + BPF_EDGE - 1) - b.c_lo + 1, 0);
    b.wide = b.wide || b.nch > cap;
    if (!ok) {  // an invalid view
        b.wide = false;
        b.nch = 0;
    }
    return b;
}

// Lanes of one pass over a view: those whose taps (channels ch .. ch + taps - 1) start within `cap` channels of the
// lowest remaining one.
struct BpfPass {
    int c_lo, nch;
    bool in;
};

__device__ __forceinline__ BpfPass bpf_pass(bool todo, int ch, int taps, int cap) {
    BpfPass q;
    q.c_lo = __reduce_min_sync(0xffffffffu, todo ? ch : INT_MAX);
    q.in = todo && ch + taps - q.c_lo <= cap;
    q.nch = __reduce_max_sync(0xffffffffu, q.in ? ch + taps - q.c_lo : 0);
    return q;
}

// What one pass over a view needs after its window has arrived.
struct BpfItem {
    bool in;       // this lane takes part
    bool tma;      // the window comes by TMA
    int off;       // window offset of the lane's first channel
    int row0;      // fan: detector row of the row buffer's row 0
    int nq;        // fan: row-buffer rows in fours
    float a[3];
    float A0, A1, c2, zv;
};

// 1 / sqrt(x) for x >= 1 (rsqrtf without its scaling of denormals).
__device__ __forceinline__ float bpf_rsqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The vertical fan of one pass: adds to acc the slices k_first .. of a tile (nsq fours) from the row sums in cache
// ([row][lane], row 0 = detector row it.row0).  Two slices at a time; the row of slice k, rint(A0 + k A1), comes from
// adding and removing 1.5 x 2^23, whose low mantissa bits are then the row (|row| < 2^22).  A voxel overlaps rows m_c
// - 1, m_c, m_c + 1 by min(max(half_w - |m_p - m|, 0), l_max); with d = m_p - m_c in [-1/2, 1/2] and A1 <= 2 the clips
// that cannot act are left out (WIDE: A1 > 2).  POWER: coefficients raised to coeff_power (1 otherwise).
template <bool POWER, bool WIDE>
__device__ __forceinline__ void bpf_vertical(bpf2 (&acc)[BPF_ST / 2], const BpfItem &it, const float *cache,
                                             float k_first, int nsq, float delta_voxel, int coeff_power) {
    const float magic = 12582912.0f;
    // byte address of a row: its bits x 128 plus this (modulo 2^32)
    const unsigned base = (unsigned)__cvta_generic_to_shared(cache) -
                          ((unsigned)__float_as_int(magic) + (unsigned)it.row0) * 128u;
    const float half_w = (it.A1 + 1.0f) * 0.5f;
    const float l_max = fminf(1.0f, it.A1);
    const float hw1 = half_w - 1.0f;
    const bpf2 A1p = bpf_pair(it.A1, it.A1), A0p = bpf_pair(it.A0, it.A0);
    const bpf2 mgp = bpf_pair(magic, magic), mgn = bpf_pair(-magic, -magic);
    const bpf2 neg = bpf_pair(-1.0f, -1.0f), one = bpf_pair(1.0f, 1.0f), two = bpf_pair(2.0f, 2.0f);
    const bpf2 hw1p = bpf_pair(hw1, hw1), c2p = bpf_pair(it.c2, it.c2);
    const bpf2 dvp = bpf_pair(delta_voxel, delta_voxel), zvp = bpf_pair(it.zv, it.zv);
    bpf2 k = bpf_pair(k_first, k_first + 1.0f);
#pragma unroll
    for (int q4 = 0; q4 < BPF_ST / 4; ++q4) {
        if (q4 >= nsq) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const bpf2 m_p = bpf_fma(k, A1p, A0p);
            const bpf2 mr = bpf_add(m_p, mgp);
            float ma, mb;
            bpf_unpair(mr, ma, mb);
            const unsigned ra = base + (unsigned)__float_as_int(ma) * 128u;
            const unsigned rb = base + (unsigned)__float_as_int(mb) * 128u;
            const bpf2 cm = bpf_pair(bpf_lds<-128>(ra), bpf_lds<-128>(rb));
            const bpf2 c0 = bpf_pair(bpf_lds<0>(ra), bpf_lds<0>(rb));
            const bpf2 cp = bpf_pair(bpf_lds<128>(ra), bpf_lds<128>(rb));
            const bpf2 d = bpf_fma(bpf_add(mr, mgn), neg, m_p);
            const bpf2 z = bpf_fma(k, dvp, zvp);
            const bpf2 q = bpf_fma(c2p, bpf_mul(z, z), one);
            float qa, qb, da, db, ma1, mb1, pa1, pb1;
            bpf_unpair(q, qa, qb);
            bpf2 sec = bpf_mul(q, bpf_pair(bpf_rsqrt(qa), bpf_rsqrt(qb)));  // 1 / cos(phi_k)
            bpf_unpair(d, da, db);
            bpf_unpair(bpf_fma(d, neg, hw1p), ma1, mb1);
            bpf_unpair(bpf_add(d, hw1p), pa1, pb1);
            ma1 = fmaxf(ma1, 0.0f);
            mb1 = fmaxf(mb1, 0.0f);
            pa1 = fmaxf(pa1, 0.0f);
            pb1 = fmaxf(pb1, 0.0f);
            if (WIDE) {
                ma1 = fminf(ma1, l_max);
                mb1 = fminf(mb1, l_max);
                pa1 = fminf(pa1, l_max);
                pb1 = fminf(pb1, l_max);
            }
            bpf2 l_m = bpf_pair(ma1, mb1), l_p = bpf_pair(pa1, pb1);
            bpf2 l_0 = bpf_pair(fminf(half_w - fabsf(da), l_max), fminf(half_w - fabsf(db), l_max));
            if (POWER && (!WIDE || coeff_power == 2)) {
                sec = bpf_mul(sec, sec);
                l_m = bpf_mul(l_m, l_m);
                l_0 = bpf_mul(l_0, l_0);
                l_p = bpf_mul(l_p, l_p);
            }
            const bpf2 x = bpf_fma(l_m, cm, bpf_fma(l_0, c0, bpf_mul(l_p, cp)));
            acc[2 * q4 + h] = bpf_fma(sec, x, acc[2 * q4 + h]);
            k = bpf_add(k, two);
        }
    }
}

__device__ __forceinline__ void bpf_vertical_fan(bpf2 (&acc)[BPF_ST / 2], const BpfItem &it, const float *cache, float k_first,
                                                 int nsq, float delta_voxel, int coeff_power) {
    if (it.A1 > 2.0f)
        bpf_vertical<true, true>(acc, it, cache, k_first, nsq, delta_voxel, coeff_power);
    else if (coeff_power == 2)
        bpf_vertical<true, false>(acc, it, cache, k_first, nsq, delta_voxel, 2);
    else
        bpf_vertical<false, false>(acc, it, cache, k_first, nsq, delta_voxel, 1);
}

// A lane's sums (list entry p, slices s0 .. s0 + ns - 1) into the output; `failed` ones leave as NaN, and `flag` says so.
__device__ __forceinline__ void bpf_write(const BpArgs &A, bpf2 (&acc)[BPF_ST / 2], bool failed, bool flag, long long p,
                                          bool active, int split, int s0, int ns, int *err) {
    if (flag) flag_error(err, MBX_ERRFLAG_CACHE);
    if (failed) {
        const float nan = __int_as_float(0x7fc00000);
#pragma unroll
        for (int s = 0; s < BPF_ST / 2; ++s) acc[s] = bpf_pair(nan, nan);
    }
    if (p >= A.num_pixels) return;
    long long row_of_out = p;
    if (A.out_by_index) {  // write into a flat recon at the pixel's index (skipped for invalid indices)
        if (!active) return;
        row_of_out = A.pix[p];
    }
    const float sc = (A.split_stride == 0) ? A.scale : 1.0f;
    if (A.out_slices > 0) {  // the one slice's value in every slice of the cylinder
        float *out = A.out + row_of_out * (long long)A.out_slices;
        float v, unused;
        bpf_unpair(acc[0], v, unused);
        v = active ? sc * v : 0.0f;
        for (int s = 0; s < A.out_slices; ++s) out[s] = v;
        return;
    }
    float *out = A.out + (long long)split * A.split_stride + row_of_out * (long long)A.g.num_recon_slices + s0;
#pragma unroll
    for (int s = 0; s < BPF_ST / 2; ++s) {
        float x, y;
        bpf_unpair(acc[s], x, y);
        if (2 * s < ns) out[2 * s] = active ? sc * x : 0.0f;
        if (2 * s + 1 < ns) out[2 * s + 1] = active ? sc * y : 0.0f;
    }
}

// One warp's unit of work: pixel group pg (32 list entries), slice tile st, view split `split`; smw: bpf_warp_floats
// of shared memory of its own.  No barrier beyond the warp.  The window of the next pass is copied while the current
// one is used: into a second buffer (parallel), or into the one buffer once the horizontal sums have been taken from
// it, during the vertical fan (fan geometries).
template <int KIND, bool TWO>
__device__ __forceinline__ void bp_fast_unit(const BpArgs &args, const CUtensorMap *tmap, int pg, int st, int split, float *smw, BpfPipe &pipe,
                                             int *err) {
    constexpr bool FAN = KIND != MBX_GEOM_PARALLEL;
    constexpr int WIN = FAN ? BPF_WIN_FAN : BPF_WIN_PARALLEL;
    constexpr unsigned ALL = 0xffffffffu;
    const BpArgs A = args;  // by value: a record in global memory is read once, not in the loops
    const mbx_geom &g = A.g;
    const BpfPlan &P = A.plan;
    const int32_t *__restrict__ pix = A.pix;
    const long long num_pixels = A.num_pixels;
    const int num_views_sel = A.num_views_sel, views_per_split = A.views_per_split, coeff_power = A.coeff_power;

    constexpr int TAPS = TWO ? 2 : 3;

    const int lane = threadIdx.x & 31;
    float *cache = smw + WIN + lane;                           // fan: row buffer [row][lane]
    const int pitch = 4 * P.boxq;                              // of a window's channels
    const int cap = bpf_window_channels(KIND, P.boxq);         // channels of a window

    const long long slot = (long long)pg * 32 + lane;
    const long long p = (A.order && slot < num_pixels) ? A.order[slot] : slot;  // list entry of this thread
    const int s0 = st * P.ts;
    const int num_slices = g.num_recon_slices;
    const int ns = min(P.ts, num_slices - s0);   // slices of this warp's tile
    if (ns <= 0) return;
    const int nsq = (ns + 3) >> 2;               // the same in fours: the slices past ns are computed, not written
    const float k_first = (float)s0, k_last = (float)(s0 + 4 * nsq - 1);
    const int v_end = min(num_views_sel, (split + 1) * views_per_split);
    const int npix_grid = g.num_recon_rows * g.num_recon_cols;

    bool active = p < num_pixels;
    float xt = 0.0f, yt = 0.0f;
    if (active) {
        const int idx = pix[p];
        active = idx >= 0 && idx < npix_grid;
        if (active)
            bpf_pixel<KIND>(g, idx, xt, yt);
        else if (st == 0 && split == 0)
            flag_error(err, MBX_ERRFLAG_PIXEL);
    }

    bpf2 acc[BPF_ST / 2];
#pragma unroll
    for (int s = 0; s < BPF_ST / 2; ++s) acc[s] = 0ull;

    float4 mine = make_float4(0.f, 0.f, 0.f, 0.f);  // constants of view vb + lane
    int vb = split * views_per_split;               // first view of the current block (32 views or all of them)
    int v = vb, v_stop = vb;                        // next view, and the end of the block
    int voff = 0;                                   // current view: offset, footprint, lanes not yet in a pass
    BpfFoot f = {};
    bool todo = false;
    // fan, current view: the rows of the warp's window
    int r0 = 0, nq = 0;
    bool fits = true;
    bool bad = false;  // a sum is not to be trusted: it leaves as NaN, and the error is flagged

    auto view_constants = [&](int t) {
        return make_float4(__shfl_sync(ALL, mine.x, t), __shfl_sync(ALL, mine.y, t), __shfl_sync(ALL, mine.z, t),
                           __shfl_sync(ALL, mine.w, t));
    };

    // what a lane's footprint f needs after its window (first channel c_lo) has arrived
    auto fill = [&](BpfItem &it, int c_lo) {
        it.off = (f.ch - c_lo) * pitch;
#pragma unroll
        for (int k = 0; k < 3; ++k) it.a[k] = f.a[k];
        it.A0 = f.A0;
        it.A1 = f.A1;
        it.c2 = f.c2;
        it.zv = f.zv;
    };

    // the next pass: its lanes, and the copy of its window into win started; false when the views are done
    auto next = [&](BpfItem &it, float *win, int b) -> bool {
        while (!__any_sync(ALL, todo)) {
            if (v >= v_stop) return false;
            const int t = (v - vb) & 31;
            if (t == 0 && v != vb) mine = bpf_view<KIND, true>(A, min(v + lane, v_stop - 1));
            const float4 vw = view_constants(t);
            ++v;
            voff = __float_as_int(vw.w);
            if (voff < 0) continue;
            bpf_footprint<KIND>(g, vw, xt, yt, coeff_power, TWO, f);
            todo = active && (f.a[0] != 0.0f || f.a[1] != 0.0f || f.a[2] != 0.0f);
            if constexpr (FAN) {
                // detector rows of this lane's slices (the affine map is monotone in the slice)
                const float m_a = rintf(fmaf(k_first, f.A1, f.A0)), m_b = rintf(fmaf(k_last, f.A1, f.A0));
                // rows near the detector (a NaN or a row far off it would not be an index): others add 0, or the NaN
                if (todo && !(fabsf(m_a) < 4.0e6f && fabsf(m_b) < 4.0e6f)) {
                    const float nan_or_0 = 0.0f * (m_a + m_b);
#pragma unroll
                    for (int s = 0; s < BPF_ST / 2; ++s) acc[s] = bpf_add(acc[s], bpf_pair(nan_or_0, nan_or_0));
                    todo = false;
                }
                const int m_lo = (int)fminf(m_a, m_b) - 1, m_hi = (int)fmaxf(m_a, m_b) + 1;
                r0 = __reduce_min_sync(ALL, todo ? m_lo : INT_MAX) & ~3;
                nq = (__reduce_max_sync(ALL, todo ? m_hi : INT_MIN) - r0 + 4) >> 2;
                fits = nq <= P.boxq;
                if (!fits) {  // each lane's own rows (of no use when no lane is to do)
                    r0 = m_lo & ~3;
                    nq = (m_hi - r0 + 4) >> 2;
                    if (todo && nq > P.boxq) {  // excluded by plan_bp_fast
                        bad = true;
                        todo = false;
                    }
                }
            }
        }
        const BpfPass w = bpf_pass(todo, f.ch, TAPS, fits ? cap : TAPS);
        bool window = fits;
        if (fits && __any_sync(ALL, todo && !w.in)) {  // several windows: unless they would be many
            const int bucket = todo ? min((f.ch - w.c_lo) / BPF_SPLIT, 31) : 31;
            window = __popc(__reduce_or_sync(ALL, todo ? 1u << bucket : 0u)) <= BPF_WINDOWS;
        }
        it.tma = window;
        it.in = w.in;
        fill(it, w.c_lo);
        if (window) {
            bpf_stage_tma(win, A, tmap, pipe, b, FAN ? r0 : s0, voff + w.c_lo + BPF_EDGE, w.nch);
        } else {  // as many lanes as there is room for, each with columns of its own
            const int rank = __popc(__ballot_sync(ALL, todo) & ((1u << lane) - 1u));
            it.in = todo && rank < WIN / (TAPS * pitch);
            it.off = rank * (TAPS * pitch);
            if (it.in)
                bpf_stage_private(win + it.off, A, voff, FAN ? r0 : s0, FAN ? nq : nsq, pitch, f.ch, TAPS);
        }
        it.row0 = r0;
        it.nq = nq;
        todo = todo && !it.in;
        return true;
    };

    // parallel: adds a pass's window in buffer b to the accumulators
    auto gather = [&](const BpfItem &it, int b) {
        const bpf2 a0 = bpf_pair(it.a[0], it.a[0]), a1 = bpf_pair(it.a[1], it.a[1]), a2 = bpf_pair(it.a[2], it.a[2]);
        const unsigned w0 = (unsigned)__cvta_generic_to_shared(smw + b * WIN + it.off);
        const unsigned w1 = w0 + 4u * (unsigned)pitch, w2 = w1 + 4u * (unsigned)pitch;
        bpf_for<0, BPF_ST / 4>([&](auto i) {
            constexpr int q = decltype(i)::value;
            if (q < nsq) {
                bpf2 x, y;
                if constexpr (!TWO) {
                    bpf_lds4<16 * q>(w2, x, y);
                    acc[2 * q] = bpf_fma(a2, x, acc[2 * q]);
                    acc[2 * q + 1] = bpf_fma(a2, y, acc[2 * q + 1]);
                }
                bpf_lds4<16 * q>(w1, x, y);
                acc[2 * q] = bpf_fma(a1, x, acc[2 * q]);
                acc[2 * q + 1] = bpf_fma(a1, y, acc[2 * q + 1]);
                bpf_lds4<16 * q>(w0, x, y);
                acc[2 * q] = bpf_fma(a0, x, acc[2 * q]);
                acc[2 * q + 1] = bpf_fma(a0, y, acc[2 * q + 1]);
            }
        });
    };
    // fan: the horizontal sums of a pass's window into the row buffer, and its vertical fan
    auto horizontal = [&](const BpfItem &it) {
        const bpf2 a0 = bpf_pair(it.a[0], it.a[0]), a1 = bpf_pair(it.a[1], it.a[1]), a2 = bpf_pair(it.a[2], it.a[2]);
        const unsigned w0 = (unsigned)__cvta_generic_to_shared(smw + it.off);
        const unsigned w1 = w0 + 4u * (unsigned)pitch, w2 = w1 + 4u * (unsigned)pitch;
        bpf_for<0, BPF_FAN_QUADS>([&](auto i) {
            constexpr int q = decltype(i)::value;
            if (q < it.nq) {
                bpf2 x0, x1, y0, y1, z0, z1;
                bpf_lds4<16 * q>(w0, x0, x1);
                bpf_lds4<16 * q>(w1, y0, y1);
                bpf_lds4<16 * q>(w2, z0, z1);
                float r[4];
                bpf_unpair(bpf_fma(a0, x0, bpf_fma(a1, y0, bpf_mul(a2, z0))), r[0], r[1]);
                bpf_unpair(bpf_fma(a0, x1, bpf_fma(a1, y1, bpf_mul(a2, z1))), r[2], r[3]);
#pragma unroll
                for (int j = 0; j < 4; ++j) cache[(4 * q + j) * 32] = r[j];
            }
        });
    };
    auto vertical = [&](const BpfItem &it) {
        bpf_vertical_fan(acc, it, cache, k_first, nsq, g.delta_voxel, coeff_power);
    };
    // parallel: the box of the warp's pixels; a box that fits one window in every view of 32 needs no search for the
    // window view by view (batched stage of 6 scans 2.16 -> 1.90 ms a step, a plain 652 x 57 x 437 subset
    // unchanged; for the fan geometries the second loop's code cost more than the searches, 6.25 -> 7.9 ms on the cone)
    int4 box = make_int4(0, 0, 0, 0);
    if constexpr (!FAN) {
        const int idx = active ? pix[p] : 0, row = idx / g.num_recon_cols, col = idx - row * g.num_recon_cols;
        box = make_int4(__reduce_min_sync(ALL, active ? row : INT_MAX), __reduce_max_sync(ALL, active ? row : INT_MIN),
                        __reduce_min_sync(ALL, active ? col : INT_MAX), __reduce_max_sync(ALL, active ? col : INT_MIN));
    }
    const bool none = !__any_sync(ALL, active);

    for (; vb < v_end && !none && !pipe.failed; vb = v_stop) {
        v = vb;
        v_stop = !FAN ? min(vb + 32, v_end) : v_end;
        mine = bpf_view<KIND, true>(A, min(vb + lane, v_stop - 1));
        BpfItem cur, nxt;
        cur.in = false;
        cur.tma = false;
        if constexpr (!FAN) {
            const BpfBounds mb = bpf_bounds(g, mine.x, mine.y, __float_as_int(mine.w) >= 0, box, cap);
            if (!__any_sync(ALL, mb.wide)) {
                const int pc = bpf_pack_window(mb.c_lo, mb.nch);
                const int nv = v_stop - vb;
                for (int t = 0; t <= nv; ++t) {
                    nxt.in = nxt.tma = false;
                    if (t < nv) {
                        const float4 vw = view_constants(t);
                        const int c = __shfl_sync(ALL, pc, t), nch = bpf_packed_channels(c), c_lo = bpf_packed_first(c);
                        nxt.tma = nch > 0;
                        if (nxt.tma)
                            bpf_stage_tma(smw + (t & 1) * WIN, A, tmap, pipe, t & 1, s0, __float_as_int(vw.w) + c_lo + BPF_EDGE, nch);
                        bpf_footprint<KIND>(g, vw, xt, yt, coeff_power, TWO, f);
                        const bool any = active && nxt.tma && (f.a[0] != 0.0f || f.a[1] != 0.0f || f.a[2] != 0.0f);
                        nxt.in = any && f.ch >= c_lo && f.ch + TAPS <= c_lo + nch;
                        if (any && !nxt.in) bad = true;  // excluded by the bounds' slack
                        fill(nxt, c_lo);
                    }
                    if (cur.tma) {
                        if (!bpf_pipe_wait(pipe, (t & 1) ^ 1, err)) {
                            if (nxt.tma) bpf_pipe_wait(pipe, t & 1, err);  // (no copy is left in flight)
                            break;
                        }
                        if (cur.in) gather(cur, (t & 1) ^ 1);
                        __syncwarp();  // this buffer takes the window after the next
                    }
                    cur = nxt;
                }
                continue;
            }
        }
        bool have = false;
        if constexpr (FAN) {
            for (;;) {
                if (have) {
                    if (cur.tma) {
                        if (!bpf_pipe_wait(pipe, 0, err)) break;
                    } else {
                        bpf_private_wait();
                    }
                    __syncwarp();
                    if (cur.in) horizontal(cur);
                    __syncwarp();  // the window may be overwritten
                }
                const bool more = next(nxt, smw, 0);
                if (have && cur.in) vertical(cur);
                if (!more) break;
                cur = nxt;
                have = true;
            }
        } else {
            for (int b = 0;; b ^= 1) {
                const bool more = next(nxt, smw + b * WIN, b);
                if (have) {
                    if (cur.tma) {
                        if (!bpf_pipe_wait(pipe, b ^ 1, err)) {
                            if (more && nxt.tma) bpf_pipe_wait(pipe, b, err);  // (no copy is left in flight)
                            break;
                        }
                    } else {
                        bpf_private_wait();
                    }
                    __syncwarp();
                    if (cur.in) gather(cur, b ^ 1);
                    __syncwarp();  // this buffer takes the window after the next
                }
                if (!more) break;
                cur = nxt;
                have = true;
            }
        }
    }
    __syncwarp();  // the warp's next unit may use the shared memory
    bpf_write(A, acc, bad || pipe.failed, bad, p, active, split, s0, ns, err);
}

// The same unit without a transposed copy to take windows of (calls whose scratch holds none, or that project ones): each
// lane reads its taps from the sinogram itself: for parallel beam those of 16 slices (8 with three taps) in flight together
// (4 scans of 180 x 20 x 200 in 4 subsets, a batch's stage: 249 us with 4 slices in flight and tiles of 20, 182 so with
// tiles of 12); for the fan geometries each detector row once, four rows in flight, into its column of the row buffer.
// Bound by the load/store pipe and the latency of the gathers.  Measured where windows copied
// by plain loads stood here before: cone 100 x 200 x 60 (subset of 8) 126 -> 45 us, 256 x 128 x 256 (subset of 8)
// 1035 -> 598 us, translation 49 x 128 x 128 (subset of 4) 85 -> 42 us, unit-weight Hessian of cone 256 x 128 x 256
// 4.66 -> 2.98 ms.
template <int KIND, bool TWO>
__device__ __forceinline__ void bp_direct_unit(const BpArgs &args, int pg, int st, int split, float *smw, int *err) {
    constexpr bool FAN = KIND != MBX_GEOM_PARALLEL;
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int TAPS = TWO ? 2 : 3;
    const BpArgs A = args;  // by value: a record in global memory is read once, not in the loops
    const mbx_geom &g = A.g;
    const int lane = threadIdx.x & 31;
    float *cache = smw + lane;  // fan: row buffer [row][lane]
    const long long slot = (long long)pg * 32 + lane;
    const long long p = (A.order && slot < A.num_pixels) ? A.order[slot] : slot;
    const int s0 = st * A.plan.ts, ns = min(A.plan.ts, g.num_recon_slices - s0);
    if (ns <= 0) return;
    const int nsq = (ns + 3) >> 2;
    const float k_first = (float)s0, k_last = (float)(s0 + 4 * nsq - 1);
    const int v_begin = split * A.views_per_split, v_end = min(A.num_views_sel, v_begin + A.views_per_split);
    const int num_rows = g.num_det_rows, num_channels = g.num_det_channels;

    bool active = p < A.num_pixels;
    float xt = 0.0f, yt = 0.0f;
    if (active) {
        const int idx = A.pix[p];
        active = idx >= 0 && idx < g.num_recon_rows * g.num_recon_cols;
        if (active)
            bpf_pixel<KIND>(g, idx, xt, yt);
        else if (st == 0 && split == 0)
            flag_error(err, MBX_ERRFLAG_PIXEL);
    }

    bpf2 acc[BPF_ST / 2];
#pragma unroll
    for (int s = 0; s < BPF_ST / 2; ++s) acc[s] = 0ull;
    bool bad = false;

    for (int vb = v_begin; vb < v_end; vb += 32) {
        const float4 mine = bpf_view<KIND, false>(A, min(vb + lane, v_end - 1));
        const int nv = min(32, v_end - vb);
        for (int t = 0; t < nv; ++t) {
            const float4 vw = make_float4(__shfl_sync(ALL, mine.x, t), __shfl_sync(ALL, mine.y, t),
                                          __shfl_sync(ALL, mine.z, t), __shfl_sync(ALL, mine.w, t));
            const int voff = __float_as_int(vw.w);
            if (voff < 0) continue;
            BpfFoot f;
            bpf_footprint<KIND>(g, vw, xt, yt, A.coeff_power, TWO, f);
            bool in = active && (f.a[0] != 0.0f || f.a[1] != 0.0f || f.a[2] != 0.0f);
            bool on[TAPS];  // taps on the detector
#pragma unroll
            for (int k = 0; k < TAPS; ++k) on[k] = (unsigned)(f.ch + k) < (unsigned)num_channels;
            if constexpr (FAN) {
                const float m_a = rintf(fmaf(k_first, f.A1, f.A0)), m_b = rintf(fmaf(k_last, f.A1, f.A0));
                if (in && !(fabsf(m_a) < 4.0e6f && fabsf(m_b) < 4.0e6f)) {  // as in bp_fast_unit
                    const float nan_or_0 = 0.0f * (m_a + m_b);
#pragma unroll
                    for (int s = 0; s < BPF_ST / 2; ++s) acc[s] = bpf_add(acc[s], bpf_pair(nan_or_0, nan_or_0));
                    in = false;
                }
                const int m_lo = (int)fminf(m_a, m_b) - 1, m_hi = (int)fmaxf(m_a, m_b) + 1;
                if (in && m_hi - m_lo >= 4 * BPF_FAN_QUADS) {  // excluded by plan_bp_fast
                    bad = true;
                    in = false;
                }
                if (in) {
                    const float ones = f.a[0] + (f.a[1] + f.a[2]);
                    int o = voff + m_lo * num_channels + f.ch;
                    float *dst = cache;
                    for (int m = m_lo; m <= m_hi; m += 4, o += 4 * num_channels, dst += 4 * 32) {
                        float x[4][TAPS];
#pragma unroll
                        for (int j = 0; j < 4; ++j)
#pragma unroll
                            for (int k = 0; k < TAPS; ++k)
                                x[j][k] = bpf_ldg(A.sino + (o + j * num_channels + k),
                                                  A.sino && on[k] && (unsigned)(m + j) < (unsigned)num_rows);
                        if (A.wts) {
#pragma unroll
                            for (int j = 0; j < 4; ++j)
#pragma unroll
                                for (int k = 0; k < TAPS; ++k)
                                    x[j][k] *= bpf_ldg(A.wts + (o + j * num_channels + k),
                                                       on[k] && (unsigned)(m + j) < (unsigned)num_rows);
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            dst[j * 32] = A.sino ? fmaf(f.a[0], x[j][0], fmaf(f.a[1], x[j][1], f.a[2] * x[j][TAPS - 1]))
                                                 : ((unsigned)(m + j) < (unsigned)num_rows ? ones : 0.0f);
                    }
                    BpfItem it;
                    it.row0 = m_lo;
                    it.A0 = f.A0;
                    it.A1 = f.A1;
                    it.c2 = f.c2;
                    it.zv = f.zv;
                    bpf_vertical_fan(acc, it, cache, k_first, nsq, g.delta_voxel, A.coeff_power);
                }
            } else if (!A.sino) {  // (the unit-weight Hessian, usually of one slice)
                if (in) {
#pragma unroll
                    for (int s = 0; s < BPF_ST / 2; ++s)
                        if (2 * s < ns)
                            acc[s] = bpf_add(bpf_pair(f.a[0], f.a[0]),
                                             bpf_add(bpf_pair(f.a[1], f.a[1]), bpf_add(bpf_pair(f.a[2], f.a[2]), acc[s])));
                }
            } else if (in) {
                int o = voff + s0 * num_channels + f.ch;
                const bpf2 a0 = bpf_pair(f.a[0], f.a[0]), a1 = bpf_pair(f.a[1], f.a[1]), a2 = bpf_pair(f.a[2], f.a[2]);
                constexpr int N = TWO ? 16 : 8;  // slices whose taps are in flight together
#pragma unroll
                for (int c = 0; c < BPF_ST / N; ++c, o += N * num_channels) {
                    if (c * N >= ns) break;
                    float x[N][TAPS];
#pragma unroll
                    for (int j = 0; j < N; ++j)
#pragma unroll
                        for (int k = 0; k < TAPS; ++k)
                            x[j][k] = bpf_ldg(A.sino + (o + j * num_channels + k), on[k] && c * N + j < ns);
                    if (A.wts) {
#pragma unroll
                        for (int j = 0; j < N; ++j)
#pragma unroll
                            for (int k = 0; k < TAPS; ++k)
                                x[j][k] *= bpf_ldg(A.wts + (o + j * num_channels + k), on[k] && c * N + j < ns);
                    }
#pragma unroll
                    for (int h = 0; h < N / 2; ++h) {
                        bpf2 a = acc[c * N / 2 + h];
                        if constexpr (!TWO) a = bpf_fma(a2, bpf_pair(x[2 * h][TAPS - 1], x[2 * h + 1][TAPS - 1]), a);
                        a = bpf_fma(a1, bpf_pair(x[2 * h][1], x[2 * h + 1][1]), a);
                        acc[c * N / 2 + h] = bpf_fma(a0, bpf_pair(x[2 * h][0], x[2 * h + 1][0]), a);
                    }
                }
            }
            __syncwarp();
        }
    }
    bpf_write(A, acc, bad, bad, p, active, split, s0, ns, err);
}

// Shared memory of one warp, in floats: window(s) and barriers (of a call with a transposed copy), row buffer; a multiple
// of the 128 bytes a TMA destination is aligned to.
__host__ __device__ constexpr int bpf_warp_floats(int kind, bool tr) {
    const int rows = kind == MBX_GEOM_PARALLEL ? 0 : 4 * BPF_FAN_QUADS * 32;
    return rows + (tr ? (kind == MBX_GEOM_PARALLEL ? 2 * BPF_WIN_PARALLEL : BPF_WIN_FAN) + 32 : 0);
}

// CTAs of two warps: a warp whose pixels span a wide window takes longer, and holds back only one other.  Resident
// CTAs per SM the kernels are compiled for (112 and 128 registers).
constexpr int BPF_LAUNCH_WARPS = 2;
__host__ __device__ constexpr int bpf_min_blocks(int kind) { return kind == MBX_GEOM_PARALLEL ? 9 : 8; }
// Without windows: CTAs of four warps on neighbouring pixels, which share lines in L1 (128 registers, 4 resident).  Cone
// 200 x 100 x 200 subset of 4, 256 x 128 x 256 subset of 8: 470 and 604 us, in CTAs of two 491 and 598, of eight 508 and 705.
constexpr int BPF_DIRECT_WARPS = 4;
__host__ __device__ constexpr int bpf_launch_warps(bool tr) { return tr ? BPF_LAUNCH_WARPS : BPF_DIRECT_WARPS; }

// Unit u of a call: the 8 units of plan tile (bx, by) are its npg pixel groups x nsl slice tiles.
template <int KIND, bool TR>
__device__ __forceinline__ void bp_fast_run(const BpArgs &A, const CUtensorMap *tmap, int tile, int w, int split, float *smw, BpfPipe &pipe,
                                            int *err) {
    const BpfPlan &P = A.plan;
    const int by = tile / P.gx, bx = tile - by * P.gx;
    const int pg = w / P.nsl;
    const int group = bx * P.npg + pg, st = by * P.nsl + (w - pg * P.nsl);
    auto unit = [&](auto two) {
        if constexpr (TR)
            bp_fast_unit<KIND, decltype(two)::value>(A, tmap, group, st, split, smw, pipe, err);
        else
            bp_direct_unit<KIND, decltype(two)::value>(A, group, st, split, smw, err);
    };
    if constexpr (KIND == MBX_GEOM_PARALLEL) {
        // voxels no wider than a channel: two taps per footprint
        if (A.g.delta_voxel * (1.0f / A.g.delta_det_channel) <= 1.0f) {
            unit(std::true_type{});
            return;
        }
    }
    unit(std::false_type{});
}

template <int KIND, bool TR>
__global__ void __launch_bounds__(32 * bpf_launch_warps(TR), TR ? bpf_min_blocks(KIND) : 4)
bp_fast_kernel(const BpArgs args, const __grid_constant__ CUtensorMap map, int *err) {
    extern __shared__ __align__(128) float smf[];
    const int warp = threadIdx.x >> 5;
    const int unit = blockIdx.x * bpf_launch_warps(TR) + warp;
    float *smw = smf + warp * bpf_warp_floats(KIND, TR);
    BpfPipe pipe = {0, 0, false};
    if (TR) pipe = bpf_pipe_init(smw + bpf_warp_floats(KIND, TR) - 32);
    if (args.views && unit == 0) {  // bad views of this split, which every unit skips
        const int v_end = min(args.num_views_sel, ((int)blockIdx.y + 1) * args.views_per_split);
        for (int v = blockIdx.y * args.views_per_split + (threadIdx.x & 31); v < v_end; v += 32)
            if (args.views[v] < 0 || args.views[v] >= args.g.num_views) flag_error(err, MBX_ERRFLAG_VIEW);
    }
    bp_fast_run<KIND, TR>(args, TR ? &map : nullptr, unit >> 3, unit & 7, blockIdx.y, smw, pipe, err);
}

inline size_t bpf_smem_bytes(int kind, int warps, bool tr) { return 4 * (size_t)warps * bpf_warp_floats(kind, tr); }

// Transposed copy of a call's views (of every view of the geometry when the call selects more, that is repeats
// some): per view, channel outermost with BPF_EDGE channels of zeros on either side, rows padded to a multiple of 4
// with zeros.
inline int bpf_padded_rows(const mbx_geom &g) { return (g.num_det_rows + 3) & ~3; }
inline int bpf_transposed_views(const mbx_geom &g, int num_views_sel) {
    return num_views_sel < g.num_views ? num_views_sel : g.num_views;
}
inline size_t bpf_transposed_bytes(const mbx_geom &g, int num_views_sel) {
    return align256((size_t)bpf_transposed_views(g, num_views_sel) * (g.num_det_channels + 2 * BPF_EDGE) *
                    bpf_padded_rows(g) * 4);
}

// The tensor map of a transposed copy at `copy`: boxes of BPF_BOX channels x 4 boxq rows.  False when it cannot be
// made (a copy that is not 16-byte aligned; defined in back_project.cu).
bool bpf_window_map(CUtensorMap &map, const float *copy, const mbx_geom &g, int num_views_sel, int boxq);

// Channels c0 .. c0 + 31 (counted with the edge channels) of one view of the transposed copy, by a block of 256 threads:
// weights x values of src (view offset soff, num_rows x num_channels), rows r_begin (a multiple of 32) .. r_end - 1, to
// dst (view offset doff).  A plain call gives each 32 rows a block of their own (views of 128 rows: a quarter of the
// serial steps).
__device__ __forceinline__ void bpf_transpose_block(const float *__restrict__ src, const float *__restrict__ wts,
                                                    float *__restrict__ dst, long long soff, long long doff, int c0,
                                                    int r_begin, int r_end, int num_rows, int num_channels, int rp) {
    __shared__ float tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    for (int r0 = r_begin; r0 < r_end; r0 += 32) {
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            const int r = r0 + ty + j, n = c0 + tx - BPF_EDGE;
            float v = 0.0f;
            if (r < num_rows && n >= 0 && n < num_channels) {
                const long long o = soff + (long long)r * num_channels + n;
                v = __ldg(src + o);
                if (wts) v *= __ldg(wts + o);
            }
            tile[ty + j][tx] = v;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            const int c = c0 + ty + j, r = r0 + tx;
            if (c < num_channels + 2 * BPF_EDGE && r < rp) dst[doff + (long long)c * rp + r] = tile[tx][ty + j];
        }
    }
}

// Slices per tile: the fewest tiles of <= most slices, the slices spread evenly over them, in fours.
inline int bpf_tile_height(int S, int most) {
    const int tiles = ceil_div(S, most);
    const int ts = ((ceil_div(S, tiles) + 3) / 4) * 4;
    return ts < most ? ts : most;
}

// The partial sums of the splits take at most BPF_PARTIAL_BYTES (which fits the scratch of the entry point that
// allocates nothing), or twice the sinogram unless `small`.
constexpr size_t BPF_PARTIAL_BYTES = MBX_NOALLOC_SCRATCH_BYTES / 4 * 3;

// Fewest views per split: a warp's views follow one another, so a small call takes as long as one warp's views
// (24 x 20 x 64 cone, subset of 4: 30 us with 8, 20 with 4, 14 with 2).
constexpr int BPF_SPLIT_VIEWS = 2;

// most_slices > 0: tiles of at most that many slices, whatever the call's size (a batch's lists).
inline BpfPlan plan_bp_fast(const mbx_geom &g, long long num_pixels, int num_views_sel, int small = 0,
                            int most_slices = 0) {
    BpfPlan pl;
    pl.inline_fp = 1;
    pl.chunk = 0;
    pl.vc = 32;
    // 32-bit element offsets address the sinogram
    pl.ok = (g.kind == MBX_GEOM_PARALLEL || g.kind == MBX_GEOM_CONE ||
             (g.kind == MBX_GEOM_TRANSLATION && g.max_magnification > 0.0f)) &&
            (g.psf_radius == 1) && g.num_det_channels >= 3 &&
            (long long)g.num_views * g.num_det_rows * g.num_det_channels < (1LL << 31);
    const int S = g.num_recon_slices;
    int most = BPF_ST;
    double slope = 1.0;
    if (g.kind != MBX_GEOM_PARALLEL) {
        // the row buffer must hold the rows of a slice tile: ts * max |dm/dk| + 4
        double max_mag = g.max_magnification;  // translation: the host's bound
        if (g.kind == MBX_GEOM_CONE) {
            const double half_r = 0.5 * (g.num_recon_rows - 1), half_c = 0.5 * (g.num_recon_cols - 1);
            const double rho = g.delta_voxel * std::sqrt(half_r * half_r + half_c * half_c);
            const double inv = 1.0 / g.magnification - (std::isinf(g.source_detector_dist) ? 0.0 : rho / g.source_detector_dist);
            max_mag = inv > 1e-6 ? 1.0 / inv : 1e6;
        }
        slope = max_mag * g.delta_voxel / g.delta_det_row;
        while (most > 4 && most * slope + 4 > BPF_CACHE_ROWS) most -= 4;
        if (bpf_tile_height(S, most) * slope + 4 > BPF_CACHE_ROWS) pl.ok = false;
    }
    const long long slots = (long long)bpf_min_blocks(g.kind) * BPF_LAUNCH_WARPS * num_sms() / BPF_WARPS;
    // translation: a pixel's magnification follows its row, so the footprints of a warp spread over more channels and
    // rows than a low tile's windows have (all pixels of 49 x 128 x 128: 121 us with 32 slices, 130 with 16, 105 with 12,
    // 132 with 8; subset of 4 of 49 x 85 x 96: 60, 46 and 41 us)
    if (g.kind == MBX_GEOM_TRANSLATION) most = std::min(most, 12);
    if (most_slices > 0)
        most = std::min(most, most_slices);
    // cone: tiles of half the height for calls whose units could not fill the chip (101 x 18 x 51, subset of 4: 20 -> 16)
    else if (g.kind == MBX_GEOM_CONE && (num_pixels + 31) / 32 * ceil_div(S, most) *
                                           std::max(1, num_views_sel / BPF_SPLIT_VIEWS) < BPF_WARPS * slots)
        most = std::min(most, BPF_ST / 2);
    pl.ts = bpf_tile_height(S, most);
    pl.tiles = ceil_div(S, pl.ts);
    // rows of a window: the tile's (parallel); its rows at the steepest slope, their rounding and some spread (fan)
    pl.boxq = g.kind == MBX_GEOM_PARALLEL ? ((pl.ts + 3) / 4) | 1
                                          : std::min(BPF_FAN_QUADS, (int)std::ceil((pl.ts * slope + 12) / 4) | 1);
    // a CTA's warps on neighbouring pixels of one slice tile (their windows overlap in L1), on several tiles only when
    // the list is shorter than a CTA
    pl.nsl = 1;
    while (pl.nsl < 8 && pl.tiles % (2 * pl.nsl) == 0 && num_pixels <= 32 * (8 / (2 * pl.nsl))) pl.nsl *= 2;
    pl.npg = 8 / pl.nsl;
    pl.lg_pcta = 5;
    while ((1 << pl.lg_pcta) < 32 * pl.npg) ++pl.lg_pcta;
    const int pcta = 32 * pl.npg;
    pl.gx = ceil_div(num_pixels > 0 ? num_pixels : 1, pcta);
    pl.gy = ceil_div(pl.tiles, pl.nsl);
    // views split over CTAs when there are few: the fewest splits (partial sums cost memory traffic) whose last wave
    // is full enough, as the time of a call is about waves / splits
    const long long base = (long long)pl.gx * pl.gy;
    long long splits = 1;
    if (base < 2 * slots && num_views_sel >= 16) {
        long long maxs = num_views_sel / BPF_SPLIT_VIEWS;
        if (maxs > 64) maxs = 64;
        size_t most_bytes = BPF_PARTIAL_BYTES;
        if (!small) most_bytes = std::max(most_bytes, (size_t)g.num_views * g.num_det_rows * g.num_det_channels * 8);
        const long long fit = (long long)most_bytes / (4 * (num_pixels > 0 ? num_pixels : 1) * S);
        if (maxs > fit) maxs = fit;
        double best = 1e300;
        for (long long s = 1; s <= maxs; ++s) {
            const double cost = (double)((base * s + slots - 1) / slots) / s * (1.0 + 0.01 * s);
            if (cost < best * 0.98) {
                best = cost;
                splits = s;
            }
        }
    }
    pl.views_per_split = ceil_div(num_views_sel, splits);
    pl.splits = ceil_div(num_views_sel, pl.views_per_split);
    pl.smem = bpf_smem_bytes(g.kind, BPF_LAUNCH_WARPS, true);
    pl.workspace = pl.splits > 1 ? align256((size_t)pl.splits * num_pixels * S * 4) : 0;
    return pl;
}

// Whether a call's back projection reads windows of a transposed copy of its views, given the plan it would have.  The copy
// and a warp's windows are paid once per view and serve 32 pixels x the slices of a tile, so small calls, lists that spread
// a warp over more channels than a window has, and calls whose warps make less than about a wave (which then take as long as
// the warp with the most windows) read their taps from the sinogram itself: the fan geometries by bp_direct_unit (the same
// sums in the same order), parallel beam by bp_gather.cuh.  A batch fills the chip with its scans, and always takes windows.
// Lines measured on 300 calls; us without / with windows:
//  * parallel, slices: 13, every pixel 70 / 107; 9, subset of 4 109 / 168; 25 70 / 89;
//    density: 35 slices, subset of 8 29 / 38; 60 slices, subset of 8 97 / 102; then by voxels x views:
//    dense lists 59 M 95 / 103, 71 M 88 / 78, 130 M 129 / 128; subsets of 4 10 M 26 / 37, 83 M 101 / 109,
//    131 M 149 / 192, 174 M 238 / 212, 322 M 405 / 370; under 0.7 waves 268 M 259 / 378, 125 M 105 / 130.
//  * cone: under a wave 464 M 1183 / 2050, 116 M 339 / 594, 742 M 1833 / 2145, but whole grids, whose warps seldom lie
//    across two rows' ends, 377 M 958 / 765, 452 M 1428 / 1203, 178 M 461 / 488; up to two waves 271 M 697 / 626,
//    135 M 524 / 328, 228 M 584 / 661; from three 418 M 1164 / 866, 544 M 1610 / 1061; by voxels x views 45 M 153 / 144,
//    66 M 208 / 240, 101 M 322 / 333, 111 M 298 / 337, 117 M 376 / 300; subset of 32 144 M 472 / 671, of 16
//    304 M 1021 / 893.
//  * translation, whose magnification differs from grid row to grid row: every pixel 23 M 64 / 65, 29 M 91 / 88,
//    39 M 121 / 108, 153 M 408 / 370; half of them 132 M 305 / 574.
constexpr int BPF_FEW_SLICES = 27;
inline bool bp_windows(const mbx_geom &g, const BpfPlan &pl, long long num_pixels, int num_views_sel) {
    const double grid = (double)g.num_recon_rows * g.num_recon_cols, dense = (double)num_pixels / grid;
    const double work = (double)num_pixels * g.num_recon_slices * num_views_sel * 1e-6;
    const double waves = (double)pl.gx * pl.gy * pl.splits * BPF_WARPS /
                         ((double)bpf_min_blocks(g.kind) * BPF_LAUNCH_WARPS * num_sms());
    switch (g.kind) {
        case MBX_GEOM_PARALLEL:
            return g.num_recon_slices >= BPF_FEW_SLICES && dense >= 1.0 / 7 && work >= (dense >= 0.375 ? 48 : 160) &&
                   waves >= 0.7;
        case MBX_GEOM_CONE: return work >= 112 && dense >= 1.0 / 24 && (waves >= 1.05 || dense > 0.9);
        default: return work >= 28 && dense > 0.5;
    }
}

}  // namespace mbx
