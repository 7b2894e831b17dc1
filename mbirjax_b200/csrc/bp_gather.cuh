// Parallel-beam back projection that gathers its taps from global memory (psf_radius == 1): the better kernel where a
// window of the view (bp_fast.cuh) costs more than it saves, for lists and recons that bp_windows() leaves out.
//
// CTA = 256 threads = 8 warps; lanes run along 32 pixels, warps along slice tiles of at most BPG_ST slices, accumulators
// in registers across all views.  A thread reads three taps per slice at constant offsets from one 32-bit element offset.
// Each thread computes its own footprints (staged once per CTA in shared memory where several slice tiles share a pixel,
// with the rows of a later view prefetched: 65 us where this takes 52, 70 x 26 x 470, subset of 8).
// Bound by instruction issue (21 per slice and view) and the latency of the gathers at 24 warps per SM.
#pragma once

#include "bp_fast.cuh"

namespace mbx {

constexpr int BPG_ST = 16;        // most slices per thread
constexpr int BPG_VIEWS = 1024;   // views per table refill

struct BpgPlan {
    int nsl, lg_pcta;  // slice tiles per CTA (warps per pixel group); log2 of the pixels per CTA
    int ts;            // slices per tile
    int gx, gy, splits, views_per_split;
    size_t workspace;
};

// For geometries that plan_bp_fast admits.  Views are split over CTAs when there are fewer than two per SM; the partial
// sums of the splits then hold at most 592 CTAs' accumulators (9.7 MB).  splits > 0: that many instead (of a call that
// stands in for one with windows: the same sums in the same order).
inline BpgPlan plan_bp_gather(const mbx_geom &g, long long num_pixels, int num_views_sel, int splits_of = 0) {
    BpgPlan pl;
    const int S = g.num_recon_slices;
    // the fewest tiles, rounded up to a power of two (at most 8) or a multiple of 8, then the slices spread evenly
    const int t0 = ceil_div(S, BPG_ST);
    int T = 1;
    if (t0 <= 8) {
        while (T < t0) T <<= 1;
    } else {
        T = ceil_div(t0, 8) * 8;
    }
    pl.ts = ceil_div(S, T);
    const int tiles = ceil_div(S, pl.ts);
    pl.nsl = 1;
    while (pl.nsl < tiles && pl.nsl < 8) pl.nsl <<= 1;
    const int pcta = 256 / pl.nsl;
    pl.lg_pcta = 5;
    while ((1 << pl.lg_pcta) < pcta) ++pl.lg_pcta;
    pl.gx = ceil_div(num_pixels > 0 ? num_pixels : 1, pcta);
    pl.gy = ceil_div(tiles, pl.nsl);
    const long long base = (long long)pl.gx * pl.gy, want = 2LL * num_sms();
    long long splits = 1;
    if (splits_of > 0)
        splits = splits_of;
    else if (base < want && num_views_sel >= 16)
        splits = std::max(1LL, std::min({(want + base - 1) / base, (long long)num_views_sel / 8, 64LL}));
    pl.views_per_split = ceil_div(num_views_sel, splits);
    pl.splits = ceil_div(num_views_sel, pl.views_per_split);
    pl.workspace = pl.splits > 1 ? align256((size_t)pl.splits * num_pixels * S * 4) : 0;
    return pl;
}

struct BpgArgs {
    mbx_geom g;
    const float *sino, *wts;
    const int32_t *pix, *views;
    long long num_pixels;
    int num_views_sel, coeff_power;
    float scale;
    float *out;
    long long split_stride;  // 0: final output; else the stride of the splits' partial sums
    BpgPlan plan;
};

// Footprint of one (pixel, view): {first channel (int bits; -1: no tap), the coefficients of channels first..first + 2}.
__device__ __forceinline__ float4 bpg_footprint(const mbx_geom &g, float cs, float sn, float xt, float yt,
                                                int coeff_power) {
    const float inv_dc = 1.0f / g.delta_det_channel;
    const float x = cs * xt - sn * yt;
    const float n_p = (x + g.det_channel_offset) * inv_dc + 0.5f * (float)(g.num_det_channels - 1);
    const float cos_alpha = fmaxf(fabsf(cs), fabsf(sn));
    const float w = (g.delta_voxel * inv_dc) * cos_alpha;
    const float scale = g.delta_voxel / cos_alpha;
    const int nc = (int)rintf(n_p);
    const float half_w = (w + 1.0f) * 0.5f, l_max = fminf(1.0f, w), d = n_p - (float)nc;
    float a[3];
#pragma unroll
    for (int k = -1; k <= 1; ++k) {
        float v = scale * fminf(fmaxf(half_w - fabsf(d - (float)k), 0.0f), l_max);
        if (nc + k < 0 || nc + k >= g.num_det_channels) v = 0.0f;
        a[k + 1] = coeff_power == 2 ? v * v : v;
    }
    // three channels on the detector; edge taps move onto them with zero coefficients
    const int first = min(max(nc - 1, 0), g.num_det_channels - 3), sh = first - (nc - 1);
    float c[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int j = k + sh;
        c[k] = j == 0 ? a[0] : (j == 1 ? a[1] : (j == 2 ? a[2] : 0.0f));
    }
    const bool any = c[0] != 0.0f || c[1] != 0.0f || c[2] != 0.0f;
    return make_float4(__int_as_float(any ? first : -1), c[0], c[1], c[2]);
}

// One view into the first TS accumulators (TS = the tile's slice count, so no slot is predicated off).
template <int TS>
__device__ __forceinline__ void bpg_rows(float (&acc)[BPG_ST], const float *__restrict__ sino, int o, int pitch,
                                         const float4 &fa) {
#pragma unroll
    for (int s = 0; s < TS; ++s) {
        const float *q = sino + o;
        acc[s] = fmaf(fa.y, __ldg(q), fmaf(fa.z, __ldg(q + 1), fmaf(fa.w, __ldg(q + 2), acc[s])));
        o += pitch;
    }
}

__global__ void __launch_bounds__(256, 3) bp_gather_kernel(const BpgArgs A, int *err) {
    const mbx_geom &g = A.g;
    const BpgPlan &P = A.plan;
    __shared__ float s_cs[BPG_VIEWS], s_sn[BPG_VIEWS];
    __shared__ int s_voff[BPG_VIEWS];  // element offset of each view (-1: invalid view)

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, pcta = 1 << P.lg_pcta;
    const int pg = warp / P.nsl, slot = pg * 32 + lane;
    const long long p = (long long)blockIdx.x * pcta + slot;
    const int s0 = (blockIdx.y * P.nsl + (warp - pg * P.nsl)) * P.ts;
    const int pitch = g.num_det_channels, ns = min(P.ts, g.num_recon_slices - s0), s0c = s0 * pitch;
    const int split = blockIdx.z;
    const int v_begin = split * P.views_per_split, v_end = min(A.num_views_sel, v_begin + P.views_per_split);
    const int npix_grid = g.num_recon_rows * g.num_recon_cols, view_stride = g.num_det_rows * pitch;
    const float *__restrict__ sino = A.sino;
    const float *__restrict__ wts = A.wts;

    bool active = false;
    float xt = 0.0f, yt = 0.0f;
    if (p < A.num_pixels) {
        const int idx = A.pix[p];
        active = idx >= 0 && idx < npix_grid;
        if (active) pixel_tilde(g, idx, xt, yt);
        else if (blockIdx.y == 0 && split == 0 && warp == pg * P.nsl) flag_error(err, MBX_ERRFLAG_PIXEL);
    }
    active = active && ns > 0;

    float acc[BPG_ST];
#pragma unroll
    for (int s = 0; s < BPG_ST; ++s) acc[s] = 0.0f;
    auto gather = [&](const float4 &fa, int voff) {
        int o = voff + s0c + __float_as_int(fa.x);
        if (wts) {
#pragma unroll
            for (int s = 0; s < BPG_ST; ++s) {
                if (s < ns) {
                    const float *q = sino + o, *qw = wts + o;
                    acc[s] = fmaf(fa.y, __ldg(q) * __ldg(qw),
                                  fmaf(fa.z, __ldg(q + 1) * __ldg(qw + 1), fmaf(fa.w, __ldg(q + 2) * __ldg(qw + 2), acc[s])));
                }
                o += pitch;
            }
            return;
        }
        switch (ns) {  // the same for every lane of the warp
            case 1: bpg_rows<1>(acc, sino, o, pitch, fa); break;
            case 2: bpg_rows<2>(acc, sino, o, pitch, fa); break;
            case 3: bpg_rows<3>(acc, sino, o, pitch, fa); break;
            case 4: bpg_rows<4>(acc, sino, o, pitch, fa); break;
            case 5: bpg_rows<5>(acc, sino, o, pitch, fa); break;
            case 6: bpg_rows<6>(acc, sino, o, pitch, fa); break;
            case 7: bpg_rows<7>(acc, sino, o, pitch, fa); break;
            case 8: bpg_rows<8>(acc, sino, o, pitch, fa); break;
            case 9: bpg_rows<9>(acc, sino, o, pitch, fa); break;
            case 10: bpg_rows<10>(acc, sino, o, pitch, fa); break;
            case 11: bpg_rows<11>(acc, sino, o, pitch, fa); break;
            case 12: bpg_rows<12>(acc, sino, o, pitch, fa); break;
            case 13: bpg_rows<13>(acc, sino, o, pitch, fa); break;
            case 14: bpg_rows<14>(acc, sino, o, pitch, fa); break;
            case 15: bpg_rows<15>(acc, sino, o, pitch, fa); break;
            default: bpg_rows<BPG_ST>(acc, sino, o, pitch, fa); break;
        }
    };

    for (int vb = v_begin; vb < v_end; vb += BPG_VIEWS) {
        const int nv = min(BPG_VIEWS, v_end - vb);
        __syncthreads();
        for (int t = tid; t < nv; t += 256) {
            const int vi = A.views ? A.views[vb + t] : vb + t;
            const bool ok = vi >= 0 && vi < g.num_views;
            if (!ok && blockIdx.x == 0 && blockIdx.y == 0) flag_error(err, MBX_ERRFLAG_VIEW);
            s_voff[t] = ok ? vi * view_stride : -1;
            const float ang = ok ? g.angles[vi] : 0.0f;
            s_cs[t] = cosf(ang);
            s_sn[t] = sinf(ang);
        }
        __syncthreads();
        if (!active) continue;
        for (int t = 0; t < nv; ++t) {
            const int voff = s_voff[t];
            if (voff < 0) continue;
            const float4 fa = bpg_footprint(g, s_cs[t], s_sn[t], xt, yt, A.coeff_power);
            if (__float_as_int(fa.x) >= 0) gather(fa, voff);
        }
    }
    if (p >= A.num_pixels || ns <= 0) return;
    const float sc = A.split_stride == 0 ? A.scale : 1.0f;
    float *out = A.out + (long long)split * A.split_stride + p * (long long)g.num_recon_slices + s0;
#pragma unroll
    for (int s = 0; s < BPG_ST; ++s)
        if (s < ns) out[s] = active ? sc * acc[s] : 0.0f;
}

}  // namespace mbx
