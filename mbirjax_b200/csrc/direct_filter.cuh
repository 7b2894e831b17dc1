// Ramp filtering of detector rows for FBP / FDK (sm_100a): the device function shared by the plain entry point
// (direct_filter.cu) and the batched VCD set-up (vcd_batched.cu).  See direct_filter.cu for the arithmetic.
#pragma once

#include <cmath>

#include "mbx_common.cuh"

namespace mbx {

constexpr int FILT_THREADS = 256;

// Scales of the ramp filter for a geometry: the filter times 1/delta_voxel^2 (FBP, parallel_beam.py:325-327) or
// delta_det_row / (delta_voxel^3 magnification) after the FDK pre-weight (cone_beam.py:825-827), and pi / views.
inline void direct_filter_scales(const mbx_geom &g, double &filter_scale, double &out_scale, int &fdk) {
    const double pi = 3.14159265358979323846;
    out_scale = pi / g.num_views;
    if (g.kind == MBX_GEOM_PARALLEL) {
        filter_scale = 1.0 / ((double)g.delta_voxel * g.delta_voxel);
        fdk = 0;
    } else {
        filter_scale = (double)g.delta_det_row /
                       ((double)g.delta_voxel * g.delta_voxel * g.delta_voxel * g.magnification);
        fdk = 1;
    }
}

// Whether rows of C channels are filtered: the longest rows the library admits (a tile of eight rows, for FDK twice, and
// its taps in 200 KB).
inline bool filter_admits(int C, int fdk) {
    return (fdk ? 2 : 1) * (size_t)C * 32 + (2 * (size_t)C - 1) * sizeof(double) <= 200 * 1024;
}

// How a block of 8 warps is spread over a tile: a warp holds 16 rows x 64 outputs of one parity (128 channels with its
// partner of the other parity).  Rows of up to 128 channels take one such pair and 4 groups of rows, up to 256 channels
// two pairs and 2 groups, longer rows four pairs at a time.
struct FiltShape {
    int outs;     // outputs of one parity (ceil(C / 2))
    int tiles;    // 64-output tiles of one parity
    int groups;   // groups of 16 rows per block
    int rows;     // rows per block
    int kc;       // samples of one parity staged at a time
    int kp;       // outs rounded up to kc
    int pitch;    // rows of a staged sample, padded by 2 against bank conflicts of the transposing stores
    int taps;     // padded doubles of one tap table
};

// groups: fewer groups of rows per block than the default (0), for calls of few rows.
__host__ __device__ inline FiltShape filter_shape(int C, int groups = 0) {
    FiltShape f;
    f.outs = (C + 1) / 2;
    f.tiles = (f.outs + 63) / 64;
    f.groups = f.tiles >= 3 ? 1 : (f.tiles == 2 ? 2 : 4);
    if (groups > 0 && groups < f.groups) f.groups = groups;
    f.rows = 16 * f.groups;
    f.kc = 2048 / f.rows;
    f.kp = (f.outs + f.kc - 1) / f.kc * f.kc;
    f.pitch = f.rows + 2;
    f.taps = 9 * ((64 * f.tiles + f.kp) / 8 + 2);
    return f;
}

// Rows whose chunks are nearly all used take them whole: 512 channels (all used) 1.50 ms with unchanging bounds and 1.56
// without, 1000 (500 of 512 samples) 624 and 644 us, but 437 (219 of 256) 569 and 501.
inline bool filter_whole(int C) {
    const FiltShape f = filter_shape(C);
    return 20 * f.outs >= 19 * f.kp;
}

inline size_t filter_smem_bytes(int C, int groups = 0) {
    const FiltShape f = filter_shape(C, groups);
    return sizeof(double) * (2 * (size_t)f.kc * f.pitch + 2 * (size_t)f.taps);
}

// Filters rows row0 .. row0 + filter_shape(C).rows - 1 (fewer at the end) of a (num_rows_total, C) stack of detector rows
// (R rows per view) with the whole block; sm holds filter_smem_bytes(C).
// The samples (FDK: pre-weighted), the taps, the sums and the scales are float64 and each output is rounded once, as the
// reference's filter is specified (a float64 evaluation of the convolution differs from any float32 one by rounding only).
//
// Only the centre tap and the odd ones are nonzero, so outputs of one parity sum samples of the other.  A lane holds 4
// rows x 8 consecutive outputs of its parity, 32 float64 accumulators; from one sample to the next its 8 taps move by
// one place, so a sample costs one tap load, two 16-byte loads of 4 rows (staged as float64, [sample][row]) and 32 FMAs,
// and the loop is bound by the float64 pipe (half the float32 rate).  The tap tables (one per parity) are padded to 9
// doubles per 8 taps, which keeps the lanes' loads, 8 taps apart, in different banks.  Measured on 360 x 256 x 512 (FDK):
// 5.53 -> 1.50 ms against one output and 8 rows per thread, whose samples were converted to float64 at every use.
// WHOLE: every chunk of samples is taken whole, zeros past the row, with bounds that do not change from chunk to chunk
// (filter_whole); else the last one ends with the row.
template <bool WHOLE = false>
__device__ __forceinline__ void direct_filter_rows(const float *__restrict__ sino, float *__restrict__ out,
                                                   long long row0, long long num_rows_total, int R, int C,
                                                   double filter_scale, double out_scale, int fdk, double D,
                                                   double delta_det_channel, double delta_det_row,
                                                   double det_channel_offset, double det_row_offset, double *sm,
                                                   int groups = 0) {
    const FiltShape f = filter_shape(C, groups);
    double *xs = sm;                              // [2][kc][pitch]: staged samples by parity
    double *taps = sm + 2 * f.kc * f.pitch;       // [2][f.taps]
    float *ot = reinterpret_cast<float *>(sm);    // finished outputs, [rows][128 * tiles of a pass] (after the last sample)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nrows = (int)min((long long)f.rows, num_rows_total - row0);
    const bool weighted = fdk && isfinite(D);

    // taps: entry E of table p holds h[2e + 1], e = E - kp - (p ? 7 : 8), at place E + E / 8
    const double kInvPi2 = 0.10132118364233778;  // 1 / pi^2
    for (int t = tid; t < 2 * f.taps; t += FILT_THREADS) {
        const int p = t >= f.taps, i = t - p * f.taps, E = i / 9 * 8 + min(i % 9, 7);
        const double d = 2.0 * (double)(E - f.kp - (p ? 7 : 8)) + 1.0;
        taps[t] = filter_scale * (-kInvPi2 / (d * d));
    }

    const int p = warp & 1, slot = warp >> 1;                       // parity; row group and tile of a pass
    const int per_pass = 4 / f.groups;                              // tiles of a pass
    const int rowl = (slot / per_pass) * 16 + (lane >> 3) * 4;      // this lane's first row
    const double *xrow = xs + (p ^ 1) * f.kc * f.pitch + rowl;      // samples of the other parity
    const double *xcen = xs + p * f.kc * f.pitch + rowl;
    for (int t0 = 0; t0 < f.tiles; t0 += per_pass) {
        const int tile = t0 + slot % per_pass;
        const int o0 = tile * 64 + (lane & 7) * 8;                  // first of this lane's outputs (channel 2 o + p)
        const double *tap = taps + p * f.taps + 9 * ((o0 + f.kp) >> 3);  // group of the taps of sample 0
        double acc[8][4], g[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[u][r] = 0.0;
        for (int k0 = 0; k0 < f.kp; k0 += f.kc) {
            __syncthreads();  // the last samples (and, at the start of a pass, its predecessor's outputs) are read
            const int kn = WHOLE ? f.kc : min(f.kc, (f.outs - k0 + 7) & ~7);  // samples of the chunk, in eights
            for (int t = tid; t < 2 * kn * f.rows; t += FILT_THREADS) {
                const int rr = t / (2 * kn), cc = t - rr * 2 * kn, j = 2 * k0 + cc;
                double v = 0.0;
                if (rr < nrows && j < C) {
                    const long long row = row0 + rr;
                    v = (double)sino[row * C + j];
                    if (weighted) {
                        const double vv = ((double)(int)(row % R) - 0.5 * (double)(R - 1)) * delta_det_row - det_row_offset;
                        const double uu = ((double)j - 0.5 * (double)(C - 1)) * delta_det_channel - det_channel_offset;
                        v *= D * rsqrt(D * D + uu * uu + vv * vv);
                    }
                }
                xs[((cc & 1) * f.kc + (cc >> 1)) * f.pitch + rr] = v;
            }
            __syncthreads();
            if (tile >= f.tiles) continue;
            if (k0 == 0) {
#pragma unroll
                for (int u = 1; u < 8; ++u) g[u] = tap[9 + u - 1];
            }
            if (o0 >= k0 && o0 < k0 + kn) {  // the centre tap
                const double h0 = 0.25 * filter_scale;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const double2 a = *reinterpret_cast<const double2 *>(xcen + (o0 - k0 + u) * f.pitch);
                    const double2 b = *reinterpret_cast<const double2 *>(xcen + (o0 - k0 + u) * f.pitch + 2);
                    acc[u][0] = fma(h0, a.x, acc[u][0]);
                    acc[u][1] = fma(h0, a.y, acc[u][1]);
                    acc[u][2] = fma(h0, b.x, acc[u][2]);
                    acc[u][3] = fma(h0, b.y, acc[u][3]);
                }
            }
            const double *x = xrow;
            for (int k = 0; k < kn; k += 8) {
#pragma unroll
                for (int s = 0; s < 8; ++s) {  // tap of output u at sample k + s: g[(u - s) & 7]
                    g[(8 - s) & 7] = tap[7 - s];
                    const double2 a = *reinterpret_cast<const double2 *>(x);
                    const double2 b = *reinterpret_cast<const double2 *>(x + 2);
                    x += f.pitch;
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const double h = g[(u - s) & 7];
                        acc[u][0] = fma(h, a.x, acc[u][0]);
                        acc[u][1] = fma(h, a.y, acc[u][1]);
                        acc[u][2] = fma(h, b.x, acc[u][2]);
                        acc[u][3] = fma(h, b.y, acc[u][3]);
                    }
                }
                tap -= 9;
            }
        }
        __syncthreads();  // the staged samples are read: their place takes the outputs, which leave coalesced
        const int width = 128 * per_pass;
        if (tile < f.tiles) {
#pragma unroll
            for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    ot[(rowl + r) * width + 2 * (o0 - 64 * t0 + u) + p] = (float)(out_scale * acc[u][r]);
        }
        __syncthreads();
        const int c0 = 128 * t0, nc = min(width, C - c0);
        for (int t = tid; t < nrows * width; t += FILT_THREADS) {
            const int rr = t / width, cc = t - rr * width;
            if (cc < nc) out[(row0 + rr) * C + c0 + cc] = ot[t];
        }
    }
    __syncthreads();  // the block may stage its next tile into sm
}

}  // namespace mbx
