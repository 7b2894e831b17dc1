// Host-only check of the parallel back projector's search for windows by the box of a warp's pixels (bp_fast.cuh): over
// recons of 1 to 40 slices, detectors up to 512 channels, grid boxes of every width and 180 views, a window that is not
// wide comes back from its one-word form as it went in; and so do all windows up to the widest that a plan has; and the taps
// of a box's pixels, with their centre channel rounded one way or another, lie in its window, for detectors up to a million
// channels; printing "ok <windows> <of more than 255 channels> <pixels>" or the first failure.  Runs on the CPU (no device call).
#include <cmath>
#include <cstdio>

#include "../mbirjax_b200/csrc/bp_fast.cuh"

namespace mbx {
int num_sms() { return 148; }  // the device query of the library, for a B200
}  // namespace mbx

using namespace mbx;

static bool packs(int c_lo, int nch) {
    const int w = bpf_pack_window(c_lo, nch);
    return bpf_packed_first(w) == c_lo && bpf_packed_channels(w) == nch;
}

int main() {
    long windows = 0, big = 0;
    for (int S : {1, 2, 3, 4, 5, 8, 9, 12, 13, 16, 17, 27, 28, 32, 40})
        for (int C : {32, 255, 256, 260, 280, 300, 512}) {
            mbx_geom g = {};
            g.kind = MBX_GEOM_PARALLEL;
            g.num_views = 180;
            g.num_det_rows = g.num_recon_slices = S;
            g.num_det_channels = g.num_recon_rows = g.num_recon_cols = C;
            g.psf_radius = 1;
            g.delta_det_channel = g.delta_det_row = g.delta_voxel = 1.0f;
            g.source_detector_dist = INFINITY;
            g.magnification = 1.0f;
            const int cap = bpf_window_channels(MBX_GEOM_PARALLEL, plan_bp_fast(g, C * C, 180).boxq);
            for (int c_lo : {-BPF_EDGE, -1, 0, 1, 255, 256, C, 100000})
                for (int nch = 0; nch <= cap; ++nch)
                    if (!packs(c_lo, nch)) {
                        std::printf("FAIL first %d channels %d\n", c_lo, nch);
                        return 1;
                    }
            for (int v = 0; v < 180; ++v)
                for (int w = 1; w <= C; w += 3) {  // boxes of w columns and a few rows, in the middle of the grid
                    const int4 box = {C / 2, C / 2 + w % 7, (C - w) / 2, (C - w) / 2 + w - 1};
                    const float a = 3.14159265f * (float)v / 180.0f;
                    const BpfBounds b = bpf_bounds(g, std::cos(a), std::sin(a), true, box, cap);
                    if (b.wide || b.nch == 0) continue;
                    ++windows;
                    big += b.nch > 255 ? 1 : 0;
                    if (!packs(b.c_lo, b.nch)) {
                        std::printf("FAIL %d slices, %d channels, view %d, box of %d: first %d channels %d\n", S, C, v, w,
                                    b.c_lo, b.nch);
                        return 1;
                    }
                }
        }
    long pixels = 0;
    unsigned rnd = 1;
    auto draw = [&rnd]() { return (rnd = rnd * 1664525u + 1013904223u) >> 8; };
    for (int C : {300, 5000, 20000, 65536, 300000, 900000})
        for (float offset : {0.0f, 0.37f, -0.25f * (float)C})
            for (int it = 0; it < 20000; ++it) {
                mbx_geom g = {};
                g.kind = MBX_GEOM_PARALLEL;
                g.num_views = 1;
                g.num_det_rows = g.num_recon_slices = 28;
                g.num_det_channels = g.num_recon_cols = C;
                g.num_recon_rows = 64 + draw() % 2000;
                g.delta_det_channel = 1.0f;
                g.delta_voxel = 0.99f;
                g.det_channel_offset = offset;
                const int r0 = (int)(draw() % (unsigned)(g.num_recon_rows - 4)), c0 = (int)(draw() % (unsigned)(C - 20));
                const int4 box = {r0, r0 + (int)(draw() % 4), c0, c0 + (int)(draw() % 16)};
                const float a = 3.14159265f * (float)(draw() % 100000) / 100000.0f, cs = std::cos(a), sn = std::sin(a);
                const BpfBounds b = bpf_bounds(g, cs, sn, true, box, 288);
                if (b.wide) continue;
                for (int row : {box.x, box.y})
                    for (int col : {box.z, box.w}) {
                        const float yt = g.delta_voxel * ((float)row - 0.5f * (float)(g.num_recon_rows - 1));
                        const float xt = g.delta_voxel * ((float)col - 0.5f * (float)(C - 1));
                        const float mid = 0.5f * (float)(C - 1);
                        const float x[3] = {cs * xt - sn * yt, std::fma(cs, xt, -(sn * yt)), std::fma(-sn, yt, cs * xt)};
                        for (int k = 0; k < 6; ++k) {
                            const float n = k < 3 ? (x[k] + offset) + mid : std::fma(x[k - 3] + offset, 1.0f, mid);
                            const int nc = (int)std::rint(n);
                            if (nc + 1 < 0 || nc - 1 >= C) continue;
                            ++pixels;
                            const int first = nc - 1 < -BPF_EDGE ? -BPF_EDGE : nc - 1;
                            if (first < b.c_lo || (nc + 1 < C ? nc + 1 : C - 1) >= b.c_lo + b.nch) {
                                std::printf("FAIL %d channels: centre %d outside %d + %d\n", C, nc, b.c_lo, b.nch);
                                return 1;
                            }
                        }
                    }
            }
    std::printf("ok %ld %ld %ld\n", windows, big, pixels);
    return windows > 0 ? 0 : 1;
}
