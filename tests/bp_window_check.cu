// Host-only check of the parallel back projector's search for windows by the box of a warp's pixels (bp_fast.cuh): over
// recons of 1 to 40 slices, detectors up to 512 channels, grid boxes of every width and 180 views, a window that is not
// wide comes back from its one-word form as it went in; and so do all windows up to the widest that a plan has; printing
// "ok <windows> <of more than 255 channels>" or the first failure.  Runs on the CPU (no device call).
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
    std::printf("ok %ld %ld\n", windows, big);
    return windows > 0 ? 0 : 1;
}
