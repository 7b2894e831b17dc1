// Host-only check of what a batch prepares for its back projections (vcd_batched.cuh): for a sweep of scans, the box of
// each back projection's tensor map has the rows of that back projection's own plan, since a copy waits for as many bytes
// as its plan's windows hold; printing "ok <scans> <scans whose plans differ>" or the first failure.  Runs on the CPU (no
// device call).
#include <cmath>
#include <cstdio>

#include "../mbirjax_b200/csrc/vcd_batched.cuh"

namespace mbx {
int num_sms() { return 148; }  // the device query of the library, for a B200
int validate_geom(const mbx_geom *) { return MBX_OK; }
}  // namespace mbx

using namespace mbx;

static mbx_scan make_scan(int kind, int V, int R, int C, int K, bool weighted) {
    static float dummy[1];
    static int32_t idummy[1];
    mbx_scan sc = {};
    mbx_geom &g = sc.geom;
    g.kind = kind;
    g.num_views = V;
    g.num_det_rows = g.num_recon_slices = R;
    g.num_det_channels = g.num_recon_rows = g.num_recon_cols = C;
    g.psf_radius = g.bp_psf_radius = 1;
    g.entries_per_cylinder_batch = 128;
    g.delta_det_channel = g.delta_det_row = g.delta_voxel = g.delta_recon_row = 1.0f;
    g.source_detector_dist = kind == MBX_GEOM_PARALLEL ? INFINITY : 4.0f * C;
    g.magnification = 1.0f;
    g.max_magnification = kind == MBX_GEOM_TRANSLATION ? 1.2f : 0.0f;
    sc.flat_recon = sc.error_sinogram = dummy;
    sc.fm_hessian = dummy;
    sc.weights = weighted ? dummy : nullptr;
    sc.sinogram = dummy;
    sc.partition = sc.full_indices = idummy;
    sc.num_full_indices = (int)(0.78 * C * C);
    sc.num_subsets = K;
    sc.subset_size = sc.num_full_indices / K;
    sc.qp.sigma_x = sc.qp.T = 1.0f;
    sc.qp.p = 2.0f;
    return sc;
}

int main() {
    long scans = 0, differ = 0;
    for (int kind : {MBX_GEOM_PARALLEL, MBX_GEOM_CONE, MBX_GEOM_TRANSLATION})
        for (int C : {48, 64, 96, 128, 192, 256})
            for (int R : {4, 16, 17, 24, 32, 40, 64, 100, 128})
                for (int V : {24, 60, 128, 180, 256})
                    for (int K : {1, 2, 4, 8, 16})
                        for (int weighted = 0; weighted < 2; ++weighted) {
                            ScanSizes z = {};
                            if (scan_sizes(make_scan(kind, V, R, C, K, weighted != 0), z) != MBX_OK) continue;
                            ++scans;
                            bool same = true;
                            for (int w = 0; w < SW_COUNT; ++w) {
                                if (scan_window_box(z, w) != scan_bp_plan(z, w).boxq) {
                                    std::printf("FAIL map %d of kind %d, %d x %d x %d in %d: box %d, plan %d\n", w, kind, V,
                                                R, C, K, scan_window_box(z, w), scan_bp_plan(z, w).boxq);
                                    return 1;
                                }
                                same = same && scan_window_box(z, w) == scan_window_box(z, 0);
                            }
                            differ += same ? 0 : 1;
                        }
    std::printf("ok %ld %ld\n", scans, differ);
    return scans > 0 ? 0 : 1;
}
