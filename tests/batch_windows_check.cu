// Host-only check of what a batch prepares for its back projections (vcd_batched.cuh), for a sweep of batches: a back
// projection that reads windows copies them through a map whose box has the rows of its own plan, since a copy waits for as
// many bytes as its plan's windows hold; one that does not has no map; the tiles are no higher than the batch says and cover
// the slices; and windows are read where the list fills the chip.  Prints "ok <scans> <scans whose plans differ> <batches
// with windows> <without>" or the first failure.  Runs on the CPU (no device call).
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
    long checked = 0, differ = 0, with = 0, without = 0;
    for (int kind : {MBX_GEOM_PARALLEL, MBX_GEOM_CONE, MBX_GEOM_TRANSLATION})
        for (int C : {48, 64, 96, 128, 192, 256})
            for (int R : {1, 4, 16, 17, 24, 32, 40, 64, 100, 128})
                for (int V : {24, 60, 180})
                    for (int K : {1, 2, 4, 16})
                        for (int n : {1, 3, 20})
                            for (int weighted = 0; weighted < 3; ++weighted) {  // 2: some scans of the batch
                                std::vector<mbx_scan> scans;
                                for (int s = 0; s < n; ++s)
                                    scans.push_back(make_scan(kind, V, R + s % 3, C + s, K, weighted == 1 || (weighted == 2 && s % 2)));
                                std::vector<ScanSizes> zs;
                                BatchBp B;
                                if (batch_sizes(scans.data(), n, zs, B) != MBX_OK) continue;
                                double units[SW_COUNT] = {};
                                auto fail = [&](const char *what, int w) {
                                    std::printf("FAIL %s: list %d of kind %d, %d scans of %d x %d x %d in %d\n", what, w,
                                                kind, n, V, R, C, K);
                                    return 1;
                                };
                                for (int s = 0; s < n; ++s) {
                                    bool same = true;
                                    ++checked;
                                    for (int w = 0; w < SW_COUNT; ++w) {
                                        const BpfPlan &p = scan_bp_plan(zs[s], w);
                                        if (kind == MBX_GEOM_TRANSLATION && w == SW_INIT) continue;  // (has none)
                                        if (scan_window_box(zs[s], w, B) != (B.windows[w] ? p.boxq : 0)) return fail("box", w);
                                        if (p.ts > B.most[w] || p.ts % 4 || p.ts * p.tiles < (zs[s].hbp_slices > 0 && w == SW_HESS ? 1 : R + s % 3))
                                            return fail("tiles", w);
                                        if (B.windows[w] && w == SW_HESS && !scans[s].weights) return fail("Hessian without weights", w);
                                        if (B.windows[w] && kind == MBX_GEOM_PARALLEL && p.boxq * 4 < p.ts) return fail("window rows", w);
                                        if (B.windows[w] && bpf_window_channels(kind, p.boxq) < BPF_BOX) return fail("window channels", w);
                                        units[w] += (double)p.gx * p.gy * BPF_WARPS / (8.0 * BPF_LAUNCH_WARPS * num_sms());
                                        same = same && p.boxq == scan_bp_plan(zs[s], SW_SUBSET).boxq;
                                    }
                                    differ += same ? 0 : 1;
                                }
                                for (int w = 0; w < SW_COUNT; ++w)
                                    if (B.windows[w] && !(kind == MBX_GEOM_TRANSLATION && w == SW_INIT) && units[w] < BATCH_WINDOW_WAVES)
                                        return fail("windows on an idle chip", w);
                                (B.windows[SW_SUBSET] ? with : without) += 1;
                            }
    std::printf("ok %ld %ld %ld %ld\n", checked, differ, with, without);
    return checked > 0 ? 0 : 1;
}
