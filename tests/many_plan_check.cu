// Host-only check of plans that plan_layout_check.cu does not reach, with its layout and back-projection checks: the forward
// projector's second variant (plan_fp_many: parallel beam 4 CTAs per SM, 64 channels and passes of 1024 records; its
// alternative lane layout and narrower blocks, and the batch's passes), and the scratch of the entry point that allocates
// nothing (the partial sums of both back projectors).  Prints "ok <plans checked>" or the first failure.  Runs on the CPU.
#define main plan_layout_main
#include "plan_layout_check.cu"
#undef main

#include "../mbirjax_b200/csrc/bp_gather.cuh"

static mbx_geom geometry(int kind, int V, int R, int C) {
    mbx_geom g = {};
    g.kind = kind;
    g.num_views = V;
    g.num_det_rows = g.num_recon_slices = R;
    g.num_det_channels = g.num_recon_rows = g.num_recon_cols = C;
    g.psf_radius = g.bp_psf_radius = 1;
    g.entries_per_cylinder_batch = 128;
    g.delta_det_channel = g.delta_det_row = g.delta_voxel = g.delta_recon_row = 1.0f;
    g.source_detector_dist = kind == MBX_GEOM_PARALLEL ? INFINITY : 4.0f * C;
    g.magnification = kind == MBX_GEOM_PARALLEL ? 1.0f : 2.0f;
    g.max_magnification = kind == MBX_GEOM_TRANSLATION ? 2.0f : 0.0f;
    return g;
}

int main() {
    long checked = 0;
    const int chans[7] = {32, 96, 131, 200, 317, 512, 1024};
    for (int kind : {MBX_GEOM_PARALLEL, MBX_GEOM_CONE, MBX_GEOM_TRANSLATION})
        for (int R = 1; R <= 260; R += R < 100 ? 1 : 13)
            for (int C : chans) {
                const mbx_geom g = geometry(kind, 64, R, C);
                for (int nb_max : {128, 64, 32})
                    for (int max_cap : {2048, 1024})
                        for (int views : {0, 5, 64})
                            for (int alt = 0; alt < 2; ++alt) {
                                const CbPlan base = plan_fp_many(g, views, 512, nb_max, 0, max_cap);
                                if (!base.ok) continue;
                                const CbPlan pl = alt ? plan_fp_many(g, views, 512, nb_max, base.ppw, max_cap) : base;
                                if (!pl.ok) continue;
                                ++checked;
                                if (pl.minb != cb_many(kind)) return fail("variant", kind, R, C);
                                if (pl.nb > nb_max || (cb_many(kind) >= 4 && pl.nb > CB_MANY_CHANNELS)) return fail("block width", kind, R, C);
                                if (pl.walk.cap > max_cap || (cb_many(kind) >= 4 && pl.walk.cap > CB_MANY_CAP)) return fail("pass size", kind, R, C);
                                if (pl.walk.smem > 200 * 1024) return fail("walk over 200 KB", kind, R, C);
                                if (!layout_ok(pl, pl.walk, kind, R, false)) return fail("walk layout", kind, R, C);
                                if (!layout_ok(pl, pl.replay, kind, R, true)) return fail("replay layout", kind, R, C);
                                if (pl.replay.smem > pl.walk.smem) return fail("replay larger than walk", kind, R, C);
                                if (!layout_ok(pl, pl.small, kind, R, false)) return fail("small layout", kind, R, C);
                                if (pl.small.smem > pl.replay.smem) return fail("small walk over replay smem", kind, R, C);
                                if (pl.rpad < R || pl.rpad != pl.row_passes * pl.rl * pl.rpl) return fail("rows", kind, R, C);
                            }
                for (long long n : {1LL, 33LL, 257LL, 1000LL, 5000LL, 20000LL, (long long)C * C})
                    for (int nv : {1, 15, 16, 180, 4096}) {
                        const BpfPlan pl = plan_bp_fast(g, n, nv, 1);
                        if (!pl.ok) continue;
                        ++checked;
                        const char *e = bp_plan_error(g, pl, n, nv);
                        if (e) return fail(e, kind, R, C);
                        if (pl.workspace > BPF_PARTIAL_BYTES + 256) return fail("partial sums over their limit", kind, R, C);
                        if (kind != MBX_GEOM_PARALLEL) continue;
                        const BpgPlan own = plan_bp_gather(g, n, nv), as = plan_bp_gather(g, n, nv, pl.splits);
                        if (own.workspace > MBX_NOALLOC_SCRATCH_BYTES) return fail("gather over the scratch", kind, R, C);
                        if (as.splits != pl.splits || as.views_per_split != pl.views_per_split || as.workspace != pl.workspace)
                            return fail("gather in the windows' splits", kind, R, C);
                        for (const BpgPlan &q : {own, as})
                            if (q.ts < 1 || q.ts > BPG_ST || (long long)q.gy * q.nsl * q.ts < R || (long long)q.gx * (256 / q.nsl) < n ||
                                (1 << q.lg_pcta) != 256 / q.nsl || (long long)q.splits * q.views_per_split < nv)
                                return fail("gather tiles", kind, R, C);
                    }
            }
    std::printf("ok %ld\n", checked);
    return checked > 0 ? 0 : 1;
}
