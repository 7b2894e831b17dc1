"""The work a user has this library do, as measurable cases: single projections, the set-up pieces of a
reconstruction (Hessian diagonal, FDK filter), the prior, a VCD subset update, a denoising and a batch of
reconstructions, each through the package's public entry points.

``listed()`` names the cases; ``draw(rng)`` makes another of the same ranges; ``prepare(case, seed)`` builds what a
program has in hand before the call; ``run(state)`` is one call; ``work(case)`` counts the bytes and operations it
cannot do without; ``exact(case, seed)`` evaluates the same outputs in 64 bits with plain torch and numpy.

Ranges: parallel beam as the benchmark's batch (views 60..720, rows 8..64, channels 96..512) and the small plain
configuration (64 x 16 x 128); cone beam around the benchmark's 256 x 128 x 256 up to 360 x 256 x 512; translation
geometry as the raster experiment (49 views of 128 x 128).  All data are float32, the one type the library computes
in; inputs are ellipsoid phantoms and their analytic line integrals with 1% noise.
"""
import math

import numpy as np
import torch

import mbirjax_b200 as mb
from mbirjax_b200 import torch_ops
from mbirjax_b200.batched import BatchedVCD
from mbirjax_b200.vcd_utils import gen_full_indices, gen_pixel_partition, morton_sorted_partition

EPS32 = 1.1920928955078125e-07
MAX_VOXEL_VIEWS = 2.5e9   # most (voxel, view) pairs of a drawn projection: no more than the largest listed one


def listed():
    return [
        # the smallest plain configuration: one full forward projection of a 128 x 128 x 16 recon
        {"name": "fp_parallel_small", "op": "fp", "kind": "parallel", "views": 64, "rows": 16, "channels": 128,
         "subsets": 1},
        # projections of one pixel subset inside a VCD iteration of a benchmark-sized parallel scan
        {"name": "fp_parallel_subset", "op": "fp", "kind": "parallel", "views": 652, "rows": 57, "channels": 437,
         "subsets": 4},
        {"name": "bp_parallel_subset", "op": "bp", "kind": "parallel", "views": 652, "rows": 57, "channels": 437,
         "subsets": 4},
        # the cone-beam benchmark scan: a subset forward projection
        {"name": "fp_cone_subset", "op": "fp", "kind": "cone", "views": 256, "rows": 128, "channels": 256,
         "subsets": 4},
        # a larger cone scan: a subset back projection
        {"name": "bp_cone_large", "op": "bp", "kind": "cone", "views": 360, "rows": 256, "channels": 512,
         "subsets": 8},
        # the translation raster experiment: back projection to the whole region of reconstruction
        {"name": "bp_translation", "op": "bp", "kind": "translation", "views": 49, "rows": 128, "channels": 128,
         "subsets": 1},
        # Hessian diagonal of a weighted cone scan of odd sizes, over every pixel of the grid
        {"name": "hessian_cone_weighted", "op": "hessian", "kind": "cone", "views": 180, "rows": 61, "channels": 203},
        # FDK filtering of a whole cone scan
        {"name": "filter_cone", "op": "filter", "kind": "cone", "views": 360, "rows": 256, "channels": 512},
        # one weighted VCD subset update of the cone-beam benchmark scan
        {"name": "vcd_step_cone", "op": "step", "kind": "cone", "views": 256, "rows": 128, "channels": 256,
         "subsets": 4},
        # value and gradient of the qGGMRF prior, as a gradient-based reconstruction calls them each step
        {"name": "prior_loss_grad", "op": "prior", "kind": "volume", "nr": 256, "nc": 256, "ns": 128},
        # qGGMRF denoising of a volume
        {"name": "denoise", "op": "denoise", "kind": "volume", "nr": 128, "nc": 128, "ns": 100, "iterations": 3},
        # reconstructions of a batch of uneven parallel scans (the first scans of the benchmark's batch)
        {"name": "batched_recon", "op": "batched", "kind": "parallel", "scans": 6, "first": 0, "iterations": 4,
         "views": 720, "rows": 64, "channels": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["fp", "bp", "fp", "bp", "hessian", "filter", "step", "prior", "denoise", "batched"])
    if op == "prior":
        return {"op": op, "kind": "volume", "nr": _log(rng, 24, 256), "nc": _log(rng, 24, 256),
                "ns": _log(rng, 8, 128)}
    if op == "denoise":
        return {"op": op, "kind": "volume", "nr": _log(rng, 24, 128), "nc": _log(rng, 24, 128),
                "ns": _log(rng, 8, 100), "iterations": 3}
    if op == "batched":
        return {"op": op, "kind": "parallel", "scans": rng.randint(2, 6), "first": rng.randint(1, 30),
                "iterations": rng.randint(2, 4), "views": _log(rng, 100, 720), "rows": _log(rng, 12, 64),
                "channels": _log(rng, 110, 400)}
    kind = rng.choice(["parallel", "cone"] if op in ("filter", "step") else ["parallel", "parallel", "cone", "cone",
                                                                             "translation"])
    while True:
        if kind == "translation":
            case = {"op": op, "kind": kind, "views": rng.choice([9, 25, 35, 49, 63]), "rows": _log(rng, 40, 128),
                    "channels": _log(rng, 40, 128)}
        elif kind == "cone":
            case = {"op": op, "kind": kind, "views": _log(rng, 24, 400), "rows": _log(rng, 12, 256),
                    "channels": _log(rng, 48, 512)}
        else:
            case = {"op": op, "kind": kind, "views": _log(rng, 60, 720), "rows": _log(rng, 8, 64),
                    "channels": _log(rng, 96, 512)}
        if op in ("fp", "bp", "step"):
            case["subsets"] = rng.choice([1, 4, 4, 8])
        if op == "filter" or _voxel_views(case) <= MAX_VOXEL_VIEWS:
            return case


# ------------------------------------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _translations(case):
    """A raster of translations 22 ALU apart in x and z (7 x 7 for 49 views), as many columns as fit the views."""
    n = case["views"]
    nx = max(k for k in range(1, int(math.sqrt(n)) + 1) if n % k == 0)
    nz = n // nx
    x = (np.arange(nx) - (nx - 1) / 2) * 22.0
    z = (np.arange(nz) - (nz - 1) / 2) * 22.0
    tv = np.zeros((n, 3))
    tv[:, 0], tv[:, 2] = np.tile(x, nz), np.repeat(z, nx)
    return tv


def _angles(case):
    stop = 2 * np.pi if case["kind"] == "cone" else np.pi
    return np.linspace(0, stop, case["views"], endpoint=False).astype(np.float32)


def _distance(case):
    """Source to detector and to isocentre (equal: magnification 1, as the benchmark's scans)."""
    return 0.5 * case["channels"] if case["kind"] == "translation" else 4.0 * case["channels"]


def _shape(case):
    return case["views"], case["rows"], case["channels"]


def _model(case):
    if case["kind"] == "parallel":
        return mb.ParallelBeamModel(_shape(case), _angles(case))
    if case["kind"] == "translation":
        return mb.TranslationModel(_shape(case), _translations(case), source_detector_dist=_distance(case),
                                   source_iso_dist=_distance(case))
    return mb.ConeBeamModel(_shape(case), _angles(case), source_detector_dist=_distance(case),
                            source_iso_dist=_distance(case))


def _recon_shape(case):
    """(recon shape, row pitch): channels x channels x rows for the rotating geometries at magnification 1; the
    translation geometry's own sizing of box and row pitch."""
    V, R, C = _shape(case)
    if case["kind"] != "translation":
        return (C, C, R), 1.0
    f32, tv, d = np.float32, _translations(case).astype(np.float32), _distance(case)
    box = np.array([C, R], dtype=f32)
    half = np.arctan2(np.max(box), f32(2 * d))
    pitch = float(f32(np.sqrt(2)) * (f32(1.0) / np.tan(half)))
    cube = np.amax(tv, axis=0) - np.amin(tv, axis=0)
    size = np.ceil(np.array([cube[0], cube[2]], dtype=f32) + box / f32(2))
    nr = np.minimum(np.ceil(f32(V * C * R) / (size[0] * size[1])), np.floor((f32(d) - cube[1]) / f32(pitch)))
    return (int(nr), int(size[0]), int(size[1])), pitch


def _subset_size(case):
    nr, nc = _recon_shape(case)[0][:2]
    if case["op"] == "hessian":
        return nr * nc
    r = (max(nr, nc) - 1) / 2
    rows, cols = np.arange(nr)[:, None] - (nr - 1) / 2, np.arange(nc)[None, :] - (nc - 1) / 2
    n = int(np.count_nonzero(rows ** 2 + cols ** 2 <= r * r))
    return -(-n // case.get("subsets", 1))


def _voxel_views(case):
    return float(case["views"]) * _subset_size(case) * _recon_shape(case)[0][2]


def _pixels(case, seed):
    """The pixel list of a call: the whole region of reconstruction in raster order, or one subset of a VCD
    partition in the order the reconstruction loop visits it."""
    shape = _recon_shape(case)[0]
    if case.get("subsets", 1) == 1:
        return np.asarray(gen_full_indices(shape, rng=np.random.RandomState(seed % (2 ** 31))), dtype=np.int32)
    part = gen_pixel_partition(shape, case["subsets"], rng=np.random.RandomState(seed % (2 ** 31)))
    return morton_sorted_partition(part, shape[1])[seed % case["subsets"]]


def _ellipsoids(seed, size, count=10):
    """Centres, half-axes, in-plane rotations and densities of seeded ellipsoids in a box of the given half-size."""
    rng = np.random.default_rng([seed, 7])
    half = np.asarray(size, dtype=np.float64)
    centre = rng.uniform(-0.6, 0.6, (count, 3)) * half
    axes = rng.uniform(0.08, 0.35, (count, 3)) * half
    return centre, axes, rng.uniform(0.0, np.pi, count), rng.uniform(0.1, 1.0, count)


def _generator(seed, salt):
    return torch.Generator(device=_device()).manual_seed((seed * 1000003 + salt) % (2 ** 31))


def _phantom(shape, seed):
    """Sum of seeded ellipsoids on the voxel grid, (rows, cols, slices) float32."""
    dev = _device()
    nr, nc, ns = shape
    y = torch.arange(nr, device=dev, dtype=torch.float32).reshape(-1, 1, 1) - (nr - 1) / 2
    x = torch.arange(nc, device=dev, dtype=torch.float32).reshape(1, -1, 1) - (nc - 1) / 2
    z = torch.arange(ns, device=dev, dtype=torch.float32).reshape(1, 1, -1) - (ns - 1) / 2
    out = torch.zeros(shape, device=dev)
    for c, a, t, d in zip(*_ellipsoids(seed, (nc / 2, nr / 2, ns / 2))):
        u = (math.cos(t) * (x - c[0]) + math.sin(t) * (y - c[1])) / a[0]
        v = (-math.sin(t) * (x - c[0]) + math.cos(t) * (y - c[1])) / a[1]
        w = (z - c[2]) / a[2]
        out += d * ((u * u + v * v) + w * w <= 1.0)
    return out


def _sinogram(case, seed, noise=0.01):
    """Line integrals of seeded ellipsoids along each view's rays (parallel rays for every geometry: the values a
    projector meets do not depend on it) plus noise of 1% of the largest, (views, rows, channels) float32."""
    dev = _device()
    V, R, C = _shape(case)
    ang = torch.as_tensor(np.linspace(0, np.pi, V, endpoint=False), dtype=torch.float32, device=dev).reshape(-1, 1, 1)
    n = torch.arange(C, device=dev, dtype=torch.float32).reshape(1, 1, -1) - (C - 1) / 2
    z = torch.arange(R, device=dev, dtype=torch.float32).reshape(1, -1, 1) - (R - 1) / 2
    out = torch.zeros((V, R, C), device=dev)
    for c, a, t, d in zip(*_ellipsoids(seed, (C / 2, C / 2, R / 2))):
        s = (n - (torch.cos(ang) * c[0] - torch.sin(ang) * c[1]))
        phi = ang + t
        width2 = (a[0] * torch.cos(phi)) ** 2 + (a[1] * torch.sin(phi)) ** 2
        w = 1.0 - ((z - c[2]) / a[2]) ** 2
        out += (2.0 * d * a[0] * a[1]) * torch.sqrt(torch.clamp(w * width2 - s * s, min=0.0)) / width2
    if noise:
        g = _generator(seed, 11)
        out += noise * float(out.max()) * torch.randn(out.shape, generator=g, device=dev)
    return out


def _inputs(case, seed):
    """The tensors of a case, by name; the same for prepare and exact."""
    op = case["op"]
    if op == "prior":
        x = _phantom((case["nr"], case["nc"], case["ns"]), seed)
        return {"x": x + 0.02 * torch.randn(x.shape, generator=_generator(seed, 3), device=x.device)}
    if op == "denoise":
        x = _phantom((case["nr"], case["nc"], case["ns"]), seed)
        return {"x": x + 0.1 * torch.randn(x.shape, generator=_generator(seed, 3), device=x.device)}
    if op == "filter":
        return {"sino": _sinogram(case, seed)}
    shape = _recon_shape(case)[0]
    if op == "hessian":
        sino = _sinogram(case, seed, noise=0.0)
        return {"weights": torch.exp(-sino / sino.max())}
    pix = torch.as_tensor(_pixels(case, seed), device=_device())
    got = {"pix": pix}
    if op == "bp":
        got["sino"] = _sinogram(case, seed)
    else:
        x = _phantom(shape, seed).reshape(-1, shape[2])
        if op == "fp":
            got["vox"] = x[pix.long()].contiguous()
    if op == "step":
        sino = _sinogram(case, seed, noise=0.0)
        top = float(sino.max())
        g = _generator(seed, 5)
        got["weights"] = torch.exp(-sino / top)
        got["err"] = 0.02 * top * torch.randn(sino.shape, generator=g, device=sino.device)
        got["recon"] = (x + 0.02 * torch.randn(x.shape, generator=g, device=x.device)).contiguous()
        got["hess"] = 0.5 * case["views"] * (0.8 + 0.4 * torch.rand(x.shape, generator=g, device=x.device))
        got["fm"] = 1.0 / (0.02 * top) ** 2
    return got


# qGGMRF parameters of the calls: the defaults p = 2, q = 1.2, T = 1 with unit neighbour weights
# (b, sigma_x, p, q, T), each a 32-bit value, as the library holds them
_QPARAMS = ([float(np.float32(1.0 / 6.0))] * 6, 0.0625, 2.0, float(np.float32(1.2)), 1.0)
_DENOISE = {"sigma": 0.1, "subsets": 16}


def _batch_shapes(case):
    """Uneven scans: the benchmark's batch draws views, rows and channels of scan i from seed i; a drawn batch caps
    them."""
    shapes = []
    for i in range(case["first"], case["first"] + case["scans"]):
        rng = np.random.default_rng(i)
        v, r, c = int(rng.integers(60, 721)), int(rng.integers(8, 65)), int(rng.integers(96, 513))
        shapes.append((min(v, case["views"]), min(r, case["rows"]), min(c, case["channels"])))
    return shapes


def prepare(case, seed):
    op = case["op"]
    state = {"op": op, "case": dict(case)}
    if op == "batched":
        state["models"], state["sinos"] = [], []
        for i, (v, r, c) in enumerate(_batch_shapes(case)):
            one = {"kind": "parallel", "views": v, "rows": r, "channels": c}
            model = _model(one)
            model.set_params(sharpness=0.0, snr_db=30.0, granularity=[4], partition_sequence=[0], verbose=0)
            state["models"].append(model)
            state["sinos"].append(_sinogram(one, seed * 64 + i))
        state["seeds"] = [(seed + i) % (2 ** 31) for i in range(case["scans"])]
        return state
    state.update(_inputs(case, seed))
    if op == "prior":
        return state
    if op == "denoise":
        model = mb.QGGMRFDenoiser((case["nr"], case["nc"], case["ns"]))
        model.set_params(no_warning=True, auto_regularize_flag=False, sigma_y=_DENOISE["sigma"],
                         sigma_x=_QPARAMS[1], granularity=[_DENOISE["subsets"]], partition_sequence=[0])
        state.update(model=model, seed=seed % (2 ** 31))
        return state
    model = _model(case)
    assert tuple(model.get_params("recon_shape")) == _recon_shape(case)[0]
    state["model"] = model
    if op == "step":
        state["ops"] = torch_ops.load()
        state["geom"] = torch_ops.geometry_args(_with_geometry(model))
        b, sigma_x, p, q, T = _QPARAMS
        state["qparams"] = torch_ops.qparams_args(b, sigma_x, p, q, T)
        state["work"] = (torch.empty_like(state["recon"]), torch.empty_like(state["err"]),
                         torch.zeros(4, dtype=torch.float64, device=state["err"].device))
    return state


def _with_geometry(model):
    model._geometry()
    return model


def run(state):
    op = state["op"]
    if op == "fp":
        return state["model"].sparse_forward_project(state["vox"], state["pix"])
    if op == "bp":
        return state["model"].sparse_back_project(state["sino"], state["pix"])
    if op == "hessian":
        return state["model"].compute_hessian_diagonal(weights=state["weights"])
    if op == "filter":
        return state["model"].direct_filter(state["sino"])
    if op == "prior":
        loss, grad = mb.qggmrf_loss_and_grad(state["x"], _QPARAMS)
        return {"loss": loss, "grad": grad}
    if op == "step":
        # the update works in place: on a copy of the state, so that every pass makes the same update
        recon, err, stats = state["work"]
        recon.copy_(state["recon"])
        err.copy_(state["err"])
        gi, gf, views = state["geom"]
        state["ops"].vcd_subset_step(gi, gf, views, recon, err, state["weights"], state["hess"], state["pix"],
                                     state["fm"], state["qparams"], stats)
        return {"recon": recon, "err": err, "stats": stats}
    if op == "denoise":
        np.random.seed(state["seed"])
        image, _ = state["model"].denoise(state["x"], sigma_noise=_DENOISE["sigma"],
                                          max_iterations=state["case"]["iterations"], stop_threshold_change_pct=0,
                                          logfile_path=None, print_logs=False)
        return image
    recons, info = BatchedVCD(state["models"], state["sinos"], seeds=state["seeds"]).recon(
        max_iterations=state["case"]["iterations"])
    return {"recons": recons, "fm_rmse": [d["fm_rmse"][-1] for d in info]}


def work(case):
    op = case["op"]
    if op == "batched":
        total = {"bytes": 0.0, "flops": 0.0}
        for v, r, c in _batch_shapes(case):
            n = math.pi / 4 * c * c
            # set-up (back projection, forward projection, a one-slice Hessian) and the projection pair of every
            # subset of every iteration; sinogram in, recon out
            total["flops"] += 6.0 * v * n * (2 * r + 1 + 2 * r * case["iterations"])
            total["bytes"] += 4.0 * (v * r * c + c * c * r)
        return total
    if case["kind"] == "volume":
        n = float(case["nr"]) * case["nc"] * case["ns"]
        if op == "prior":
            return {"bytes": 8.0 * n, "flops": 90.0 * n}
        return {"bytes": 8.0 * n * case["iterations"], "flops": 150.0 * n * case["iterations"]}
    V, R, C = (float(v) for v in _shape(case))
    if op == "filter":
        return {"bytes": 8.0 * V * R * C, "flops": V * R * C * C}
    shape = _recon_shape(case)[0]
    N, S = float(_subset_size(case)), float(shape[2])
    # per (pixel, view): three channel taps per detector row, and for the fan geometries three row taps per slice
    pair = V * N * (6.0 * S if case["kind"] == "parallel" else 6.0 * (R + S))
    if op == "fp" or op == "bp":
        return {"bytes": 4.0 * (N * S + N + V * R * C), "flops": pair}
    if op == "hessian":
        return {"bytes": 4.0 * (N * S + V * R * C), "flops": pair}
    return {"bytes": 4.0 * (3.0 * V * R * C + 4.0 * N * S + N), "flops": 2.0 * pair + 60.0 * N * S}


# ------------------------------------------------------------------------------------------------ 64-bit values
class _Projector:
    """The projection pair of a case in float64: separable footprints, voxel widths projected onto channels and
    (cone, translation) rows, each coefficient the overlap of the projected voxel with the detector element."""

    def __init__(self, case, pix):
        self.case, self.kind = case, case["kind"]
        (self.nr, self.nc, self.ns), pitch = _recon_shape(case)
        self.V, self.R, self.C = _shape(case)
        pix = pix.long()
        row, col = torch.div(pix, self.nc, rounding_mode="floor"), pix % self.nc
        self.x = col.double() - (self.nc - 1) / 2
        self.y = float(np.float32(pitch)) * (row.double() - (self.nr - 1) / 2)
        self.views = (_translations(case).astype(np.float32) if self.kind == "translation" else _angles(case)).astype(
            np.float64)
        self.D = _distance(case)

    def channels(self, v):
        """(centre channel, three coefficients (N, 3), magnification or None, z shift) of every pixel in view v."""
        zoff = 0.0
        if self.kind == "parallel":
            c, s = math.cos(self.views[v]), math.sin(self.views[v])
            n_p = c * self.x - s * self.y + (self.C - 1) / 2
            cos_alpha = max(abs(c), abs(s))
            w = torch.full_like(n_p, cos_alpha)
            scale, mag = torch.full_like(n_p, 1.0 / cos_alpha), None
        elif self.kind == "cone":
            c, s = math.cos(self.views[v]), math.sin(self.views[v])
            mag = 1.0 / (1.0 - (s * self.x + c * self.y) / self.D)
            u = mag * (c * self.x - s * self.y)
            n_p = u + (self.C - 1) / 2
            theta = torch.atan2(u, torch.full_like(u, self.D))
            d = self.views[v] - theta
            cos_alpha = torch.maximum(torch.cos(d).abs(), torch.sin(d).abs())
            w, scale = mag * cos_alpha / torch.cos(theta), 1.0 / cos_alpha
        else:
            tx, ty, tz = self.views[v]
            mag = 1.0 / (1.0 - (self.y - ty) / self.D)
            u = mag * (self.x - tx)
            n_p = u + (self.C - 1) / 2
            w, scale = mag, 1.0 / torch.cos(torch.atan2(u, torch.full_like(u, self.D)))
            zoff = -tz
        n_c = torch.round(n_p)
        k = torch.arange(-1, 2, device=n_p.device, dtype=torch.float64)
        n = n_c[:, None] + k
        a = torch.minimum(torch.clamp((w[:, None] + 1) / 2 - (n_p[:, None] - n).abs(), min=0.0),
                          torch.clamp(w[:, None], max=1.0)) * scale[:, None]
        a = torch.where((n >= 0) & (n < self.C), a, torch.zeros_like(a))
        return n.long().clamp(0, self.C - 1), a, mag, zoff

    def _secant(self, mag, z):
        return torch.sqrt(1.0 + (mag[:, None] * z / self.D) ** 2)

    def back(self, sino, power=1):
        """sum over views of A^power applied to the sinogram: (N, S) float64."""
        dev, N = sino.device, self.x.numel()
        out = torch.zeros((N, self.ns), dtype=torch.float64, device=dev)
        k = torch.arange(self.ns, device=dev, dtype=torch.float64) - (self.ns - 1) / 2
        for v in range(self.V):
            n, a, mag, zoff = self.channels(v)
            view = sino[v].double().t().contiguous()  # (C, R)
            a = a ** power
            rows = sum(a[:, j:j + 1] * view[n[:, j]] for j in range(3))  # (N, R)
            if mag is None:
                out += rows
                continue
            z = k + zoff
            m_p = mag[:, None] * z + (self.R - 1) / 2
            sec = self._secant(mag, z)
            w = mag[:, None]
            for j in (-1, 0, 1):
                m = torch.round(m_p) + j
                lap = torch.minimum(torch.clamp((w + 1) / 2 - (m_p - m).abs(), min=0.0), torch.clamp(w, max=1.0))
                lap = torch.where((m >= 0) & (m < self.R), (lap * sec) ** power, torch.zeros_like(lap))
                out += lap * torch.gather(rows, 1, m.long().clamp(0, self.R - 1))
        return out

    def forward(self, vox):
        """A applied to the voxel cylinders (N, S): (V, R, C) float64."""
        dev = vox.device
        vox = vox.double()
        out = torch.zeros((self.V, self.R, self.C), dtype=torch.float64, device=dev)
        m = torch.arange(self.R, device=dev, dtype=torch.float64) - (self.R - 1) / 2
        for v in range(self.V):
            n, a, mag, zoff = self.channels(v)
            if mag is None:
                rows = vox
            else:
                w = mag[:, None]
                k_m = (m / w - zoff) + (self.ns - 1) / 2
                rows = torch.zeros((vox.shape[0], self.R), dtype=torch.float64, device=dev)
                for j in (-1, 0, 1):
                    k = torch.round(k_m) + j
                    lap = torch.minimum(torch.clamp((w + 1) / 2 - (w * (k - k_m)).abs(), min=0.0),
                                        torch.clamp(w, max=1.0))
                    sec = torch.sqrt(1.0 + (w * (k - (self.ns - 1) / 2 + zoff) / self.D) ** 2)
                    lap = torch.where((k >= 0) & (k < self.ns), lap * sec, torch.zeros_like(lap))
                    rows += lap * torch.gather(vox, 1, k.long().clamp(0, self.ns - 1))
            view = torch.zeros((self.C, self.R), dtype=torch.float64, device=dev)
            for j in range(3):
                view.index_add_(0, n[:, j], a[:, j:j + 1] * rows)
            out[v] = view.t()
        return out


def _two_b_tilde(delta, b, sigma_x, p, q, T):
    s = delta.abs() / (T * sigma_x) + EPS32
    d_q2, d_qp = s ** (q - 2.0), s ** (q - p)
    return b * (T ** (p - 2.0) / sigma_x ** 2) * d_q2 * (q / p + d_qp) / (1.0 + d_qp) ** 2


def _prior_grad_hess(x, params):
    """Surrogate gradient and Hessian of the qGGMRF prior at every voxel of x (rows, cols, slices), float64."""
    b, sigma_x, p, q, T = params
    grad, hess = torch.zeros_like(x), torch.zeros_like(x)
    for axis in range(3):
        n = x.shape[axis]
        idx = torch.arange(n, device=x.device)
        for j, step in enumerate((1, -1)):
            nbr = x.index_select(axis, (idx + step).clamp(0, n - 1))
            bt = _two_b_tilde(x - nbr, b[2 * axis + j], sigma_x, p, q, T)
            grad += bt * (x - nbr)
            hess += bt
    return grad, hess


def _exact_prior(x, params):
    b, sigma_x, p, q, T = params
    x = x.double()
    loss, grad = torch.zeros((), dtype=torch.float64, device=x.device), torch.zeros_like(x)
    a_min = T * sigma_x * EPS32
    for axis in range(3):
        n = x.shape[axis]
        if n < 2:
            continue
        w = (b[2 * axis] + b[2 * axis + 1]) / (2.0 * sum(b))
        d = x.narrow(axis, 1, n - 1) - x.narrow(axis, 0, n - 1)
        a = torch.clamp(d.abs(), min=a_min)
        u = (a / (T * sigma_x)) ** (q - p)
        loss += w * torch.sum(a ** p / (p * sigma_x ** p) * u / (1.0 + u))
        dr = torch.sign(d) * a ** (p - 1.0) / sigma_x ** p * u * (q / p + u) / (1.0 + u) ** 2
        dr = w * torch.where(d.abs() < a_min, torch.zeros_like(dr), dr)
        grad.narrow(axis, 1, n - 1).add_(dr)
        grad.narrow(axis, 0, n - 1).sub_(dr)
    return {"loss": loss, "grad": grad}


def _exact_denoise(case, seed, x):
    shape = (case["nr"], case["nc"], case["ns"])
    np.random.seed(seed % (2 ** 31))
    count = shape[0] * shape[1]
    k = min(_DENOISE["subsets"], count)
    per = int(np.ceil(count / k))
    idx = np.random.permutation(np.arange(count, dtype=np.int32))
    extra = np.random.choice(idx[:(k - 1) * per], size=k * per - count, replace=False)
    subsets = np.sort(np.concatenate((idx, extra)).reshape(k, -1), axis=1)
    image = x.double().reshape(-1, shape[2]).clone()
    err = torch.zeros_like(image)
    fm = float(np.float32(1.0 / _DENOISE["sigma"] ** 2))
    for _ in range(case["iterations"]):
        for sub in subsets:
            sub = torch.as_tensor(sub, device=x.device).long()
            grad, hess = _prior_grad_hess(image.reshape(shape), _QPARAMS)
            gp, hp, e = grad.reshape(image.shape)[sub], hess.reshape(image.shape)[sub], err[sub]
            delta = (fm * e - gp) / (1.0 + hp)
            num = fm * torch.sum(e * delta) - torch.sum(gp * delta)
            den = fm * torch.sum(delta * delta) + torch.sum(hp * delta * delta) / 1.1 + EPS32
            alpha = float((num / den).clamp(EPS32, 1.5))
            image.index_add_(0, sub, alpha * delta)
            err[sub] = e - alpha * delta
    return image.reshape(shape)


def exact(case, seed):
    op = case["op"]
    if op == "batched":
        return None  # a whole batch of reconstructions in 64 bits takes minutes
    got = _inputs(case, seed)
    if op == "prior":
        return _exact_prior(got["x"], _QPARAMS)
    if op == "denoise":
        return _exact_denoise(case, seed, got["x"])
    if op == "filter":
        V, R, C = _shape(case)
        dev = got["sino"].device
        n = torch.arange(C, device=dev)
        d = (n[:, None] - n[None, :]).double()
        taps = torch.where(d == 0, torch.full_like(d, 0.25),
                           torch.where(d.long() % 2 != 0, -1.0 / (math.pi * d) ** 2, torch.zeros_like(d)))
        sino = got["sino"].double()
        if case["kind"] == "cone":
            u = n.double() - (C - 1) / 2
            w = torch.arange(R, device=dev).double() - (R - 1) / 2
            D = _distance(case)
            sino = sino * (D / torch.sqrt(D * D + u[None, :] ** 2 + w[:, None] ** 2))
        return (math.pi / V) * (sino.reshape(-1, C) @ taps.t()).reshape(V, R, C)
    if op == "hessian":
        shape = _recon_shape(case)[0]
        pix = torch.arange(shape[0] * shape[1], device=got["weights"].device)
        return _Projector(case, pix).back(got["weights"], power=2).reshape(shape)
    proj = _Projector(case, got["pix"])
    if op == "bp":
        return proj.back(got["sino"])
    if op == "fp":
        return proj.forward(got["vox"])
    # one VCD subset update
    shape, pix = _recon_shape(case)[0], got["pix"].long()
    err, w, recon = got["err"].double(), got["weights"].double(), got["recon"].double()
    fm = float(np.float32(got["fm"]))
    gf = -fm * proj.back(w * err)
    hf = fm * got["hess"].double()[pix]
    grad, hess = _prior_grad_hess(recon.reshape(shape), _QPARAMS)
    gp, hp = grad.reshape(recon.shape)[pix], hess.reshape(recon.shape)[pix]
    delta = -(gf + gp) / (hf + hp)
    ds = proj.forward(delta)
    num = fm * torch.sum(w * err * ds) - torch.sum(gp * delta)
    den = fm * torch.sum(w * ds * ds) + 0.5 * torch.sum(hp * delta * delta) + EPS32
    alpha = (num / den).clamp(EPS32, 1.5)
    out = recon.clone()
    out.index_add_(0, pix, alpha * delta)
    stats = torch.stack([alpha, torch.sum((alpha * delta).abs()), num, den])
    return {"recon": out, "err": err - alpha * ds, "stats": stats}
