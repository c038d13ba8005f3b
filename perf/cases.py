"""The work that users of this framework have it do, as timed and checked cases.

Each case goes through the public entry points on the sizes of the repository's
own workloads: training steps (the fused trainer on static and dynamic scans,
mixed precision and plain fp32, the continuous-scan step, and the module loop
of QuadCubes), the module's forward and backward at loose points, the queries
(slice, volume, re-projection) and the ray sampler.

``exact`` restates a case in fp64 with plain torch on the GPU: the hash-grid
encoding (positions rounded to fp32 as the encoding defines them), the MLP, the
line integral, the loss, their gradients and Adam.
"""
import math

import torch

from nect_b200.config import HashEncoderConfig, MLPNetConfig, ModelConfig, get_model
from nect_b200.quadcubes import ModuleTrainer
from nect_b200.sampling import Geometry, ct_sampling
from nect_b200.serving import query_points, reproject, slice_items, volume_items
from nect_b200.trainer import RayBatch, Trainer, Workspace, scan_step

DEV = "cuda"
STEP_COUNT = 500          # Adam steps a training state has behind it
LR, BETAS, EPS = 1e-3, (0.9, 0.999), 1e-8
PRIMES = (1, 2654435761, 805459861, 2246822519)

# The models: the benchmark's static and dynamic grids, and the defaults of reconstruct().
MODELS = {
    "static": dict(model="hash_grid", dims=3, levels=16, features=2, base=16, hidden=2, width=64, act="ReLU",
                   out_act="Softplus"),
    "dynamic": dict(model="hash_grid_4d", dims=4, levels=16, features=2, base=16, hidden=2, width=64, act="ReLU",
                    out_act="Softplus"),
    "large": dict(model="hash_grid_4d", dims=4, levels=16, features=4, base=16, hidden=3, width=64, act="ReLU",
                  out_act="Softplus"),
    "static_default": dict(model="hash_grid", dims=3, levels=19, features=4, base=8, hidden=6, width=64,
                           act="LeakyReLU", out_act="ReLU"),
    "quadcubes": dict(model="quadcubes", dims=3, levels=23, features=4, base=16, hidden=4, width=128,
                      act="LeakyReLU", out_act="None"),
}


def listed():
    return [
        # one small oblique slice of a dynamic reconstruction on a viewer's screen: the shortest call
        dict(name="slice_256", kind="slice", model="dynamic", log2=21, precision="mixed", n=256),
        # the export of a static reconstruction with the default model
        dict(name="volume_256_default", kind="volume", model="static_default", log2=21, precision="mixed", n=256),
        # the same export from an fp32 model, at an odd size
        dict(name="volume_129_fp32", kind="volume", model="static", log2=19, precision="plain_fp32", n=129),
        # a detector view of a dynamic reconstruction, as the consistency check against a projection
        dict(name="reproject_512", kind="reproject", model="dynamic", log2=21, precision="mixed", det=512, S=512,
             beam="cone"),
        # the benchmark's step: every pixel of a 512 x 512 projection, 4D cone beam
        dict(name="train_dynamic_full", kind="train", model="dynamic", log2=21, precision="mixed", det=512,
             rays=262144, S=512, beam="cone", loss="l2"),
        # the trainer's own batch in reconstruct(): 2.5 M points of random pixels, early (few points per ray)
        dict(name="train_dynamic_batch", kind="train", model="dynamic", log2=21, precision="mixed", det=256,
             rays=24999, S=100, beam="cone", loss="l1"),
        # the same batch late in a static run with the default model (19 x 4 levels, 6 hidden layers)
        dict(name="train_default_batch", kind="train", model="static_default", log2=21, precision="mixed", det=512,
             rays=4882, S=512, beam="cone", loss="l1"),
        # plain fp32 training of the static parallel-beam scan, one 128 x 128 projection
        dict(name="train_fp32_parallel", kind="train", model="static", log2=19, precision="plain_fp32", det=128,
             rays=16384, S=256, beam="parallel", loss="l2"),
        # a continuous-rotation step: four sub-angles averaged per pixel
        dict(name="scan_dynamic", kind="scan", model="dynamic", log2=21, precision="mixed", det=512, rays=8191, S=384,
             beam="cone", loss="l2", sub=4),
        # the reference's default dynamic model through the module loop, 2.5 M points (low quality's 2^19 entries)
        dict(name="train_quadcubes", kind="quadcubes", model="quadcubes", log2=19, precision="mixed", det=512,
             rays=4882, S=512, beam="cone", loss="l1"),
        # the module itself in a user's own training loop: model(points, t) and its backward
        dict(name="module_backward", kind="module_backward", model="dynamic", log2=21, precision="mixed", n=300007),
        # the drop-in sampler feeding such a loop: 5 M points
        dict(name="sample_5M", kind="sample", det=512, rays=9765, S=512, beam="cone"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["slice", "volume", "reproject", "train", "train", "train", "scan", "quadcubes",
                       "module_forward", "module_backward", "sample"])
    beam = rng.choice(["cone", "cone", "parallel", "cylinder"])
    if kind == "sample":
        S = _log_int(rng, 32, 1024)
        return dict(kind=kind, det=512, rays=_log_int(rng, 100, min(262144, 20_000_000 // S)), S=S, beam=beam)
    if kind == "quadcubes":
        S = _log_int(rng, 64, 512)
        return dict(kind=kind, model="quadcubes", log2=rng.choice([17, 19]), precision=rng.choice(["mixed", "mixed",
                    "plain_fp32"]), det=512, rays=_log_int(rng, 200, 2_500_000 // S), S=S, beam=beam,
                    loss=rng.choice(["l1", "l2"]))
    model = rng.choice(["static", "dynamic", "dynamic", "large", "static_default"])
    precision = rng.choice(["mixed", "mixed", "plain_fp32"])
    if kind == "scan":
        model = rng.choice(["static", "dynamic"])
    case = dict(kind=kind, model=model, log2=rng.choice([17, 19, 20, 21] if MODELS[model]["features"] == 2
                                                        else [17, 19, 20]), precision=precision)
    deep = MODELS[model]["hidden"] > 2 or MODELS[model]["features"] > 2
    if kind in ("slice", "volume"):
        top = {"slice": 1024, "volume": 256 if precision == "mixed" else 160}[kind]
        return dict(case, n=_log_int(rng, 33, top))
    if kind in ("module_forward", "module_backward"):
        return dict(case, n=_log_int(rng, 1000, 400_000 if deep else 2_000_000))
    S = _log_int(rng, 50, 512)
    if kind == "reproject":
        return dict(case, det=_log_int(rng, 48, 256 if precision != "mixed" or deep else 512), S=S, beam=beam)
    points = _log_int(rng, 100_000, 2_500_000 if precision != "mixed" else (8_000_000 if deep else 60_000_000))
    det = rng.choice([256, 512])
    rays = max(64, min(det * det, points // S))
    case = dict(case, det=det, rays=rays, S=S, beam=beam, loss=rng.choice(["l1", "l2"]))
    return dict(case, rays=max(64, rays // 4), sub=rng.choice([2, 3, 4, 5])) if kind == "scan" else case


# ------------------------------------------------------------------- inputs ----
def _geometry(case):
    n, beam = case.get("det", 512), case.get("beam", "cone")
    vox = dict(nVoxel=[256] * 3, dVoxel=[1.0] * 3)
    if beam == "parallel":
        return dict(nDetector=[n, n], dDetector=[256.0 / n] * 2, mode="parallel", **vox)
    more = dict(reconstruction_mode="cylindrical") if beam == "cylinder" else {}
    return dict(nDetector=[n, n], dDetector=[512.0 / n] * 2, mode="cone", DSD=1000.0, DSO=500.0, **vox, **more)


def _config(case):
    m = MODELS[case["model"]]
    enc = HashEncoderConfig(n_levels=m["levels"], n_features_per_level=m["features"], log2_hashmap_size=case["log2"],
                            base_resolution=m["base"], finest_resolution=1024,
                            base_resolution_t=4 if m["dims"] == 4 else None)
    net = MLPNetConfig(n_hidden_layers=m["hidden"], n_neurons=m["width"], activation=m["act"],
                       output_activation=m["out_act"], include_identity=True if case["model"] == "quadcubes" else None)
    return ModelConfig(m["model"], enc, net, case["precision"])


def _layout(case):
    """Per level: (resolutions, first entry, entries, hashed), and all entries."""
    m = MODELS[case["model"]]
    scale = (1024 / m["base"]) ** (1 / (m["levels"] - 1))
    levels, off = [], 0
    for k in range(m["levels"]):
        r = int(math.floor(m["base"] * math.pow(scale, k)))
        res = [r, r, r] + ([int(math.floor(4 * math.pow(scale, k)))] if m["dims"] == 4 else [])
        verts = math.prod(v + 1 for v in res)
        hashed = verts > 1 << case["log2"]
        entries = 1 << case["log2"] if hashed else (verts + 7) // 8 * 8
        levels.append((res, off, entries, hashed))
        off += entries
    return levels, off


def _n_inputs(case):
    m = MODELS[case["model"]]
    return m["levels"] * m["features"] * (4 if case["model"] == "quadcubes" else 1) + (
        4 if case["model"] == "quadcubes" else 0)


def _shapes(case):
    m = MODELS[case["model"]]
    return [(m["width"], _n_inputs(case))] + [(m["width"], m["width"])] * (m["hidden"] - 1) + [(1, m["width"])]


def _inputs(case, seed):
    """Everything a case starts from, made on the GPU from the seed: trained-like
    tables and weights, optimizer moments, rays, points, projections."""
    g = torch.Generator(device=DEV).manual_seed(1_000_003 * (seed % 1_000_000_007) + 17)

    def rand(*shape):
        return torch.rand(*shape, device=DEV, generator=g)

    x = {"t": float(rand(1).item()), "angle": float(rand(1).item()) * 2 * math.pi}
    if case["kind"] != "sample":
        F, grids = MODELS[case["model"]]["features"], 4 if case["model"] == "quadcubes" else 1
        total = _layout(case)[1]
        x["tables"] = [torch.randn(total, F, device=DEV, generator=g) * 0.1 for _ in range(grids)]
        x["weights"] = [(rand(*s) * 2 - 1) * math.sqrt(6.0 / sum(s)) for s in _shapes(case)]
    if case["kind"] in ("module_forward", "module_backward"):
        # the points of a user's loop: consecutive samples of random rays through the unit cube
        n = case["n"]
        rays = -(-n // 300)
        a, b = rand(rays, 1, 3), rand(rays, 1, 3)
        u = (torch.arange(300, device=DEV) + 0.5).view(1, -1, 1) / 300
        x["points"] = (a + (b - a) * u).reshape(-1, 3)[:n].contiguous()
        x["dsigma"] = (rand(n) - 0.5) / n
    if case["kind"] in ("train", "scan", "quadcubes", "sample"):
        R, k, P = case["rays"], case.get("sub", 1), case["det"] ** 2
        x["perm"] = torch.randperm(P, device=DEV, generator=g)
        x["jitter"] = rand(R * k) - 0.5
        x["offset"] = torch.zeros(R * k, 2, device=DEV)
        i = torch.arange(P, device=DEV)
        smooth = torch.sin(i % case["det"] * (3.0 / case["det"])) * torch.sin(i // case["det"] * (3.0 / case["det"]))
        x["projection"] = (0.6 * smooth + 0.05 * rand(P)).float().clamp(0, 1).contiguous()
        x["sub_angles"] = [x["angle"] + 0.02 * j / max(k, 1) for j in range(k)]
    if case["kind"] in ("train", "quadcubes"):
        size = 1.0 / (case["rays"] * case["S"])
        flat = x["tables"] + (x["weights"] if case["kind"] == "quadcubes" else
                              [torch.cat([w.reshape(-1) for w in x["weights"]])])
        x["moments"] = [(torch.randn(p.shape, device=DEV, generator=g) * size,
                         (0.5 + rand(*p.shape)) * (4 * size) ** 2) for p in flat]
    if case["kind"] == "slice":
        q = torch.linalg.qr(torch.randn(3, 3, device=DEV, generator=g).double())[0].tolist()
        x["u"], x["v"] = q[0], q[1]
    return x


def _model(case, x):
    model = get_model(_config(case), device=DEV)
    with torch.no_grad():
        if case["model"] == "quadcubes":
            for p, v in zip(model.tables, x["tables"]):
                p.copy_(v)
            for lin, v in zip(model.layers, x["weights"]):
                lin.weight.copy_(v)
        else:
            model.table.copy_(x["tables"][0])
            model.mlp.copy_(torch.cat([w.reshape(-1) for w in x["weights"]]))
            model.refresh_half()
    return model


def prepare(case, seed):
    x = _inputs(case, seed)
    state = {"case": case, "x": x}
    kind = case["kind"]
    if kind != "sample":
        state["model"] = _model(case, x)
    if kind in ("slice", "volume"):
        n = case["n"]
        state["out"] = torch.empty((n, n) if kind == "slice" else (n, n, n), device=DEV)
    if kind in ("reproject", "train", "scan", "quadcubes", "sample"):
        geo = state["geometry"] = Geometry(**_geometry(case))
        state["c_geometry"] = geo.get_c_geometry()
    if kind in ("train", "scan", "quadcubes"):
        state["batch"] = RayBatch(perm=x["perm"], start=0, num_rays=case["rays"], points_per_ray=case["S"],
                                  angle=x["angle"], max_ray_distance_per_point=geo.max_distance_traveled / case["S"],
                                  jitter=x["jitter"], detector_offset=x["offset"], projection=x["projection"],
                                  t=x["t"])
    if kind in ("train", "quadcubes"):
        make = ModuleTrainer if kind == "quadcubes" else Trainer
        trainer = make(state["model"], geo, points_per_batch=case["rays"] * case["S"], points_per_ray=case["S"],
                       loss=case["loss"], lr=LR, betas=BETAS, eps=EPS, device=DEV)
        trainer.load_optimizer_moments(x["moments"])
        trainer.step_count = STEP_COUNT
        state["trainer"] = trainer
        state["params"] = list(state["model"].parameters())
    if kind == "scan":
        state["grads"] = [torch.zeros_like(p) for p in (state["model"].table, state["model"].mlp)]
        state["workspace"] = Workspace()
    for name in ("tables", "weights", "moments"):   # now in the model and the trainer
        x.pop(name, None)
    return state


def run(state):
    case, x, kind = state["case"], state["x"], state["case"]["kind"]
    if kind == "sample":
        geo = state["geometry"]
        return ct_sampling.sample_with_draws(x["perm"], state["c_geometry"], x["angle"], case["S"], case["rays"], 0,
                                             geo.max_distance_traveled / case["S"], True, x["jitter"], x["offset"])
    model = state["model"]
    if kind == "slice":
        query_points(model, slice_items(state["out"], state["out"].shape, x["t"], u=x["u"], v=x["v"]))
        return state["out"]
    if kind == "volume":
        query_points(model, volume_items(state["out"], state["out"].shape, x["t"]))
        return state["out"]
    if kind == "reproject":
        return reproject(model, state["geometry"], x["angle"], x["t"], case["S"])
    if kind in ("module_forward", "module_backward"):
        args = (x["points"],) + ((x["t"],) if MODELS[case["model"]]["dims"] == 4 else ())
        if kind == "module_forward":
            with torch.no_grad():
                return model(*args)
        sigma = model(*args)
        grads = torch.autograd.grad(sigma, [model.table, model.mlp], x["dsigma"].view(-1, 1))
        return {"sigma": sigma, "table": grads[0], "mlp": grads[1]}
    if kind == "scan":
        for g in state["grads"]:
            g.zero_()
        loss, y = scan_step(model, state["c_geometry"], state["batch"], x["sub_angles"],
                            state["geometry"].max_distance_traveled, *state["grads"], state["workspace"],
                            loss=case["loss"])
        return {"loss": loss, "y": y, "table": state["grads"][0], "mlp": state["grads"][1]}
    loss = state["trainer"].step(state["batch"])
    return {"loss": loss.view(1), "params": [p.data for p in state["params"]],
            "moments": [list(mv) for mv in state["trainer"].optimizer_moments()]}


# --------------------------------------------------------------------- work ----
def _points(case):
    """Valid points of a case (for rays: the mean share of a ray's samples that lie in the object)."""
    kind = case["kind"]
    if kind in ("module_forward", "module_backward"):
        return case["n"]
    if kind in ("slice", "volume"):
        return case["n"] ** (2 if kind == "slice" else 3)
    rays = case["det"] ** 2 if kind == "reproject" else case["rays"] * case.get("sub", 1)
    return rays * case["S"] * 0.64


def work(case):
    kind = case["kind"]
    if kind == "sample":
        return {"bytes": case["rays"] * (12.0 * case["S"] + 8 + 12 + 4), "flops": 9.0 * case["rays"] * case["S"]}
    m = MODELS[case["model"]]
    n, grids = _points(case), 4 if kind == "quadcubes" else 1
    params = float(sum(a * b for a, b in _shapes(case)))
    entries, F = float(_layout(case)[1]), m["features"]
    lerp = 2.0 * m["levels"] * F * grids * 2 ** m["dims"]
    flops = n * (2 * params + lerp)
    table = (2 if case["precision"] == "mixed" and kind != "quadcubes" else 4) * F * entries * grids
    # entries a pass cannot reach are not read: at most one per corner and point
    reach = min(1.0, n * m["levels"] * 2 ** m["dims"] / entries)
    if kind in ("train", "quadcubes"):   # forward and backward, Adam on every parameter
        return {"bytes": 24.0 * (entries * F * grids + params) + 28.0 * case["rays"], "flops": 3 * flops}
    if kind in ("scan", "module_backward"):
        io = 16.0 * n if kind == "module_backward" else 28.0 * case["rays"] * case["sub"]
        return {"bytes": table * reach + 4.0 * entries * F + io, "flops": 3 * flops}
    out = {"reproject": 4.0 * case.get("det", 0) ** 2, "module_forward": 16.0 * n}.get(kind, 4.0 * n)
    return {"bytes": table * reach + out, "flops": flops}


# -------------------------------------------------------------------- exact ----
DSO, DSD, SIDE = 500.0, 1000.0, 256.0   # source, detector and object (256^3 voxels of size 1) of _geometry


def _longest(case):
    """The longest way through the object: its diagonal across the rotation axis, tilted by a cone's opening."""
    length = math.sqrt(2) * (SIDE - 1)
    if case.get("beam") == "parallel":
        return length
    return length / math.cos(math.atan((SIDE - 1) / 2 / (DSO + length / 2)))


def _ray_points(case, angle, jitter, perm):
    """The sampler's points: (z, y, x) fp32 [R, S, 3], which samples exist [R, S], and the spacing a
    point stands for.  Poses and crossings in fp64 with the sampler's fp32 scalars."""
    S, f32, f64 = case["S"], torch.float32, torch.float64
    det, R = case["det"], jitter.numel()
    rows, cols = perm[:R] // det, perm[:R] % det
    beam = case["beam"]
    pitch = torch.tensor((SIDE if beam == "parallel" else 2 * SIDE) / det, dtype=f32, device=DEV)
    py = -((cols - (det - 1) / 2).to(f32) * pitch).to(f64)
    pz = ((rows - (det - 1) / 2).to(f32) * pitch).to(f64)
    ang = torch.tensor(angle, dtype=f32, device=DEV)
    c, s = torch.cos(ang).to(f64), torch.sin(ang).to(f64)
    if beam == "parallel":
        far = float(torch.tensor(2 * SIDE ** 2, dtype=f32).sqrt())
        a = torch.stack([torch.full_like(py, -far), py, pz], 1)
        b = torch.stack([torch.full_like(py, far), py, pz], 1)
    else:
        a = torch.tensor([-DSO, 0.0, 0.0], dtype=f64, device=DEV).expand(R, 3)
        b = torch.stack([torch.full_like(py, DSD - DSO), py, pz], 1)

    def turn(p):
        return torch.stack([c * p[:, 0] - s * p[:, 1], s * p[:, 0] + c * p[:, 1], p[:, 2]], 1)

    if beam == "cylinder":
        d = b - a
        qa = (d[:, 0] ** 2 + d[:, 1] ** 2).to(f32)
        qb = (2 * a[:, 0] * d[:, 0] + 2 * a[:, 1] * d[:, 1]).to(f32)
        qc = (a[:, 0] ** 2 + a[:, 1] ** 2 - (SIDE / 2) ** 2).to(f32)
        disc = torch.addcmul(qb * qb, qa, qc, value=-4)
        hit = disc > 0
        root = disc.clamp(min=0).sqrt()
        t0, t1 = ((-qb - root) / (2 * qa)).to(f64)[:, None], ((-qb + root) / (2 * qa)).to(f64)[:, None]
        base = torch.tensor([1.0, 1.0, 0.0], dtype=f64, device=DEV)
        s0, e0 = turn(a * base + t0 * d), turn(a * base + t1 * d)
    else:
        a, b = turn(a), turn(b)
        half, d = (SIDE - 0.5) / 2, b - a
        ta, tb = (-half - a) / d, (half - a) / d
        along = ta.isnan() | tb.isnan()   # a ray inside a face of the box: that axis does not bound it
        t0 = torch.minimum(ta, tb).masked_fill(along, -math.inf).amax(1, keepdim=True)
        t1 = torch.maximum(ta, tb).masked_fill(along, math.inf).amin(1, keepdim=True)
        hit = ((t0 <= t1) & (t0 >= 0) & (t1 <= 1)).squeeze(1)
        s0, e0 = a + t0 * d, a + t1 * d
    step = e0 - s0
    length = step.norm(dim=1, keepdim=True).to(f32).to(f64)
    maxd = float(torch.tensor(_longest(case) / S, dtype=f32))
    step = step / length * maxd / SIDE
    first = s0 / SIDE + 0.5 + jitter.to(f64)[:, None] * step
    end = e0 / SIDE + 0.5 + (step if beam != "cylinder" else 0)
    if beam == "cylinder":
        end[:, 2] = e0[:, 2]   # the sampler leaves the exit height unscaled; its breaks do not use it
    first, end = first.clamp(0, 1), end.clamp(0, 1)
    i = torch.arange(S, device=DEV, dtype=f64).view(1, S, 1)
    pos = (first[:, None] + i * step[:, None]).to(f32)
    st, en = step[:, None], end[:, None]
    if beam == "cylinder":
        past = ((st > 0) & (pos.to(f64) > en)) | ((st < 0) & (pos.to(f64) < en))
        by_x = (st[..., 0] != 0)
        out = torch.where(by_x, past[..., 0], past[..., 1]) | (pos[..., 2] < 0) | (pos[..., 2] > 1)
    else:
        eps = torch.tensor(1e-5, dtype=f32, device=DEV)
        out = (((st > 0) & ((pos - eps).to(f64) > en)) | ((st < 0) & ((pos + eps).to(f64) < en))).any(2)
    there = (out.cumsum(1) == 0) & hit[:, None]
    return pos.flip(2), there, torch.where(hit, maxd, 0.0)


def _corners(levels, log2, k, p):
    """Entries [N, 2^d] of level k's corners around points p [N, d] and their fp64 weights."""
    res, off, _, hashed = levels[k]
    r = torch.tensor(res, dtype=torch.float32, device=p.device)
    q = p * r
    c = torch.minimum(torch.floor(q), r - 1).clamp(min=0)
    f = (q - c).double()
    c = c.to(torch.int64)
    idx, wts = [], []
    for corner in range(1 << len(res)):
        e, w, stride = 0, 1.0, 1
        for a in range(len(res)):
            bit = corner >> a & 1
            v = c[:, a] + bit
            e = e ^ ((v * PRIMES[a]) & 0xFFFFFFFF) if hashed else e + v * stride
            stride *= res[a] + 1
            w = w * (f[:, a] if bit else 1 - f[:, a])
        idx.append((e & ((1 << log2) - 1) if hashed else e) + off)
        wts.append(w)
    return torch.stack(idx, 1), torch.stack(wts, 1)


class _Exact:
    """The model of a case in fp64: sigma at points and its gradients."""

    def __init__(self, case, x):
        self.case, self.m = case, MODELS[case["model"]]
        self.levels = _layout(case)[0]
        self.tables = [t.double() for t in x["tables"]]
        self.weights = [w.double().requires_grad_() for w in x["weights"]]
        self.grads = None
        self.t = x["t"]

    def grids(self, p):
        """The input of each table's grid at points p [N, 3]."""
        t = torch.full((p.shape[0], 1), self.t, dtype=torch.float32, device=DEV)
        if self.case["model"] == "quadcubes":
            return [p] + [torch.cat([p[:, c], t], 1) for c in ([1, 2], [2, 0], [0, 1])]
        return [torch.cat([p, t], 1) if self.m["dims"] == 4 else p]

    def encode(self, p):
        out = []
        for q, table in zip(self.grids(p), self.tables):
            for k in range(len(self.levels)):
                idx, w = _corners(self.levels, self.case["log2"], k, q)
                out.append((table[idx] * w[..., None]).sum(1))
        if self.case["model"] == "quadcubes":
            out.append(torch.cat([p, torch.full_like(p[:, :1], self.t)], 1).double())
        return torch.cat(out, 1)

    def mlp(self, h):
        act = {"ReLU": torch.relu, "LeakyReLU": lambda v: torch.nn.functional.leaky_relu(v, 0.01)}[self.m["act"]]
        for w in self.weights[:-1]:
            h = act(h @ w.t())
        z = (h @ self.weights[-1].t()).squeeze(1)
        return {"Softplus": torch.nn.functional.softplus, "ReLU": torch.relu, "None": lambda v: v}[self.m["out_act"]](z)

    def sigma(self, p):
        with torch.no_grad():
            return torch.cat([self.mlp(self.encode(q)) for q in p.split(1 << 19)]) if p.shape[0] else p.new_zeros(0)

    def backward(self, p, dsigma):
        """Adds the gradients of sum(dsigma * sigma(p)) to self.grads (tables, weights)."""
        if self.grads is None:
            self.grads = ([torch.zeros_like(t) for t in self.tables], [torch.zeros_like(w) for w in self.weights])
        F = self.m["features"]
        for q, g in zip(p.split(1 << 19), dsigma.split(1 << 19)):
            h = self.encode(q).requires_grad_()
            got = torch.autograd.grad(self.mlp(h), [h] + self.weights, g)
            for a, b in zip(self.grads[1], got[1:]):
                a += b
            col = 0
            for z, table in zip(self.grids(q), self.grads[0]):
                for k in range(len(self.levels)):
                    idx, w = _corners(self.levels, self.case["log2"], k, z)
                    d = got[0][:, col:col + F]
                    for c in range(idx.shape[1]):
                        table.index_add_(0, idx[:, c], w[:, c, None] * d)
                    col += F


def _exact_rays(net, case, x, loss):
    """(loss, y_pred) of a batch with dL/d(parameters) left in net.grads; loss None: y_pred alone."""
    reproj = loss is None
    P = case["det"] ** 2
    perm = torch.arange(P, device=DEV) if reproj else x["perm"]
    R, k = (P, 1) if reproj else (case["rays"], case.get("sub", 1))
    jitter = torch.zeros(P, device=DEV) if reproj else x["jitter"]
    angles = x["sub_angles"] if k > 1 else [x["angle"]]
    y = torch.zeros(R, dtype=torch.float64, device=DEV)
    chunk = max(1, (1 << 22) // case["S"])
    parts = [(j, r0, min(R, r0 + chunk)) for j in range(k) for r0 in range(0, R, chunk)]

    def rays(j, r0, r1):
        pos, there, dist = _ray_points(case, angles[j], jitter[j * R + r0:j * R + r1], perm[r0:r1])
        pos = pos.clamp(0, 1)
        keep = there & (pos != 0).any(2)
        return pos[keep], keep, dist.double() / _longest(case) / k

    for j, r0, r1 in parts:
        p, keep, scale = rays(j, r0, r1)
        full = torch.zeros(keep.shape, dtype=torch.float64, device=DEV)
        full[keep] = net.sigma(p)
        y[r0:r1] += full.sum(1) * scale
    if reproj:
        return None, y
    diff = y - x["projection"][perm[:R]].double()
    value = (diff.abs() if loss == "l1" else diff ** 2).mean()
    dy = (torch.sign(diff) if loss == "l1" else 2 * diff) / R
    for j, r0, r1 in parts:
        p, keep, scale = rays(j, r0, r1)
        net.backward(p, (dy[r0:r1] * scale)[:, None].expand(keep.shape)[keep])
    return value, y


def _adam(p, g, m, v):
    step = STEP_COUNT + 1
    m = m.double() + (g - m.double()) * (1 - BETAS[0])
    v = v.double() * BETAS[1] + (1 - BETAS[1]) * g * g
    denom = v.sqrt() / math.sqrt(1 - BETAS[1] ** step) + EPS
    return p.double() - LR / (1 - BETAS[0] ** step) * m / denom, m, v


def _query_positions(case, x):
    n = case["n"]
    if case["kind"] == "volume":
        c = [(torch.arange(n, device=DEV) + 0.5).float() / n] * 3
        return torch.stack(torch.meshgrid(*c, indexing="ij"), -1).reshape(-1, 3).float()
    u, v = (torch.tensor(x[k], dtype=torch.float64, device=DEV) for k in "uv")
    g = (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n - 0.5
    return (0.5 + g[None, :, None] * u + g[:, None, None] * v).clamp(0, 1).reshape(-1, 3).float()


def exact(case, seed):
    x, kind = _inputs(case, seed), case["kind"]
    if kind == "sample":
        pos, there, dist = _ray_points(case, x["angle"], x["jitter"], x["perm"])
        return pos.double() * there[..., None], dist.double()
    net = _Exact(case, x)
    if kind in ("slice", "volume"):
        return net.sigma(_query_positions(case, x)).view([case["n"]] * (2 if kind == "slice" else 3))
    if kind == "reproject":
        return _exact_rays(net, case, x, None)[1].view(case["det"], case["det"])
    if kind == "module_forward":
        return net.sigma(x["points"]).view(-1, 1)
    if kind == "module_backward":
        net.backward(x["points"], x["dsigma"].double())
        return {"sigma": net.sigma(x["points"]).view(-1, 1), "table": net.grads[0][0],
                "mlp": torch.cat([w.reshape(-1) for w in net.grads[1]])}
    loss, y = _exact_rays(net, case, x, case["loss"])
    tables, weights = net.grads
    if kind == "scan":
        return {"loss": loss.view(1), "y": y, "table": tables[0], "mlp": torch.cat([w.reshape(-1) for w in weights])}
    if kind == "train":
        params = [x["tables"][0], torch.cat([w.reshape(-1) for w in x["weights"]])]
        grads = [tables[0], torch.cat([w.reshape(-1) for w in weights])]
    else:
        params, grads = x["tables"] + x["weights"], tables + weights
    done = [_adam(p, g, *mv) for p, g, mv in zip(params, grads, x["moments"])]
    return {"loss": loss.detach().view(1), "params": [d[0] for d in done], "moments": [[d[1], d[2]] for d in done]}
