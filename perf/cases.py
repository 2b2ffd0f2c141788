"""Timed cases of the framework: the calls that a training run, an evaluation render and a
mesh extraction make, through the package's public entry points, from a 64-ray step to the
16384 x 128 step.

Sizes: the small and full field configurations (``field_config``), the 512 rays x 128 samples
per GPU of a default training iteration, the 16384 x 128 samples of the benchmark, 16..256
samples per ray for ragged batches, 129-point lattice blocks of the mesh extraction.
``exact`` restates each case in float64 with plain torch operations.
"""
import copy
import math

import numpy as np
import torch

from neuralangelo_gb300 import config, render, workloads
from neuralangelo_gb300.dense import EPI_RELU, EPI_SOFTPLUS, dense
from neuralangelo_gb300.encoding import HashGridEncoding
from neuralangelo_gb300.fused import CapturedStep, FusedField
from neuralangelo_gb300.inference import Inference, camera_rays
from neuralangelo_gb300.mesh import FieldSDF, MarchingCubes
from neuralangelo_gb300.model import FieldModel
from neuralangelo_gb300.sampler import HierarchicalSampler, field_sdf_fn

DEV = "cuda"
N_IMAGES, APP_DIM, N_BG, BETA, OUTSIDE = 100, 16, 32, 100.0, 1000.0


# --------------------------------------------------------------------------- the cases

def _train(name, field, rays, samples, taps, active, background=False, ragged=False, captured=True,
           importance=False):
    return dict(name=name, kind="train", field=field, rays=rays, samples=samples, taps=taps, active=active,
                background=background, ragged=ragged, captured=captured, importance=importance)


def listed():
    return [
        # the smallest training call: the small field, one CUDA graph; launches and latency
        _train("train_small_64x32", "small", 64, 32, 6, 8),
        # a default iteration on one GPU: 512 rays, 64 coarse + 64 importance samples, 4 taps,
        # background NeRF and appearance codes on, half of the levels annealed in
        _train("train_default_512x128", "full", 512, 128, 4, 8, background=True, importance=True),
        # the last three quarters of a training run: all 16 levels active, rays culled to
        # different sample counts, so that no step repeats a shape and none is captured
        _train("train_ragged_16lv", "full", 2048, 256, 6, 16, ragged=True, captured=False),
        # the benchmark's step: 2.1 M samples
        _train("train_16384x128", "full", 16384, 128, 6, 8),
        # an evaluation view during training, all levels, background behind the object
        dict(name="image_256x192", kind="image", height=192, width=256, active=16, background=True),
        # the no-grad sampling pre-pass of a default iteration
        dict(name="sampler_512", kind="sampler", rays=512, active=8),
        # one block of the mesh extraction: the lattice's SDF, then its marching cubes
        dict(name="lattice_129", kind="lattice", points=129, active=16),
        dict(name="marching_cubes_129", kind="mc", points=129),
        # the drop-in encoder under someone else's training loop: forward and backward
        dict(name="hashgrid_200k", kind="hashgrid", points=200_003, half=False),
        dict(name="hashgrid_half_1m", kind="hashgrid", points=1 << 20, half=True),
        # the drop-in rendering functions: alpha, weights, composite and their backward
        dict(name="neus_8192x128", kind="neus", rays=8192, samples=128),
        # one MLP layer: 256 x 256 with hi + lo operands (the feature layer of 65536 samples)
        dict(name="dense_softplus_65536", kind="dense", rows=65536, k=256, n=256, epi=EPI_SOFTPLUS, pair=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "train", "image", "sampler", "lattice", "mc", "hashgrid", "neus",
                       "dense"])
    if kind == "train":
        field = rng.choice(["small", "full", "full"])
        ragged = rng.random() < 0.3
        taps = rng.choice([4, 6])
        samples = rng.randint(16, 256) if ragged else rng.choice([32, 48, 96, 128, rng.randint(17, 160)])
        most = 1_000_000 // samples
        c = _train("", field, _log(rng, 48, most), samples, taps,
                   rng.randint(4, 8 if field == "small" else 14 if taps == 4 else 16),
                   background=field == "full" and rng.random() < 0.4, ragged=ragged,
                   captured=not ragged and rng.random() < 0.7, importance=not ragged and rng.random() < 0.5)
        del c["name"]
        return c
    if kind == "image":
        return dict(kind=kind, height=rng.randint(24, 192), width=rng.randint(24, 256), active=rng.randint(4, 16),
                    background=rng.random() < 0.5)
    if kind == "sampler":
        return dict(kind=kind, rays=_log(rng, 64, 16384), active=rng.randint(4, 16))
    if kind == "lattice":
        return dict(kind=kind, points=rng.randint(17, 160), active=rng.randint(4, 16))
    if kind == "mc":
        return dict(kind=kind, points=rng.randint(17, 160))
    if kind == "hashgrid":
        return dict(kind=kind, points=_log(rng, 1000, 1 << 20), half=rng.random() < 0.4)
    if kind == "neus":
        return dict(kind=kind, rays=_log(rng, 64, 16384), samples=rng.randint(16, 160))
    return dict(kind=kind, rows=_log(rng, 256, 1 << 19), k=rng.choice([128, 256, 304]), n=rng.choice([64, 128, 256]),
                epi=rng.choice([EPI_RELU, EPI_SOFTPLUS]), pair=rng.random() < 0.5)


# --------------------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV)


_blank = {}     # one unfilled model per configuration: building the table on the host takes seconds


def _model(field, seed, active, taps=6, background=False):
    """A field in the middle of its training: geometric initialisation, encoder columns and
    table of order 1e-2, at the iteration where ``active`` levels are annealed in."""
    key = (field, background)
    if key not in _blank:
        _blank[key] = FieldModel(config.field_config(field, background=background)).to(DEV)
    m = copy.deepcopy(_blank[key])
    m.cfg.sdf.gradient.taps = m.neural_sdf.cfg_sdf.gradient.taps = taps
    g = _gen(seed)
    with torch.no_grad():
        for name, p in m.named_parameters():
            if name.endswith("tcnn_encoding.params"):
                p.uniform_(-1e-2, 1e-2, generator=g)
            elif name.endswith(("weight_v", "weight")) and p.dim() == 2 and "appear" not in name:
                p.uniform_(-1.0, 1.0, generator=g).mul_(p.shape[1] ** -0.5)
            elif name.endswith("bias"):
                p.uniform_(-0.05, 0.05, generator=g)
            elif "appear" in name:
                p.normal_(generator=g)
        l0, l1 = m.neural_sdf.mlp.linears
        l0.weight_v.normal_(0.0, math.sqrt(2 / 256), generator=g)
        l0.weight_v[:, 3:].normal_(0.0, 1e-2, generator=g)
        l1.weight_v.normal_(0.0, math.sqrt(2 / 256), generator=g)
        m.neural_sdf.mlp.linear_sdf.weight.normal_(math.sqrt(math.pi / 256), 1e-4, generator=g)
        m.neural_sdf.mlp.linear_sdf.bias.fill_(-0.5)
        for lin in m.modules():
            if hasattr(lin, "weight_g"):
                lin.weight_g.copy_(lin.weight_v.norm(dim=1, keepdim=True))
    m.schedule(workloads.full_field_iteration(active))
    return m


def _rays(g, R):
    c = _randn(g, R, 3)
    c = 3.0 * c / c.norm(dim=-1, keepdim=True)
    d = -c + 0.3 * _randn(g, R, 3)
    d = d / d.norm(dim=-1, keepdim=True)
    near, far, outside = workloads.sphere_bounds(c, d)
    return c, d, near, far, outside


def _batch(case, seed):
    """A training batch of cameras on a radius-3 sphere: stratified samples, or half of them
    stratified and half gathered around a surface of radius one half, as the sampler leaves them."""
    g = _gen(seed + 1)
    R, S = case["rays"], case["samples"]
    c, d, near, far, outside = _rays(g, R)
    b = dict(center=c, ray_unit=d, far=far, outside=outside, target=_rand(g, R, 3),
             app_idx=torch.randint(0, N_IMAGES, (R,), generator=g, device=DEV))
    if case["ragged"]:
        counts = torch.randint(min(16, S), S + 1, (R,), generator=g, device=DEV)
        counts[outside[:, 0] | (_rand(g, R) < 0.3)] = 0
        offs = torch.zeros(R + 1, dtype=torch.int64, device=DEV)
        offs[1:] = counts.cumsum(0)
        ray = torch.repeat_interleave(torch.arange(R, device=DEV), counts)
        k = torch.arange(ray.numel(), device=DEV) - offs[ray]
        t = (k + _rand(g, ray.numel())) / counts[ray]
        b.update(dists=t * (far - near)[ray, 0] + near[ray, 0], ray_offsets=offs, sample_ray=ray.to(torch.int32))
    else:
        n = S // 2 if case["importance"] else S
        t = (torch.arange(n, device=DEV)[None] + _rand(g, R, n)) / n * (far - near) + near
        if case["importance"]:
            mid = -(c * d).sum(-1, keepdim=True)
            hit = mid - (mid ** 2 - 8.75).clamp(min=0).sqrt()
            close = hit + 0.05 * _randn(g, R, S - n)
            t = torch.cat([t, torch.minimum(torch.maximum(close, near), far)], dim=1).sort(dim=1).values
        b["dists"] = t
    if case["background"]:
        b["dists_bg"] = workloads.background_dists(far, N_BG, _rand(g, R, N_BG))
    return b


def _encoder(half):
    key = ("encoder", half)
    if key not in _blank:
        conf = dict(otype="HashGrid", n_levels=16, n_features_per_level=8, log2_hashmap_size=22, base_resolution=32,
                    per_level_scale=float(np.exp(np.log(64) / 15)))
        _blank[key] = HashGridEncoding(3, conf, dtype=torch.float16 if half else torch.float32).to(DEV)
    return copy.deepcopy(_blank[key])


def _camera(g, H, W):
    """A camera at distance 3 that looks at the origin: world-to-camera [R|t] and intrinsics."""
    z = _randn(g, 3)
    z = z / z.norm()
    x = torch.linalg.cross(_randn(g, 3), z)
    x = x / x.norm()
    rot = torch.stack([x, torch.linalg.cross(z, x), z])
    t = torch.tensor([[0.0], [0.0], [3.0]], device=DEV)
    f = 1.2 * max(H, W)
    intr = torch.tensor([[f, 0.0, W / 2], [0.0, f, H / 2], [0.0, 0.0, 1.0]], device=DEV)
    return torch.cat([rot, t], dim=1), intr


def prepare(case, seed):
    kind = case["kind"]
    g = _gen(seed + 1)
    if kind == "train":
        m = _model(case["field"], seed, case["active"], case["taps"], case["background"])
        b = _batch(case, seed)
        ff = FusedField(m)
        step = CapturedStep(ff, b) if case["captured"] else None
        return dict(kind=kind, model=m, batch=b, fused=ff, step=step)
    if kind == "image":
        m = _model("full", seed, case["active"], background=case["background"])
        pose, intr = _camera(g, case["height"], case["width"])
        return dict(kind=kind, inference=Inference(m), pose=pose, intr=intr, size=(case["height"], case["width"]))
    if kind == "sampler":
        m = _model("full", seed, case["active"])
        c, d, near, far, _ = _rays(g, case["rays"])
        return dict(kind=kind, sampler=HierarchicalSampler(), sdf=field_sdf_fn(m.neural_sdf), model=m,
                    args=(c, d, near, far), u=_rand(g, case["rays"], 64))
    if kind == "lattice":
        m = _model("full", seed, case["active"])
        return dict(kind=kind, sdf=FieldSDF(m.neural_sdf), model=m, axes=_axes(g, case["points"]))
    if kind == "mc":
        # the surface runs between the same lattice points whatever the seed, which sets where
        # on their edges it does: the number of triangles belongs to the size
        n = case["points"]
        xs = _axes(_gen(0), n)
        X = torch.stack(torch.meshgrid(*xs, indexing="ij"), dim=-1)
        vol = (0.5 + X.norm(dim=-1).neg() + 0.1 * torch.sin(9 * X).prod(dim=-1)) * (0.5 + _rand(g, n, n, n))
        return dict(kind=kind, mc=MarchingCubes(n, DEV), vol=vol, origin=tuple(float(a[0]) for a in xs),
                    step=float(xs[0][1] - xs[0][0]))
    if kind == "hashgrid":
        enc = _encoder(case["half"])
        with torch.no_grad():
            enc.params.uniform_(-1e-2, 1e-2, generator=g)
        return dict(kind=kind, enc=enc, x=_rand(g, case["points"], 3) * 0.5 + 0.25,
                    d=_randn(g, case["points"], enc.n_output_dims) * 1e-3)
    if kind == "neus":
        R, S = case["rays"], case["samples"]
        _, d, near, far, _ = _rays(g, R)
        dists = (torch.arange(S, device=DEV)[None] + _rand(g, R, S)) / S * (far - near) + near
        sdf = (dists - 2.5).abs() - 0.1 + 0.01 * _randn(g, R, S)
        grad = _randn(g, R, S, 3)
        grad = grad / grad.norm(dim=-1, keepdim=True) * (1 + 0.1 * _randn(g, R, S, 1))
        leaves = [t.requires_grad_() for t in (sdf, grad, _rand(g, R, S, 3), torch.full((), 3.0, device=DEV))]
        return dict(kind=kind, ray=d, dists=dists, far=far, leaves=leaves, d=_randn(g, R, 3))
    M, K, N = case["rows"], case["k"], case["n"]
    X = _randn(g, M, K)
    W = (_randn(g, N, K) * (2 / K) ** 0.5).half()
    hi = X.half()
    lo = (X - hi.float()).half() if case["pair"] else None
    out = torch.empty(M, N, device=DEV, dtype=torch.float16)
    return dict(kind="dense", X=hi, lo=lo, W=W, b=0.1 * _randn(g, N), epi=case["epi"], out=out,
                out_lo=torch.empty_like(out) if case["pair"] else None)


def _axes(g, n):
    """Lattice axes of one block: spacing of a 512-point grid over [-1, 1]."""
    lo = _rand(g, 3) * 0.4 - 0.6
    return [lo[i] + torch.arange(n, device=DEV) * (2.0 / 512) * (129.0 / n) for i in range(3)]


# --------------------------------------------------------------------------- one pass

def run(state):
    kind = state["kind"]
    if kind == "train":
        m = state["model"]
        if state["step"] is not None:
            out = state["step"].replay(state["batch"])
        else:
            m.zero_grad()
            out = state["fused"].step(state["batch"], compute_loss=False)
        return dict(rgb=out["rgb"], grads={n: p.grad for n, p in m.named_parameters()})
    if kind == "image":
        return state["inference"].render_image(state["pose"], state["intr"], *state["size"])
    if kind == "sampler":
        return state["sampler"](state["sdf"], *state["args"], u=state["u"])
    if kind == "lattice":
        return state["sdf"].lattice(*state["axes"])
    if kind == "mc":
        return list(state["mc"](state["vol"], state["origin"], state["step"]))
    if kind == "hashgrid":
        enc = state["enc"]
        enc.params.grad = None
        y = enc(state["x"])
        y.backward(state["d"])
        return [y.detach(), enc.params.grad]
    if kind == "neus":
        for t in state["leaves"]:
            t.grad = None
        sdf, grad, rgbs, s_var = state["leaves"]
        a = render.compute_neus_alphas(state["ray"], sdf, grad, state["dists"], s_var, dist_far=state["far"],
                                       progress=0.05)
        w = render.alpha_compositing_weights(a)
        rgb = render.composite(rgbs, w)
        rgb.backward(state["d"])
        return [rgb.detach(), w.detach()] + [t.grad for t in state["leaves"]]
    y = dense(state["X"], state["W"], state["b"], epi=state["epi"], out=state["out"], X_lo=state["lo"],
              out_lo=state["out_lo"])
    return [y] if state["out_lo"] is None else [y, state["out_lo"]]


# --------------------------------------------------------------------------- what a pass cannot do without

def _grid(levels=16, F=8, log2T=22, base=32, growth=None):
    """Level table of the hash grid: (scale, resolution, size, hashed) per level, in the float32
    steps that define the table's format."""
    growth = np.float32(growth or np.exp(np.log(64) / 15))
    lg = np.float32(np.log2(np.float64(growth)))
    out = []
    for lv in range(levels):
        s = np.float32(np.exp2(np.float64(np.float32(lv) * lg))) * np.float32(base) - np.float32(1)
        res = int(np.ceil(np.float64(s))) + 1
        size = min((res ** 3 + 7) // 8 * 8, 1 << log2T)
        out.append((float(s), res, size, res ** 3 > size))
    return out


def _field_grid(field):
    return _grid() if field == "full" else _grid(8, 4, 16, 16, 1.5)


def _table(field, active, evals):
    """Table values that ``evals`` evaluations can touch in the active levels."""
    F = 8 if field == "full" else 4
    return sum(min(size, 8 * evals) for _, _, size, _ in _field_grid(field)[:active]) * F


def _mlp_macs(field, active, taps):
    k0 = 3 + active * (8 if field == "full" else 4)
    h, n = (256, 4) if field == "full" else (128, 2)
    dims = [278 + (APP_DIM if field == "full" else 0)] + [h] * n + [3]
    return (1 + taps) * (k0 * 256 + 256) + 256 * 256 + sum(a * b for a, b in zip(dims, dims[1:]))


BG_MACS = 84 * 256 + 6 * 256 * 256 + 340 * 256 - 256 * 256 + 257 * 256 + (272 + APP_DIM) * 128 + 128 * 3


def work(case):
    kind = case["kind"]
    if kind == "train":
        share = 0.7 * (min(16, case["samples"]) + case["samples"]) / (2 * case["samples"]) if case["ragged"] else 1.0
        n = int(case["rays"] * case["samples"] * share)
        nb = case["rays"] * N_BG if case["background"] else 0
        touched = _table(case["field"], case["active"], n * (1 + case["taps"]))
        # table read and its gradient written in float32; distances in, colours out
        return dict(bytes=8 * touched + 4 * n + 4 * nb + 60 * case["rays"],
                    flops=6 * (n * _mlp_macs(case["field"], case["active"], case["taps"]) + nb * BG_MACS))
    if kind == "image":
        R = case["height"] * case["width"]
        evals = R * (64 + 48 + 128 * 7)
        f = R * ((64 + 48) * (3 + 8 * case["active"] + 1) * 256 + 128 * _mlp_macs("full", case["active"], 6)
                 + (N_BG * BG_MACS if case["background"] else 0))
        return dict(bytes=4 * _table("full", case["active"], evals) + 32 * R, flops=2 * f)
    if kind in ("sampler", "lattice"):
        n = case["rays"] * 112 if kind == "sampler" else case["points"] ** 3
        io = case["rays"] * (128 + 64 + 8) * 4 if kind == "sampler" else 4 * n
        # the weights and the table are handed over in float32 once and kept as float16
        return dict(bytes=2 * _table("full", case["active"], n) + io,
                    flops=2 * n * (3 + 8 * case["active"] + 1) * 256)
    if kind == "mc":
        return dict(bytes=4 * case["points"] ** 3 + 36 * 4 * case["points"] ** 2, flops=0)
    if kind == "hashgrid":
        n, el = case["points"], 2 if case["half"] else 4
        whole = sum(size for _, _, size, _ in _grid()) * 8
        return dict(bytes=n * (12 + 2 * 128 * 4) + el * _table("full", 16, n) + el * whole, flops=n * 16 * 8 * 8 * 4)
    if kind == "neus":
        return dict(bytes=case["rays"] * (case["samples"] * 4 * (1 + 1 + 3 + 3 + 1 + 1 + 3 + 3) + 40),
                    flops=case["rays"] * case["samples"] * 120)
    M, K, N = case["rows"], case["k"], case["n"]
    return dict(bytes=2 * (M * (K + N) * (2 if case["pair"] else 1) + K * N), flops=2 * M * K * N)


# --------------------------------------------------------------------------- the same in 64 bits

def _corners(x01, lv):
    """Entry indices [M, 8] and trilinear weights [M, 8] of points in [0, 1]^3 on one level."""
    scale, res, size, hashed = lv
    p = x01 * scale + 0.5
    base = p.floor()
    frac = p - base
    base = base.long()
    idx, wgt = [], []
    for c in range(8):
        bit = [(c >> i) & 1 for i in range(3)]
        x, y, z = ((base[:, i] + bit[i]) & 0xffffffff for i in range(3))
        if hashed:
            i = (x ^ (y * 2654435761 & 0xffffffff) ^ (z * 805459861 & 0xffffffff)) % size
        else:
            i = ((x + y * res + z * res * res) & 0xffffffff) % size
        w = 1.0
        for i_ in range(3):
            w = w * (frac[:, i_] if bit[i_] else 1 - frac[:, i_])
        idx.append(i)
        wgt.append(w)
    return torch.stack(idx, 1), torch.stack(wgt, 1)


def _encode(x01, tables, grid):
    """tables: per level [size, F] float64 -> [M, levels * F]."""
    out = []
    for tab, lv in zip(tables, grid):
        idx, wgt = _corners(x01, lv)
        rows = tab.index_select(0, idx.reshape(-1)).reshape(*idx.shape, -1)
        out.append((rows * wgt[..., None]).sum(1))
    return torch.cat(out, 1)


def _softplus(x, beta=1.0):
    return torch.nn.functional.softplus(x, beta=beta, threshold=40.0)


def _sh(d):
    x, y, z = d.unbind(-1)
    k1, k2, k3 = math.sqrt(3 / (4 * math.pi)), math.sqrt(15 / (4 * math.pi)), math.sqrt(5 / (16 * math.pi))
    a, b = math.sqrt(35 / (32 * math.pi)), math.sqrt(105 / (4 * math.pi))
    c, e = math.sqrt(21 / (32 * math.pi)), math.sqrt(7 / (16 * math.pi))
    f = math.sqrt(105 / (16 * math.pi))
    return torch.stack([
        torch.full_like(x, math.sqrt(1 / (4 * math.pi))), -k1 * y, k1 * z, -k1 * x,
        k2 * x * y, -k2 * y * z, k3 * (2 * z * z - x * x - y * y), -k2 * x * z, k2 / 2 * (x * x - y * y),
        -a * y * (3 * x * x - y * y), b * x * y * z, -c * y * (4 * z * z - x * x - y * y),
        e * z * (2 * z * z - 3 * x * x - 3 * y * y), -c * x * (4 * z * z - x * x - y * y), f * z * (x * x - y * y),
        -a * x * (x * x - 3 * y * y)], dim=-1)


class _Exact:
    """The field of a model's parameters in float64, the table as one leaf per active level."""

    def __init__(self, model, case):
        self.field = case.get("field", "full")
        self.grid = _field_grid(self.field)
        self.F = 8 if self.field == "full" else 4
        self.active = case["active"]
        self.taps = case.get("taps", 6)
        growth = math.exp(math.log(64) / 15) if self.field == "full" else 1.5
        base = 32 if self.field == "full" else 16
        self.eps = 1.0 / (int(math.floor(base * growth ** (self.active - 1))) + 1)
        self.params = {n: p.detach() for n, p in model.named_parameters()}
        self.p = {n: p.double().requires_grad_() for n, p in self.params.items() if not n.endswith("encoding.params")}
        flat, at, self.tables = self.params["neural_sdf.tcnn_encoding.params"], 0, []
        for lv in self.grid[:self.active]:
            n = lv[2] * self.F
            self.tables.append(flat[at:at + n].double().reshape(-1, self.F).requires_grad_())
            at += n
        iteration = 5000 + self.active * 5000
        self.anneal = min(iteration / 500000 / 0.1, 1.0)
        self.w_curv = 5e-4 / growth ** (self.active - 1)

    def linear(self, name, x):
        p = self.p
        if name + ".weight_v" in p:
            v = p[name + ".weight_v"]
            w = v * (p[name + ".weight_g"] / v.norm(dim=1, keepdim=True))
        else:
            w = p[name + ".weight"]
        return x @ w.t() + p[name + ".bias"]

    def hidden(self, x):
        enc = _encode((x + 2) / 4, self.tables, self.grid)
        pad = torch.zeros(x.shape[0], len(self.grid) * self.F - enc.shape[1], dtype=x.dtype, device=x.device)
        return _softplus(self.linear("neural_sdf.mlp.linears.0", torch.cat([x, enc, pad], 1)), BETA)

    def sdf(self, x):
        return self.linear("neural_sdf.mlp.linear_sdf", self.hidden(x))[:, 0]

    def geometry(self, x, outside):
        """SDF (overwritten outside), features, numerical gradient and Laplacian of points [M, 3]."""
        h = self.hidden(x)
        f0 = self.linear("neural_sdf.mlp.linear_sdf", h)[:, 0].masked_fill(outside, OUTSIDE)
        feat = _softplus(self.linear("neural_sdf.mlp.linears.1", h), BETA)
        e = self.eps
        if self.taps == 6:
            grad, lap = [], 0.0
            for i in range(3):
                step = torch.zeros(3, dtype=x.dtype, device=x.device)
                step[i] = e
                fp, fm = self.sdf(x + step), self.sdf(x - step)
                grad.append((fp - fm) / (2 * e))
                lap = lap + (fp + fm - 2 * f0) / e ** 2
            return f0, feat, torch.stack(grad, 1), lap
        e = e / math.sqrt(3)
        ks = torch.tensor([[1, -1, -1], [-1, -1, 1], [-1, 1, -1], [1, 1, 1]], dtype=x.dtype, device=x.device)
        f = [self.sdf(x + e * k) for k in ks]
        return f0, feat, sum(k * v[:, None] for k, v in zip(ks, f)) / (4 * e), (sum(f) / 2 - 2 * f0) / e ** 2

    def colour(self, x, d, grad, feat, app):
        parts = [x, _sh(d), torch.nn.functional.normalize(grad, dim=-1), feat] + ([app] if app is not None else [])
        h = torch.cat(parts, 1)
        n = 4 if self.field == "full" else 2
        for i in range(n):
            h = torch.relu(self.linear(f"neural_rgb.mlp.linears.{i}", h))
        return torch.sigmoid(self.linear(f"neural_rgb.mlp.linears.{n}", h))

    def background(self, x, d, app):
        r = x.norm(dim=-1, keepdim=True)
        q = torch.cat([x / r, 1 / r], 1)
        freq = math.pi * 2.0 ** torch.arange(10, dtype=x.dtype, device=x.device)
        s = q[..., None] * freq
        code = torch.cat([q, torch.stack([s.sin(), s.cos()], dim=-2).reshape(x.shape[0], -1)], 1)
        h = code
        for i in range(8):
            h = torch.cat([h, code], 1) if i == 4 else h
            h = self.linear(f"background_nerf.mlp_feat.linears.{i}", h)
            h = torch.relu(h) if i < 7 else h
        g = torch.cat([torch.relu(h[:, 1:]), _sh(d), app], 1)
        g = torch.relu(self.linear("background_nerf.mlp_rgb.linears.0", g))
        return torch.sigmoid(self.linear("background_nerf.mlp_rgb.linears.1", g)), _softplus(h[:, 0])

    def render(self, b, train):
        """Per-ray colour and composites, and this batch's sums of the losses."""
        d, far, dists = b["ray_unit"], b["far"][:, 0], b["dists"]
        R = d.shape[0]
        if dists.dim() == 2:
            counts = torch.full((R,), dists.shape[1], device=DEV)
            dists = dists.reshape(-1)
        else:
            counts = b["ray_offsets"][1:] - b["ray_offsets"][:-1]
        ray = torch.repeat_interleave(torch.arange(R, device=DEV), counts)
        first = counts.cumsum(0) - counts
        k = torch.arange(ray.numel(), device=DEV) - first[ray]
        last = k == counts[ray] - 1
        step = torch.where(last, far[ray], torch.cat([dists[1:], dists[:1]])) - dists
        out = b["outside"].reshape(-1)[ray]
        x, dr = b["center"][ray] + d[ray] * dists[:, None], d[ray]
        f0, feat, grad, lap = self.geometry(x, out)
        app = self.p["appear_embed.weight"][b["app_idx"]][ray] if "appear_embed.weight" in self.p else None
        rgbs = self.colour(x, dr, grad, feat, app)
        cos = (dr * grad).sum(-1)
        ic = -(torch.relu(0.5 - 0.5 * cos) * (1 - self.anneal) + torch.relu(-cos) * self.anneal)
        s = self.p["s_var"].exp()
        prev, nxt = torch.sigmoid((f0 - ic * step / 2) * s), torch.sigmoid((f0 + ic * step / 2) * s)
        alpha = ((prev - nxt) / (prev + 1e-5)).clamp(0, 1)

        def padded(v, width=int(counts.max())):
            full = torch.zeros(R, width, *v.shape[1:], dtype=v.dtype, device=DEV)
            return full.index_put((ray, k), v)

        alpha, rgbs, dist, grads = padded(alpha), padded(rgbs), padded(dists), padded(grad)
        n_obj = alpha.shape[1]
        if "dists_bg" in b:
            t = b["dists_bg"]
            xb = (b["center"][:, None] + d[:, None] * t[..., None]).reshape(-1, 3)
            db = d[:, None].expand(-1, t.shape[1], -1).reshape(-1, 3)
            ab = self.p["appear_embed_outside.weight"][b["app_idx"]].repeat_interleave(t.shape[1], 0)
            cb, sigma = self.background(xb, db, ab)
            gap = torch.cat([t[:, 1:], torch.full_like(t[:, :1], 1e10)], 1) - t
            alpha = torch.cat([alpha, 1 - torch.exp(-sigma.reshape(t.shape) * gap)], 1)
            rgbs = torch.cat([rgbs, cb.reshape(R, -1, 3)], 1)
            dist = torch.cat([dist, t], 1)
        front = torch.cumprod(torch.cat([torch.ones_like(alpha[:, :1]), 1 - alpha[:, :-1]], 1), 1)
        w = alpha * front
        rgb = (w[..., None] * rgbs).sum(1)
        if not train:
            wo = w[:, :n_obj]
            return dict(rgb=rgb, opacity=wo.sum(1, keepdim=True), gradient=(wo[..., None] * grads).sum(1),
                        dist=(w * dist).sum(1, keepdim=True))
        inside = (~out).double()
        sums = ((rgb - b["target"]).abs().sum(), ((grad.norm(dim=-1) - 1) ** 2 * inside).sum(),
                (lap.abs() * inside).sum())
        return rgb, sums


def _double(b):
    return {k: v.double() if v.is_floating_point() else v for k, v in b.items()}


def _exact_train(case, seed):
    m = _model(case["field"], seed, case["active"], case["taps"], case["background"])
    ex, b = _Exact(m, case), _double(_batch(case, seed))
    R, ns = case["rays"], b["dists"].numel()
    # rays at a time, so that the float64 activations fit
    chunk = max(1, 32768 * 7 // (1 + case["taps"]) // case["samples"])
    rgb = torch.empty(R, 3, dtype=torch.float64, device=DEV)
    for i in range(0, R, chunk):
        part = {k: v[i:i + chunk] for k, v in b.items() if k not in ("ray_offsets", "sample_ray", "dists")}
        if case["ragged"]:
            o = b["ray_offsets"][i:i + chunk + 1]
            part.update(ray_offsets=o - o[0], dists=b["dists"][int(o[0]):int(o[-1])])
            if part["dists"].numel() == 0:
                rgb[i:i + chunk] = 0
                continue
        else:
            part["dists"] = b["dists"][i:i + chunk]
        out, (l1, eik, curv) = ex.render(part, True)
        (l1 / R + 0.1 * eik / ns + ex.w_curv * curv / ns).backward()
        rgb[i:i + chunk] = out.detach()
    grads = {n: (p.grad if p.grad is not None else torch.zeros_like(p)) for n, p in ex.p.items()}
    name = "neural_sdf.tcnn_encoding.params"
    flat = torch.zeros(m.get_parameter(name).numel(), dtype=torch.float64, device=DEV)
    at = 0
    for t in ex.tables:
        flat[at:at + t.numel()] = t.grad.reshape(-1)
        at += t.numel()
    grads[name] = flat
    return dict(rgb=rgb, grads=grads)


def _pdf(bins, w, n):
    pdf = w / w.sum(-1, keepdim=True).clamp(min=1e-12)
    cdf = torch.cat([torch.zeros_like(pdf[:, :1]), pdf.cumsum(-1)], -1)
    u = ((torch.arange(n, dtype=bins.dtype, device=DEV) + 0.5) / n).expand(bins.shape[0], n).contiguous()
    hi = torch.searchsorted(cdf, u, right=True)
    lo, hi = (hi - 1).clamp(min=0), hi.clamp(max=cdf.shape[1] - 1)
    c0, c1 = cdf.gather(1, lo), cdf.gather(1, hi)
    b0, b1 = bins.gather(1, lo), bins.gather(1, hi)
    return b0 + (u - c0) / (c1 - c0 + 1e-8) * (b1 - b0)


def _exact_dists(ex, c, d, near, far, u):
    """64 stratified distances and four rounds of 16 drawn from the NeuS weights."""
    t = (torch.arange(64, device=DEV)[None] + u) / 64 * (far - near) + near

    def sdf(t):
        return ex.sdf((c[:, None] + d[:, None] * t[..., None]).reshape(-1, 3)).reshape(t.shape)

    f = sdf(t)
    for h in range(4):
        gap = t[:, 1:] - t[:, :-1]
        mid = (f[:, 1:] + f[:, :-1]) / 2
        cos = (f[:, 1:] - f[:, :-1]) / (gap + 1e-5)
        cos = torch.minimum(torch.cat([torch.zeros_like(cos[:, :1]), cos[:, :-1]], 1), cos)
        s = 64.0 * 2 ** h
        prev, nxt = torch.sigmoid((mid - cos * gap / 2) * s), torch.sigmoid((mid + cos * gap / 2) * s)
        a = ((prev - nxt) / (prev + 1e-5)).clamp(0, 1)
        w = a * torch.cumprod(torch.cat([torch.ones_like(a[:, :1]), 1 - a[:, :-1]], 1), 1)
        fine = _pdf(t, w, 16)
        both = torch.cat([t, fine], 1)
        order = both.argsort(dim=1, stable=True)
        if h < 3:
            f = torch.cat([f, sdf(fine)], 1).gather(1, order)
        t = both.gather(1, order)
    return t


@torch.no_grad()
def _exact_image(case, seed):
    H, W = case["height"], case["width"]
    ex = _Exact(_model("full", seed, case["active"], background=case["background"]), case)
    pose, intr = _camera(_gen(seed + 1), H, W)
    center, ray = (v.double() for v in camera_rays(pose.double(), intr.double(), H, W))
    unit = ray / ray.norm(dim=-1, keepdim=True)
    near, far, outside = workloads.sphere_bounds(center, unit)
    parts = []
    for i in range(0, H * W, 256):
        c, d, n, f, o = (v[i:i + 256] for v in (center, unit, near, far, outside))
        b = dict(center=c, ray_unit=d, far=f, outside=o, dists=_exact_dists(ex, c, d, n, f, 0.5),
                 app_idx=torch.zeros(c.shape[0], dtype=torch.long, device=DEV))
        if case["background"]:
            b["dists_bg"] = workloads.background_dists(f, N_BG).double()
        parts.append(ex.render(b, False))
    out = {k: torch.cat([p[k] for p in parts]) for k in parts[0]}
    normal = -out["gradient"] @ pose[:, :3].double().t()
    depth = out["dist"] / ray.norm(dim=-1, keepdim=True)
    maps = dict(rgb_map=out["rgb"], opacity_map=out["opacity"], depth_map=depth, normal_map=normal)
    return {k: v.t().reshape(-1, H, W) for k, v in maps.items()}


def exact(case, seed):
    kind = case["kind"]
    s = None
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "image":
        return _exact_image(case, seed)
    if kind in ("sampler", "lattice"):
        g = _gen(seed + 1)
        ex = _Exact(_model("full", seed, case["active"]), case)
        with torch.no_grad():
            if kind == "sampler":
                c, d, near, far, _ = (v.double() for v in _rays(g, case["rays"]))
                u = _rand(g, case["rays"], 64).double()
                return torch.cat([_exact_dists(ex, *(v[i:i + 1024] for v in (c, d, near, far, u)))
                                  for i in range(0, case["rays"], 1024)])
            xs = [a.double() for a in _axes(g, case["points"])]
            X = torch.stack(torch.meshgrid(*xs, indexing="ij"), dim=-1).reshape(-1, 3)
            return -torch.cat([ex.sdf(p) for p in X.split(1 << 17)]).reshape([case["points"]] * 3)
    if kind == "mc":
        return None          # vertices come in an order of the kernel's own
    s = prepare(case, seed)
    if kind == "hashgrid":
        params, x, d = s["enc"].params.detach(), s["x"].double(), s["d"].double()
        grid, tables, at = _grid(), [], 0
        for lv in grid:
            tables.append(params[at:at + lv[2] * 8].double().reshape(-1, 8).requires_grad_())
            at += lv[2] * 8
        ys = []
        for p, q in zip(x.split(1 << 17), d.split(1 << 17)):
            y = _encode(p, tables, grid)
            y.backward(q)
            ys.append(y.detach())
        return [torch.cat(ys), torch.cat([t.grad.reshape(-1) for t in tables])]
    if kind == "neus":
        sdf, grad, rgbs, s_var = (t.detach().double().requires_grad_() for t in s["leaves"])
        d, dists, far = s["ray"].double(), s["dists"].double(), s["far"].double()
        cos = (d[:, None] * grad).sum(-1)
        ic = -(torch.relu(0.5 - 0.5 * cos) * 0.5 + torch.relu(-cos) * 0.5)
        step = torch.cat([dists[:, 1:], far], 1) - dists
        k = s_var.exp()
        prev, nxt = torch.sigmoid((sdf - ic * step / 2) * k), torch.sigmoid((sdf + ic * step / 2) * k)
        a = ((prev - nxt) / (prev + 1e-5)).clamp(0, 1)
        w = a * torch.cumprod(torch.cat([torch.ones_like(a[:, :1]), 1 - a[:, :-1]], 1), 1)
        rgb = (w[..., None] * rgbs).sum(1)
        rgb.backward(s["d"].double())
        return [rgb.detach(), w.detach()[..., None]] + [t.grad for t in (sdf, grad, rgbs, s_var)]
    x = s["X"].double() + (s["lo"].double() if s["lo"] is not None else 0.0)
    y = x @ s["W"].double().t() + s["b"].double()
    y = torch.relu(y) if case["epi"] == EPI_RELU else _softplus(y, BETA)
    hi = y.half().double()
    return [y] if not case["pair"] else [hi, y - hi]
