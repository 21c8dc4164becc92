"""Timed cases: the work a user of voxneus_b200 has it do, through its public entry points.

Training steps, inference renders (a small request, a whole view), a differentiable render inside a
user's own training loop, SDF and normal queries (scattered points, a lattice, with gradients), the
appearance modules, compositing of given samples, and the active-vertex regularizers. Every input is
made on the GPU from a seed; `exact` restates each path in float64 with plain torch operations.
"""

import math

import torch
import torch.nn.functional as F

from voxneus_b200 import ops, regularization, rendering, training
from voxneus_b200.models import DenseSDFGrid, RadianceHashGrid, RadianceMLP, SphericalHarmonicsEmbedder, VoxNeuS

DEV = "cuda"
LO, HI = (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0)
STEP0 = 5009  # past the trainer's 5000-step s warm-up, as most of a 40k-step run is
W_EIK, W_CURV, BAND = 0.1, 5e-4, 3.0


def listed():
    return [
        # the training-throughput workload: 256^3 grid, 8192 rays a step
        {"name": "train_256", "kind": "train", "res": 256, "rays": 8192, "coarse": 64, "fine": 64},
        # the plain training configuration: 64^3 grid, 2048 rays a step
        {"name": "train_64", "kind": "train", "res": 64, "rays": 2048, "coarse": 64, "fine": 64},
        # the smallest render request of the serving mix
        {"name": "render_small", "kind": "render", "res": 256, "rays": 4096, "coarse": 64, "fine": 64},
        # the largest: a whole 800x600 view
        {"name": "render_view", "kind": "render", "res": 256, "rays": 480000, "coarse": 64, "fine": 64},
        # the fused render inside a user's own loop: every output returned, autograd, ragged sizes
        {"name": "render_grad", "kind": "render_grad", "res": 96, "rays": 1021, "coarse": 48, "fine": 32},
        # the smallest query of the serving mix, with an odd count
        {"name": "query_small", "kind": "query", "res": 256, "points": 65537},
        # the large-grid query: 2^24 scattered points of a 512^3 grid
        {"name": "query_large", "kind": "query", "res": 512, "points": 1 << 24},
        # a loss on queried SDF values and normals, differentiated to the grid
        {"name": "query_grad", "kind": "query_grad", "res": 128, "points": 300007},
        # the large-grid lattice: SDF and normals at 320^3 points of a 512^3 grid
        {"name": "lattice", "kind": "lattice", "res": 512, "side": 320},
        # the appearance modules on their own, coarse-to-fine levels still opening, forward and backward
        {"name": "appearance", "kind": "appearance", "points": 200003, "levels": 10.5},
        # compositing of a caller's samples, longer rays than the renderer's own, forward and backward
        {"name": "composite", "kind": "composite", "rays": 4099, "samples": 256},
        # active vertices of a batch's corners and both closed-form regularizers on the list
        {"name": "regularize", "kind": "regularize", "res": 256, "points": 262144},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "render", "render", "render_grad", "query", "query", "query_grad", "lattice",
                       "appearance", "composite", "regularize"])
    coarse, fine = rng.choice([(64, 64), (64, 64), (64, 64), (32, 32), (64, 32), (48, 48), (40, 20)])
    if kind == "train":
        return {"kind": kind, "res": rng.choice([64, 96, 128, 192, 256, rng.randint(60, 256)]),
                "rays": _log(rng, 512, 8192), "coarse": coarse, "fine": fine}
    if kind == "render":
        return {"kind": kind, "res": rng.choice([96, 128, 256, rng.randint(60, 256)]), "rays": _log(rng, 1000, 480000),
                "coarse": coarse, "fine": fine}
    if kind == "render_grad":
        return {"kind": kind, "res": rng.randint(32, 160), "rays": _log(rng, 200, 4096), "coarse": coarse, "fine": fine}
    if kind == "query":
        return {"kind": kind, "res": rng.choice([128, 256, 512, rng.randint(64, 512)]),
                "points": _log(rng, 1 << 14, 1 << 24)}
    if kind == "query_grad":
        return {"kind": kind, "res": rng.randint(64, 256), "points": _log(rng, 20000, 2000000)}
    if kind == "lattice":
        return {"kind": kind, "res": rng.choice([256, 512, rng.randint(96, 512)]), "side": rng.randint(64, 320)}
    if kind == "appearance":
        return {"kind": kind, "points": _log(rng, 10000, 1000000), "levels": rng.choice([16.0, round(rng.uniform(4, 16), 2)])}
    if kind == "composite":
        return {"kind": kind, "rays": _log(rng, 500, 8192), "samples": rng.randint(32, 300)}
    return {"kind": kind, "res": rng.choice([96, 128, 256, rng.randint(64, 256)]), "points": _log(rng, 20000, 262144)}


# ---------------------------------------------------------------------------------- inputs ----


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rand(g, *shape, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(*shape, device=DEV, generator=g)


def _grid(res, g, noise):
    """A union of 4 spheres and 4 boxes as an SDF on a res^3 lattice, with a little noise."""
    ax = torch.linspace(-1.0, 1.0, res, device=DEV)
    c = _rand(g, 8, 3, lo=-0.5, hi=0.5).tolist()
    r = _rand(g, 8, 3, lo=0.1, hi=0.28).tolist()
    f = torch.empty(res, res, res, device=DEV)
    for i0 in range(0, res, 64):
        x, y, z = ax[i0:i0 + 64].view(-1, 1, 1), ax.view(1, -1, 1), ax.view(1, 1, -1)
        best = None
        for k in range(8):
            q = (x - c[k][0], y - c[k][1], z - c[k][2])
            if k % 2 == 0:
                fk = (q[0] ** 2 + q[1] ** 2 + q[2] ** 2).sqrt() - r[k][0]
            else:
                h = [q[a].abs() - r[k][a] for a in range(3)]
                out = (h[0].clamp(min=0) ** 2 + h[1].clamp(min=0) ** 2 + h[2].clamp(min=0) ** 2).sqrt()
                fk = out + torch.maximum(torch.maximum(h[0], h[1]), h[2]).clamp(max=0)
            best = fk if best is None else torch.minimum(best, fk)
        f[i0:i0 + 64] = best
    f += noise * torch.randn(f.shape, device=DEV, generator=g)
    return f.reshape(1, 1, res, res, res)


def _view_frame(el, az):
    pos = torch.tensor([3 * math.cos(el) * math.cos(az), 3 * math.cos(el) * math.sin(az), 3 * math.sin(el)],
                       dtype=torch.float64)
    fwd = -pos / pos.norm()
    right = torch.linalg.cross(fwd, torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64))
    right = right / right.norm()
    down = torch.linalg.cross(fwd, right)
    return pos, torch.stack([right, down, fwd], 1)


def _rays(n, g, scattered):
    """800x600 pinhole rays towards the origin: random pixels of 64 hemisphere cameras (a training
    batch), or n consecutive pixels of one camera (a render request)."""
    n_cams = 64 if scattered else 1
    spin = float(_rand(g, 1))
    frames = [_view_frame(math.radians(5 + 80 * ((c + spin) / n_cams)), 2 * math.pi * ((c * 0.618034 + spin) % 1.0))
              for c in range(n_cams)]
    pos = torch.stack([p for p, _ in frames]).float().to(DEV)
    rot = torch.stack([m for _, m in frames]).float().to(DEV)
    if scattered:
        cam = torch.randint(0, n_cams, (n,), device=DEV, generator=g)
        pix = torch.randint(0, 800 * 600, (n,), device=DEV, generator=g)
    else:
        cam = torch.zeros(n, dtype=torch.long, device=DEV)
        pix = (torch.arange(n, device=DEV) + (800 * 600 - n) // 2) % (800 * 600)
    px, py = (pix % 800).float() + 0.5, (pix // 800).float() + 0.5
    v = torch.stack([(px - 400) / 700, (py - 300) / 700, torch.ones_like(px)], -1)
    d = torch.einsum("nij,nj->ni", rot[cam], v)
    return pos[cam].contiguous(), (d / d.norm(dim=-1, keepdim=True)).contiguous()


def _mlp_weights(g):
    """The module's own initialisation (Kaiming-uniform weights) with small biases, from the seed."""
    b0, b1 = math.sqrt(6 / 51), math.sqrt(6 / 64)
    return (_rand(g, 64, 51, lo=-b0, hi=b0), _rand(g, 64, lo=-0.1, hi=0.1), _rand(g, 3, 64, lo=-b1, hi=b1),
            _rand(g, 3, lo=-0.1, hi=0.1))


def _inputs(case, seed):
    """What the case's path is given, as plain tensors."""
    g, k = _gen(seed), case["kind"]
    x = {}
    if k in ("train", "render", "render_grad"):
        x["grid"] = _grid(case["res"], g, 0.01 if case["res"] <= 96 else 0.003)
        x["emb"] = _rand(g, 16, 1 << 19, 2, lo=-1e-2, hi=1e-2)
        x["mlp"] = _mlp_weights(g)
        x["o"], x["d"] = _rays(case["rays"], g, k != "render")
        x["target"] = _rand(g, case["rays"], 3)
        if k == "render_grad":
            n, per = case["rays"], case["fine"] // 4
            x["randoms"] = (_rand(g, n, case["coarse"]), _rand(g, 4, n, per))
    elif k in ("query", "query_grad"):
        x["grid"] = _grid(case["res"], g, 0.003)
        x["pts"] = _rand(g, case["points"], 3, lo=-1.0, hi=1.0)
        if k == "query_grad":
            x["w"] = torch.randn(case["points"], 1, device=DEV, generator=g)
            x["wn"] = torch.randn(case["points"], 3, device=DEV, generator=g)
    elif k == "lattice":
        x["grid"] = _grid(case["res"], g, 0.003)
    elif k == "appearance":
        n = case["points"]
        x["emb"] = _rand(g, 16, 1 << 19, 2, lo=-1e-2, hi=1e-2)
        x["mlp"] = _mlp_weights(g)
        x["pts"] = _rand(g, n, 3)
        x["dirs"] = F.normalize(torch.randn(n, 3, device=DEV, generator=g), dim=-1)
        x["normals"] = F.normalize(torch.randn(n, 3, device=DEV, generator=g), dim=-1)
        x["w"] = torch.randn(n, 3, device=DEV, generator=g)
    elif k == "composite":
        n, s = case["rays"], case["samples"]
        z = 2.0 + 2.0 * (torch.arange(s, device=DEV) + _rand(g, n, s)) / s
        x["z"], x["dists"] = z, torch.cat([z[:, 1:] - z[:, :-1], z[:, -1:] - z[:, -2:-1]], -1)
        hit = _rand(g, n, 1, lo=2.4, hi=4.4)  # some rays miss
        x["sdf"] = (0.6 * (hit - z) + 0.01 * torch.randn(n, s, device=DEV, generator=g)).unsqueeze(-1)
        x["dirs"] = F.normalize(torch.randn(n, 3, device=DEV, generator=g), dim=-1)
        x["normals"] = F.normalize(-x["dirs"][:, None] + 0.5 * torch.randn(n, s, 3, device=DEV, generator=g), dim=-1)
        x["colors"] = _rand(g, n, s, 3)
        x["pts"] = (-3.0 * x["dirs"])[:, None] + x["dirs"][:, None] * z[..., None]
        x["w"] = torch.randn(n, 3, device=DEV, generator=g)
        x["wd"] = torch.randn(n, 1, device=DEV, generator=g)
    else:
        res, n = case["res"], case["points"]
        x["grid"] = _grid(res, g, 0.003)
        # corners of sample cells that crowd around the surface, as a batch's do
        p = _rand(g, 4 * n, 3, lo=-0.95, hi=0.95)
        c = (p * 0.5 + 0.5) * (res - 1)
        f = x["grid"][0, 0][tuple(c.round().long().unbind(-1))]
        c = c[torch.argsort(f.abs() + 0.3 * _rand(g, 4 * n))[:n]].floor().long()
        off = torch.tensor([[a, b, e] for a in (0, 1) for b in (0, 1) for e in (0, 1)], device=DEV)
        x["corners"] = (c[:, None] + off).contiguous()
    return x


def _set_mlp(mlp, w):
    with torch.no_grad():
        for p, v in zip((mlp.net[0].weight, mlp.net[0].bias, mlp.net[2].weight, mlp.net[2].bias), w):
            p.copy_(v)


def _model(case, x):
    m = VoxNeuS(grid_res=case["res"]).to(DEV)
    with torch.no_grad():
        m.sdf_grid.grid.copy_(x["grid"])
        m.radiance_hash.encoder.embeddings.copy_(x["emb"])
    _set_mlp(m.radiance_mlp, x["mlp"])
    return m


def _sdf_grid(x, res):
    s = DenseSDFGrid(resolution=res, init_mode="zero").to(DEV)
    with torch.no_grad():
        s.grid.copy_(x["grid"])
    return s


def prepare(case, seed):
    x, k = _inputs(case, seed), case["kind"]
    st = {"case": case, "x": x}
    if k in ("train", "render", "render_grad"):
        st["model"] = _model(case, x)
        st["sampler"] = rendering.RaySampler(case["coarse"], case["fine"], perturb=k != "render")
        del x["grid"], x["emb"]
    if k == "train":
        # Learning rates of zero: the optimizers run in full, but every pass meets the same weights, so
        # that passes can be repeated and compared. The first steps are eager, then the step is a graph.
        st["trainer"] = training.FusedTrainer(st["model"], st["sampler"], w_eik=W_EIK, w_curv=W_CURV, band_voxels=BAND,
                                              lr_sdf=0.0, lr_hash=0.0, lr_mlp=0.0, lr_variance=0.0, cuda_graph=True)
        torch.manual_seed(seed)
        for i in range(3):
            st["trainer"].step(x["o"], x["d"], x["target"], step=STEP0 + i)
        st["step"] = STEP0 + 3
        torch.manual_seed(seed)  # the sampler's uniforms of the passes to come
    elif k in ("query", "query_grad", "lattice"):
        st["sdf"] = _sdf_grid(x, case["res"])
        del x["grid"]
    elif k == "appearance":
        st["hash"] = RadianceHashGrid().to(DEV)
        st["sh"] = SphericalHarmonicsEmbedder()
        st["mlp"] = RadianceMLP().to(DEV)
        with torch.no_grad():
            st["hash"].encoder.embeddings.copy_(x["emb"])
        _set_mlp(st["mlp"], x["mlp"])
        x["normals"].requires_grad_()
        del x["emb"]
    elif k == "composite":
        for n in ("colors", "sdf", "normals"):
            x[n].requires_grad_()
        x["s"] = torch.tensor(64.0, device=DEV, requires_grad=True)
    elif k == "regularize":
        st["res"] = [case["res"]] * 3
        st["eps"] = torch.full((3,), 2.0 / (case["res"] - 1), device=DEV)
    return st


def _take(p):
    g, p.grad = p.grad, None
    return g


def _model_params(m):
    n = m.radiance_mlp.net
    return {"grid": m.sdf_grid.grid, "emb": m.radiance_hash.encoder.embeddings, "v": m.variance_net.variance,
            "W0": n[0].weight, "b0": n[0].bias, "W1": n[2].weight, "b1": n[2].bias}


def run(st):
    x, k = st["x"], st["case"]["kind"]
    if k == "train":
        out = st["trainer"].step(x["o"], x["d"], x["target"], step=st["step"])
        st["step"] += 1
        return {"loss": out["loss_rgb"], "eik": out["loss_eik"], "curv": out["loss_curv"], "n_active": out["n_active"],
                "rgb": out["rgb"], "grad": {n: p.grad for n, p in _model_params(st["model"]).items()}}
    if k == "render":
        with torch.no_grad():
            out = st["model"].render(x["o"], x["d"], st["sampler"], extras=False)
        return {n: out[n] for n in ("rgb", "depth", "normal", "opacity")}
    if k == "render_grad":
        out = st["model"].render(x["o"], x["d"], st["sampler"], randoms=x["randoms"])
        loss = rendering.compute_huber_color_loss(out["rgb"], x["target"])
        loss.backward()
        return {"loss": loss.detach(), "corners": out["corner_indices"],
                **{n: out[n].detach() for n in ("rgb", "depth", "normal", "opacity", "weights", "sdf_samples")},
                "grad": {n: _take(p) for n, p in _model_params(st["model"]).items()}}
    if k == "query":
        with torch.no_grad():
            sdf = st["sdf"].query_sdf(x["pts"])
            grad, normal, _, _ = st["sdf"].query_normals(x["pts"], return_corners=False)
        return {"sdf": sdf, "grad": grad, "normal": normal}
    if k == "query_grad":
        sdf = st["sdf"].query_sdf(x["pts"])
        _, normal, _, _ = st["sdf"].query_normals(x["pts"], return_corners=False)
        torch.autograd.backward([sdf, normal], [x["w"], x["wn"]])
        return {"sdf": sdf.detach(), "normal": normal.detach(), "grad": _take(st["sdf"].grid)}
    if k == "lattice":
        sdf, normal = ops.field_query_lattice(st["sdf"].grid.detach(), LO, HI, [st["case"]["side"]] * 3, LO, HI)
        return {"sdf": sdf, "normal": normal}
    if k == "appearance":
        feats = st["hash"](x["pts"], st["case"]["levels"])
        rgb = st["mlp"](feats, st["sh"](x["dirs"]), x["normals"])
        rgb.backward(x["w"])
        n = st["mlp"].net
        return {"rgb": rgb.detach(), "emb": _take(st["hash"].encoder.embeddings), "normals": _take(x["normals"]),
                "W0": _take(n[0].weight), "b0": _take(n[0].bias), "W1": _take(n[2].weight), "b1": _take(n[2].bias)}
    if k == "composite":
        out = rendering.volume_render_from_samples(x["colors"], x["sdf"], x["normals"], x["dirs"], x["z"], x["dists"],
                                                   x["s"], pts=x["pts"])
        torch.autograd.backward([out["rgb"], out["depth"]], [x["w"], x["wd"]])
        return {**{n: out[n].detach() for n in ("rgb", "depth", "normal", "opacity", "weights", "transmittance")},
                "grad": {n: _take(x[n]) for n in ("colors", "sdf", "normals", "s")}}
    verts, _ = regularization.extract_active_vertices(x["corners"], st["res"])
    acc = torch.zeros_like(x["grid"])
    eik, _ = regularization.compute_eikonal_loss_and_gradient(x["grid"], verts, st["eps"], st["res"],
                                                              accumulate_grad=acc, weight=W_EIK)
    curv, _ = regularization.compute_curvature_loss_and_gradient(x["grid"], verts, st["eps"], st["res"],
                                                                 accumulate_grad=acc, weight=W_CURV)
    return {"count": verts.shape[0], "eik": eik, "curv": curv, "grad": acc}


def work(case):
    """Each input read once, each output written once. A render's inputs are its rays and the model's
    grid and table (the part of them that its samples can touch), its outputs a few floats a ray;
    training adds the gradients, and the optimizers' reads and writes of all parameters and moments."""
    k = case["kind"]
    if k in ("train", "render", "render_grad"):
        n = case["rays"] * (case["coarse"] + case["fine"])
        vox, table = case["res"] ** 3, 16 * (1 << 19) * 2
        model = 4 * (min(vox, 32 * n) + min(table, 256 * n))
        mlp = 2 * (51 * 64 + 64 * 3)
        if k == "render":
            return {"bytes": model + 4 * 14 * case["rays"], "flops": n * (mlp + 1500)}
        if k == "render_grad":
            return {"bytes": 2 * model + 4 * (vox + table) + 4 * 17 * case["rays"] + n * (8 * 24 + 20),
                    "flops": n * (3 * mlp + 4000)}
        return {"bytes": model + 28 * table + 8 * vox + 4 * 12 * case["rays"], "flops": n * (3 * mlp + 4000)}
    if k in ("query", "query_grad"):
        n, vox = case["points"], case["res"] ** 3
        if k == "query":
            return {"bytes": n * (12 + 28) + 4 * min(vox, 32 * n), "flops": n * 200}
        return {"bytes": n * (12 + 16 + 16) + 4 * min(vox, 32 * n) + 4 * vox, "flops": n * 500}
    if k == "lattice":
        n = case["side"] ** 3
        return {"bytes": 16 * n + 4 * min(case["res"] ** 3, 32 * n), "flops": n * 200}
    if k == "appearance":
        n, table = case["points"], math.ceil(case["levels"]) * (1 << 19) * 2
        return {"bytes": n * 4 * (3 + 3 + 3 + 3 + 3 + 3) + 4 * min(table, 256 * n) + 4 * 16 * (1 << 19) * 2,
                "flops": n * (6 * (51 * 64 + 64 * 3) + 1500)}
    if k == "composite":
        n = case["rays"] * case["samples"]
        return {"bytes": n * 4 * (3 + 1 + 3 + 3 + 2 + 2 + 7) + case["rays"] * 4 * 15, "flops": n * 200}
    vox = case["res"] ** 3
    return {"bytes": case["points"] * 192 + 8 * vox, "flops": case["points"] * 300}


# ------------------------------------------------------------------------ float64 values ------


def _sdf64(f, p):
    """Trilinear value of the (R,R,R) grid f at points p, coordinates clamped to the grid."""
    r = f.shape[0]
    c = ((p + 1.0) * 0.5 * (r - 1)).clamp(0, r - 1)
    i = c.floor().long().clamp(max=r - 2)
    t = c - i
    out = 0.0
    for a in (0, 1):
        for b in (0, 1):
            for e in (0, 1):
                w = (t[..., 0] if a else 1 - t[..., 0]) * (t[..., 1] if b else 1 - t[..., 1]) * (
                    t[..., 2] if e else 1 - t[..., 2])
                out = out + w * f[i[..., 0] + a, i[..., 1] + b, i[..., 2] + e]
    return out


def _normal64(f, p):
    """Trilinear blend of the corners' central differences (one-sided at the border), and the unit
    vector along it; the lower corners' indices too."""
    r, eps = f.shape[0], 2.0 / (f.shape[0] - 1)
    c = ((p + 1.0) * 0.5 * (r - 1)).clamp(0, r - 1.0001)
    i = c.floor().long()
    t = c - i
    g = 0.0
    for a in (0, 1):
        for b in (0, 1):
            for e in (0, 1):
                w = (t[..., 0] if a else 1 - t[..., 0]) * (t[..., 1] if b else 1 - t[..., 1]) * (
                    t[..., 2] if e else 1 - t[..., 2])
                q = [i[..., 0] + a, i[..., 1] + b, i[..., 2] + e]
                n = []
                for ax in range(3):
                    up, dn = list(q), list(q)
                    up[ax], dn[ax] = (q[ax] + 1).clamp(max=r - 1), (q[ax] - 1).clamp(min=0)
                    n.append((f[tuple(up)] - f[tuple(dn)]) / ((up[ax] - dn[ax]) * eps))
                g = g + w[..., None] * torch.stack(n, -1)
    return g, g / (g.norm(dim=-1, keepdim=True) + 1e-8), i


def _hash64(emb, x, levels=16.0):
    b = math.exp((math.log(2048) - math.log(16)) / 15)
    out = []
    for lv in range(16):
        lw = min(1.0, max(0.0, levels - lv))
        s = x.clamp(0, 1) * math.floor(16 * b ** lv)
        i = s.floor().long()
        t, v = s - i, 0.0
        if lw > 0:
            for a in (0, 1):
                for c in (0, 1):
                    for e in (0, 1):
                        h = ((i[:, 0] + a) ^ ((i[:, 1] + c) * 2654435761) ^ ((i[:, 2] + e) * 805459861)) % emb.shape[1]
                        w = (t[:, 0] if a else 1 - t[:, 0]) * (t[:, 1] if c else 1 - t[:, 1]) * (
                            t[:, 2] if e else 1 - t[:, 2])
                        v = v + w[:, None] * emb[lv][h]
            out.append(lw * v)
        else:
            out.append(torch.zeros(x.shape[0], 2, dtype=x.dtype, device=x.device))
    return torch.cat(out, -1)


def _sh64(d):
    """Real spherical harmonics up to degree 3 of unit vectors, from their closed forms."""
    x, y, z = d.unbind(-1)
    pi = math.pi
    c1, c2, c20 = math.sqrt(3 / (4 * pi)), math.sqrt(15 / (4 * pi)), math.sqrt(5 / (16 * pi))
    c33, c32, c31, c30 = (math.sqrt(v / pi) for v in (35 / 32, 105 / 4, 21 / 32, 7 / 16))
    return torch.stack([
        torch.full_like(x, math.sqrt(1 / (4 * pi))), -c1 * y, c1 * z, -c1 * x, c2 * x * y, -c2 * y * z,
        c20 * (2 * z * z - x * x - y * y), -c2 * x * z, c2 / 2 * (x * x - y * y), -c33 * y * (3 * x * x - y * y),
        c32 * x * y * z, -c31 * y * (4 * z * z - x * x - y * y), c30 * z * (2 * z * z - 3 * x * x - 3 * y * y),
        -c31 * x * (4 * z * z - x * x - y * y), c32 / 2 * z * (x * x - y * y), -c33 * x * (x * x - 3 * y * y)], -1)


def _mlp64(w, feats, sh, normals):
    h = torch.relu(torch.cat([feats, sh, normals], -1) @ w[0].T + w[1])
    return torch.sigmoid(h @ w[2].T + w[3])


def _composite64(colors, sdf, normals, dirs, z, dists, pts, s):
    cos = (normals * dirs[:, None]).sum(-1)
    off = 0.5 * dists * cos
    p0, p1 = torch.sigmoid(s * (sdf - off)), torch.sigmoid(s * (sdf + off))
    alpha = ((p0 - p1) / p0.clamp(min=1e-5)).clamp(0, 1) * (pts.norm(dim=-1) < 1.0)
    q = (1 - alpha + 1e-7).clamp(0, 1)
    t = torch.cumprod(torch.cat([torch.ones_like(q[:, :1]), q], 1), 1)[:, :-1]
    w = torch.where(t < 1e-4, torch.zeros_like(t), alpha * t)
    nsum = (w[..., None] * normals).sum(1)
    return {"rgb": (w[..., None] * colors).sum(1), "depth": (w * z).sum(1, keepdim=True),
            "normal": nsum / (nsum.norm(dim=-1, keepdim=True) + 1e-8), "opacity": w.sum(1, keepdim=True),
            "weights": w, "transmittance": t}


def _sample64(f, o, d, coarse, fine, randoms):
    """The 4-step inverse-CDF sampler (occupancy all set): sample depths."""
    n = o.shape[0]
    mid = -(o * d).sum(-1, keepdim=True) / (d * d).sum(-1, keepdim=True)
    near = (mid - 1).clamp(min=0.05)
    far = torch.maximum(mid + 1, near + 0.1)
    t = torch.linspace(0, 1, coarse, device=DEV, dtype=torch.float64)
    z = near * (1 - t) + far * t
    if randoms is not None:
        m = 0.5 * (z[:, 1:] + z[:, :-1])
        lo, hi = torch.cat([z[:, :1], m], 1), torch.cat([m, z[:, -1:]], 1)
        z = lo + (hi - lo) * randoms[0].double()

    def at(zz):
        return o[:, None] + d[:, None] * zz[..., None]

    sdf, per = _sdf64(f, at(z)), fine // 4
    for k in range(4):
        inside = (at(z).norm(dim=-1) < 1.0)
        ins = (inside[:, :-1] | inside[:, 1:]).double()
        f0, f1, gap = sdf[:, :-1], sdf[:, 1:], z[:, 1:] - z[:, :-1]
        cos = (f1 - f0) / (gap + 1e-5)
        cos = torch.minimum(cos, torch.cat([torch.zeros_like(cos[:, :1]), cos[:, :-1]], 1)).clamp(-1e3, 0) * ins
        fm, inv_s = 0.5 * (f0 + f1), 64.0 * 2 ** k
        c0, c1 = torch.sigmoid((fm - cos * gap * 0.5) * inv_s), torch.sigmoid((fm + cos * gap * 0.5) * inv_s)
        alpha = (c0 - c1 + 1e-5) / (c0 + 1e-5)
        trans = torch.cumprod(torch.cat([torch.ones_like(alpha[:, :1]), 1 - alpha + 1e-7], 1), 1)[:, :-1]
        pm = at(0.5 * (z[:, 1:] + z[:, :-1]))
        occ = ((pm >= -1) & (pm <= 1)).all(-1).double()
        w = alpha * trans * (0.9 * occ + 0.1) + 1e-5
        cdf = torch.cumsum(w / w.sum(1, keepdim=True), 1)
        cdf = torch.cat([torch.zeros_like(cdf[:, :1]), cdf], 1)
        if randoms is not None:
            u = randoms[1][k].double().contiguous()
        else:
            u = torch.linspace(0.5 / per, 1 - 0.5 / per, per, device=DEV, dtype=torch.float64).expand(n, per).contiguous()
        i = torch.searchsorted(cdf, u, right=True)
        lo, hi = (i - 1).clamp(min=0), i.clamp(max=cdf.shape[1] - 1)
        c0, c1, z0, z1 = cdf.gather(1, lo), cdf.gather(1, hi), z.gather(1, lo), z.gather(1, hi)
        den = torch.where(c1 - c0 < 1e-5, torch.ones_like(c0), c1 - c0)
        new = z0 + (u - c0) / den * (z1 - z0)
        z, order = torch.sort(torch.cat([z, new], 1), dim=1)
        sdf = torch.cat([sdf, _sdf64(f, at(new))], 1).gather(1, order)
    return z


def _render64(w, o, d, z):
    """Colours, SDF, ... of given depths, as autograd can differentiate them; corner indices too."""
    dists = torch.cat([z[:, 1:] - z[:, :-1], z[:, -1:] - z[:, -2:-1]], 1)
    mid = z + 0.5 * dists
    pts = o[:, None] + d[:, None] * mid[..., None]
    f = w["grid"].reshape(w["grid"].shape[-3:])
    sdf = _sdf64(f, pts)
    _, normal, low = _normal64(f, pts)
    feats = _hash64(w["emb"], (pts.reshape(-1, 3) + 1) * 0.5)
    sh = _sh64(d)[:, None].expand(-1, z.shape[1], -1).reshape(-1, 16)
    colors = _mlp64(w["mlp"], feats, sh, normal.reshape(-1, 3)).reshape(*z.shape, 3)
    s = torch.exp(w["v"] * 10).clamp(1e-4, 300)
    out = _composite64(colors, sdf, normal, d, mid, dists, pts, s)
    out["sdf_samples"] = sdf.unsqueeze(-1)
    return out, low


def _double(x):
    w = {"grid": x["grid"].double(), "emb": x["emb"].double(), "mlp": [v.double() for v in x["mlp"]],
         "v": torch.tensor(0.3, device=DEV).double()}
    return w


def _regularize64(f, lin, grad):
    """Losses over the interior vertices of the list, weighted gradients added into grad."""
    r = f.shape[0]
    eps, nv = 2.0 / (r - 1), lin.numel()
    v = torch.stack([lin // (r * r), lin // r % r, lin % r], -1)
    v = v[((v > 0) & (v < r - 1)).all(-1)]
    c = (v[:, 0] * r + v[:, 1]) * r + v[:, 2]
    ff, gg, step = f.reshape(-1), grad.reshape(-1), (r * r, r, 1)
    n = torch.stack([(ff[c + s] - ff[c - s]) / (2 * eps) for s in step], -1)
    lap = torch.stack([(ff[c + s] + ff[c - s] - 2 * ff[c]) / eps ** 2 for s in step], -1)
    ln = n.norm(dim=-1, keepdim=True)
    dn = W_EIK * 2 / nv * (1 - 1 / (ln + 1e-8)) * n / (2 * eps)
    dl = W_CURV * 2 / nv * lap / eps ** 2
    for a, s in enumerate(step):
        gg.index_add_(0, c + s, dn[:, a] + dl[:, a])
        gg.index_add_(0, c - s, dl[:, a] - dn[:, a])
    gg.index_add_(0, c, -2 * dl.sum(-1))
    return ((ln - 1) ** 2).mean(), (lap ** 2).sum(-1).mean()


def _train64(case, x, randoms, amplify):
    """Loss, outputs, parameter gradients and the corners' bitmap of one render and its Huber loss."""
    w = _double(x)
    leaves = {"grid": w["grid"], "emb": w["emb"], "v": w["v"], "W0": w["mlp"][0], "b0": w["mlp"][1], "W1": w["mlp"][2],
              "b1": w["mlp"][3]}
    for t in leaves.values():
        t.requires_grad_()
    n, r, f = case["rays"], case["res"], w["grid"].detach()[0, 0]
    seen = torch.zeros(r * r * r, dtype=torch.bool, device=DEV)
    outs, loss = {}, 0.0
    for i in range(0, n, 512):
        o, d = x["o"][i:i + 512].double(), x["d"][i:i + 512].double()
        rnd = None if randoms is None else (randoms[0][i:i + 512], randoms[1][:, i:i + 512])
        with torch.no_grad():
            z = _sample64(f, o, d, case["coarse"], case["fine"], rnd)
        out, low = _render64(w, o, d, z)
        e = (out["rgb"] - x["target"][i:i + 512].double()).abs()
        part = torch.where(e <= 0.1, 5.0 * e * e, e - 0.05).sum() / (3 * n)
        part.backward()
        loss = loss + part.detach()
        for name, t in out.items():
            outs.setdefault(name, []).append(t.detach())
        for a in (0, 1):
            for b in (0, 1):
                for c in (0, 1):
                    seen[((low[..., 0] + a) * r + low[..., 1] + b) * r + low[..., 2] + c] = True
    grads = {name: t.grad for name, t in leaves.items()}
    if amplify and grads["v"] < 0:
        grads["v"] = 5.0 * grads["v"]
    return loss, {name: torch.cat(v) for name, v in outs.items()}, grads, seen


def exact(case, seed):
    x, k = _inputs(case, seed), case["kind"]
    if k == "train":
        g = _gen(seed)  # the draws of the first pass after prepare's
        n, per = case["rays"], case["fine"] // 4
        rnd = (torch.rand(n, case["coarse"], device=DEV, generator=g),
               torch.stack([torch.rand(n, per, device=DEV, generator=g) for _ in range(4)]))
        loss, out, grads, seen = _train64(case, x, rnd, True)
        r, f = case["res"], x["grid"].double()[0, 0]
        lin = seen.nonzero().squeeze(1)
        v = torch.stack([lin // (r * r), lin // r % r, lin % r], -1) * (2.0 / (r - 1)) - 1.0
        near = v.norm(dim=-1) < 1.2
        lin = lin[near] if bool(near.any()) else lin
        lin = lin[f.reshape(-1)[lin].abs() < BAND * 2.0 / (r - 1)]
        eik, curv = _regularize64(f, lin, grads["grid"])
        return {"loss": loss, "eik": eik, "curv": curv, "n_active": None, "rgb": out["rgb"], "grad": grads}
    if k == "render":
        w, outs = _double(x), {}
        with torch.no_grad():
            for i in range(0, case["rays"], 4096):
                o, d = x["o"][i:i + 4096].double(), x["d"][i:i + 4096].double()
                z = _sample64(w["grid"][0, 0], o, d, case["coarse"], case["fine"], None)
                out, _ = _render64(w, o, d, z)
                for name in ("rgb", "depth", "normal", "opacity"):
                    outs.setdefault(name, []).append(out[name])
        return {name: torch.cat(v) for name, v in outs.items()}
    if k == "render_grad":
        loss, out, grads, _ = _train64(case, x, x["randoms"], False)
        names = ("rgb", "depth", "normal", "opacity", "weights", "sdf_samples")
        return {"loss": loss, "corners": None, **{n: out[n] for n in names}, "grad": grads}
    if k in ("query", "query_grad", "lattice"):
        f = x["grid"].double()[0, 0]
        if k == "lattice":
            a = torch.linspace(-1.0, 1.0, case["side"], device=DEV).double()
            pts = torch.stack(torch.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 3)
        else:
            pts = x["pts"].double()
        f.requires_grad_(k == "query_grad")
        got = {"sdf": [], "grad": [], "normal": []}
        for i in range(0, pts.shape[0], 1 << 20):
            p = pts[i:i + (1 << 20)]
            sdf, (g, n, _) = _sdf64(f, p), _normal64(f, p)
            if k == "query_grad":
                torch.autograd.backward([sdf, n], [x["w"][i:i + (1 << 20), 0].double(), x["wn"][i:i + (1 << 20)].double()])
            for name, t in (("sdf", sdf), ("grad", g), ("normal", n)):
                got[name].append(t.detach())
        got = {name: torch.cat(v) for name, v in got.items()}
        if k == "lattice":
            return {"sdf": got["sdf"], "normal": got["normal"]}
        if k == "query":
            return {"sdf": got["sdf"][:, None], "grad": got["grad"], "normal": got["normal"]}
        return {"sdf": got["sdf"][:, None], "normal": got["normal"], "grad": f.grad[None, None]}
    if k == "appearance":
        emb, mlp = x["emb"].double().requires_grad_(), [v.double().requires_grad_() for v in x["mlp"]]
        normals, rgb = x["normals"].double().requires_grad_(), []
        for i in range(0, case["points"], 1 << 17):
            j = slice(i, i + (1 << 17))
            out = _mlp64(mlp, _hash64(emb, x["pts"][j].double(), case["levels"]), _sh64(x["dirs"][j].double()), normals[j])
            out.backward(x["w"][j].double())
            rgb.append(out.detach())
        return {"rgb": torch.cat(rgb), "emb": emb.grad, "normals": normals.grad, "W0": mlp[0].grad, "b0": mlp[1].grad,
                "W1": mlp[2].grad, "b1": mlp[3].grad}
    if k == "composite":
        y = {n: x[n].double().requires_grad_() for n in ("colors", "sdf", "normals")}
        y["s"] = torch.tensor(64.0, device=DEV, dtype=torch.float64, requires_grad=True)
        out = _composite64(y["colors"], y["sdf"].squeeze(-1), y["normals"], x["dirs"].double(), x["z"].double(),
                           x["dists"].double(), x["pts"].double(), y["s"])
        torch.autograd.backward([out["rgb"], out["depth"]], [x[n].double() for n in ("w", "wd")])
        return {**{n: t.detach() for n, t in out.items()}, "grad": {n: t.grad for n, t in y.items()}}
    r, c = case["res"], x["corners"].reshape(-1, 3)
    lin = torch.unique((c[:, 0] * r + c[:, 1]) * r + c[:, 2])
    grad = torch.zeros(r, r, r, device=DEV, dtype=torch.float64)
    eik, curv = _regularize64(x["grid"].double()[0, 0], lin, grad)
    return {"count": None, "eik": eik, "curv": curv, "grad": grad[None, None]}
