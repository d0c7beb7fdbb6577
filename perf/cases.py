"""The work a user of the tracer has it do, as measurable cases: frames of a
viewer, batches of views, training steps and scene loading, each through the
public Python API (gtrace.tracer) and over the sizes of the synthetic
configurations (gtrace.synth, bench.py) and around them.

A case is a dict of plain values:

  kind      "frame"    one view of a scene the program holds
            "display"  progressive anti-aliased frames of one view, each tone-mapped
                       to the 8-bit image that is shown
            "batch"    views of several scenes in one call
            "train"    checkpointing render, L2 loss and backward on device buffers
            "train_batch"  the gradient of several views, host buffers
            "scene"    a scene loaded and its first frame shown
  scene     "uniform" (the small configuration's distributions) or "clusters"
            (the 64-cluster mixture of the larger ones), n Gaussians
  w, h, k, alpha_min, t_stop (transmittance cutoff), deg (SH degree), radius
            (camera distance from the origin)
  out       where a frame goes: "queued" and "device" (device buffer, the call
            returns once queued or done), "host", "pinned" (page-locked)
  source    what a scene is loaded from: "device", "host" (packed records),
            "ply" (the file's bytes); fast: the quick hierarchy
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "webgpu-gaussiantracer_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from gtrace import _lib as L  # noqa: E402
from gtrace import synth  # noqa: E402
from gtrace.ply import write_ply  # noqa: E402
from gtrace.tracer import Context, Scene  # noqa: E402
from gtrace.uniforms import with_fields  # noqa: E402

_FRAME = dict(kind="frame", scene="clusters", k=16, alpha_min=0.01, t_stop=0.01, deg=3, radius=12.0)


def listed():
    return [
        # the smallest call: a thumbnail with the reference app's own settings
        # (k 6, alpha_min 0.2, cutoff 0.03); launches and latency count
        dict(_FRAME, name="thumbnail", scene="uniform", n=16384, w=64, h=64, k=6, alpha_min=0.2, t_stop=0.03,
             radius=4.0, out="queued"),
        # the small configuration as an application without device buffers calls it
        dict(_FRAME, name="small_host", scene="uniform", n=16384, w=256, h=256, k=6, radius=4.0, out="host"),
        # an interactive preview of a large scene, odd sizes
        dict(_FRAME, name="preview_1m", n=1_000_000, w=481, h=271, out="device"),
        # a quarter of full HD, frames queued one after another
        dict(_FRAME, name="quarter_hd_1m", n=1_000_000, w=960, h=540, out="queued"),
        # the headline: full HD of 1M Gaussians into a page-locked host image
        dict(_FRAME, name="full_hd_1m", n=1_000_000, w=1920, h=1080, out="pinned"),
        # a still picture refined over frames and shown, from coarse settings
        dict(_FRAME, name="display_200k", kind="display", n=200_000, w=1280, h=720, k=8, alpha_min=0.05, frames=2),
        # offline rendering: uneven views of several scenes in one call
        dict(_FRAME, name="batch_8_views", kind="batch", n=250_000, scenes=3, views=8, w=820, h=460, radius=11.0),
        # one optimisation step of the differentiable configuration
        dict(_FRAME, name="train_200k", kind="train", n=200_000, w=800, h=800, k=8),
        # gradients of a few small ragged views, host buffers (a debugging or early-training size)
        dict(_FRAME, name="train_batch_16k", kind="train_batch", scene="uniform", n=16384, w=97, h=75, views=3, k=6,
             radius=4.0),
        # opening a large scene that is on the GPU already, with its first frame
        dict(_FRAME, name="open_1m", kind="scene", n=1_000_000, w=160, h=90, source="device", fast=False),
        # a scene rebuilt every step with the quick hierarchy, from host records
        dict(_FRAME, name="rebuild_65k", kind="scene", n=65_536, w=200, h=150, k=8, source="host", fast=True),
        # opening a PLY file's bytes
        dict(_FRAME, name="open_ply_100k", kind="scene", n=100_000, w=160, h=120, k=6, alpha_min=0.05, t_stop=0.03,
             source="ply", fast=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "display", "batch", "train", "train_batch", "scene"])
    scene = rng.choice(["uniform", "clusters", "clusters"])
    c = dict(kind=kind, scene=scene, k=rng.choice([1, 4, 6, 7, 8, 16, 16, 32]),
             alpha_min=rng.choice([0.01, 0.01, 0.05, 0.1, 0.2]), t_stop=rng.choice([0.01, 0.03]),
             deg=rng.choice([0, 1, 2, 3, 3, 3]))
    c["radius"] = round(rng.uniform(3.5, 6.0), 2) if scene == "uniform" else round(rng.uniform(8.0, 14.0), 2)
    # uniform scenes are compact: dense beyond real use above some 10^5
    c["n"] = _log(rng, 4096, 65_536) if scene == "uniform" else _log(rng, 50_000, 1_000_000)
    if kind in ("frame", "display"):
        c["w"] = _log(rng, 64, 1920)
        c["h"] = max(48, min(1080, int(c["w"] * rng.uniform(0.5, 1.0))))
        if kind == "frame":
            c["out"] = rng.choice(["queued", "device", "host", "pinned"])
        else:
            c["w"], c["h"] = min(c["w"], 1280), min(c["h"], 720)
            c["frames"] = rng.randint(1, 3)
    elif kind == "batch":
        c["scenes"], c["views"] = rng.randint(1, 4), rng.randint(2, 9)
        c["n"] = min(c["n"], 300_000)
        c["w"], c["h"] = _log(rng, 64, 900), _log(rng, 48, 500)
    elif kind == "train":
        c["n"] = min(c["n"], 400_000)
        c["w"], c["h"] = _log(rng, 64, 900), _log(rng, 64, 800)
    elif kind == "train_batch":
        c["n"] = min(c["n"], 65_536)
        c["views"] = rng.randint(1, 4)
        c["w"], c["h"] = _log(rng, 32, 400), _log(rng, 32, 300)
    else:
        c["w"], c["h"] = _log(rng, 32, 400), _log(rng, 32, 300)
        c["source"] = rng.choice(["device", "host", "ply"])
        c["fast"] = rng.choice([False, False, True])
        if c["source"] != "device":
            c["n"] = min(c["n"], 200_000)
    return c


# ------------------------------------------------------------------ inputs
_shared = {}


def _context():
    """One context for the process, as a program keeps it."""
    if "ctx" not in _shared:
        _shared["ctx"] = Context(0)
    return _shared["ctx"]


def _raw(case, seed):
    """Pre-activation Gaussians on the GPU: the distributions of gtrace.synth."""
    g = torch.Generator(device="cuda")
    g.manual_seed(0x6A5C0000 + seed)
    n = case["n"]

    def uni(*s):
        return torch.rand(*s, generator=g, device="cuda")

    def nor(*s):
        return torch.randn(*s, generator=g, device="cuda")

    if case["scene"] == "uniform":
        xyz = nor(n, 3).clamp_(-3.0, 3.0)
        log_s = uni(n, 3) * 2.0 - 4.5
        o = 0.05 + 0.94 * uni(n)
        logit = torch.log(o / (1.0 - o))
    else:
        centres = uni(64, 3) * 10.0 - 5.0
        sig = 0.1 + 0.7 * uni(64)
        pick = torch.randint(0, 64, (n,), generator=g, device="cuda")
        xyz = centres[pick] + sig[pick, None] * nor(n, 3)
        lx = uni(n, 1) * 3.0 - 5.0
        log_s = torch.cat([lx, (lx - uni(n, 2) * math.log(10.0)).clamp_(min=-5.0)], 1)
        logit = 1.5 * nor(n)
    rot = nor(n, 4)
    sh = 0.05 * nor(n, 16, 3)
    sh[:, 0] = 0.5 * nor(n, 3)
    return {"xyz": xyz, "log_scale": log_s, "rot": rot, "opacity_logit": logit, "sh": sh}


def _packed(raw):
    """Activated 320-byte records, as the PLY loader packs them."""
    n = raw["xyz"].shape[0]
    rec = torch.zeros(n, 80, device="cuda")
    rec[:, 0:3] = raw["xyz"]
    rec[:, 4:7] = torch.exp(raw["log_scale"].double())
    q = raw["rot"].double()
    rec[:, 8:12] = q / q.norm(dim=1, keepdim=True)
    rec[:, 12] = torch.sigmoid(raw["opacity_logit"].double())
    rec[:, 16:80].view(n, 16, 4)[:, :, :3] = raw["sh"]
    return rec


def _camera(case, seed, i=0):
    """Camera i of a case: on the sphere of its radius, looking at the origin."""
    r = np.random.default_rng(1000 * seed + i)
    v = r.normal(size=3)
    v[1] *= 0.5
    return tuple(case["radius"] * v / np.linalg.norm(v))


def _uniforms(case, w, h, seed, i=0):
    v = synth.view(w, h, _camera(case, seed, i), k=case["k"], alpha_min=case["alpha_min"], T_min=case["t_stop"])
    return with_fields(v.uniforms, sh_degree_max=case["deg"])


def _view_sizes(case):
    """Uneven sizes of the views of a batch, the largest first."""
    return [(max(8, case["w"] - 43 * i % case["w"]), max(8, case["h"] - 29 * i % case["h"]))
            for i in range(case["views"])]


def _scene_of(ctx, case, rec):
    torch.cuda.synchronize()  # the records come from torch's stream
    return Scene(ctx, None, case["alpha_min"], device_ptr=rec.data_ptr(), n=rec.shape[0], stride=320)


class _State:
    """What a program holds between calls; its scenes go with it."""

    def __init__(self, case):
        self.case = case
        self.scenes = []

    def __del__(self):
        for s in self.scenes:
            s.close()


def prepare(case, seed):
    ctx = _context()
    s = _State(case)
    kind, w, h = case["kind"], case["w"], case["h"]
    raw = _raw(case, seed)
    if kind == "scene":
        s.u = _uniforms(case, w, h, seed)
        s.rgba = torch.empty(h, w, 4, device="cuda")
        if case["source"] == "ply":
            s.data = write_ply({k: v.cpu().numpy() for k, v in raw.items()})
        else:
            s.data = _packed(raw)
            if case["source"] == "host":
                s.data = s.data.cpu().numpy()
        return s
    rec = _packed(raw)
    s.scenes.append(_scene_of(ctx, case, rec))
    if kind in ("frame", "display"):
        s.u = _uniforms(case, w, h, seed)
        if kind == "display" or case["out"] == "pinned":
            s.rgba = torch.empty(h, w, 4, pin_memory=True).numpy()  # page-locked
        elif case["out"] == "host":
            s.rgba = np.zeros((h, w, 4), np.float32)
        else:
            s.rgba = torch.empty(h, w, 4, device="cuda")
    elif kind == "batch":
        for i in range(1, case["scenes"]):
            s.scenes.append(_scene_of(ctx, case, _packed(_raw(dict(case, n=case["n"] // (i + 1)), seed + 7919 * i))))
        s.images = [torch.empty(hh, ww, 4, device="cuda") for ww, hh in _view_sizes(case)]
        s.views = [(s.scenes[i % case["scenes"]], _uniforms(case, ww, hh, seed, i), ww, hh, s.images[i].data_ptr())
                   for i, (ww, hh) in enumerate(_view_sizes(case))]
    elif kind == "train":
        s.u = _uniforms(case, w, h, seed)
        s.rgba = torch.empty(h, w, 4, device="cuda")
        s.target = torch.empty(h, w, 4, device="cuda")
        s.dl = torch.empty(h, w, 4, device="cuda")
        s.grad = torch.empty(59, case["n"], device="cuda")
        # the target is the scene with positions, opacities and base colours perturbed
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        for name, sd in (("xyz", 0.01), ("opacity_logit", 0.1)):
            raw[name] = raw[name] + sd * torch.randn(raw[name].shape, generator=g, device="cuda")
        raw["sh"][:, 0] += 0.05 * torch.randn(case["n"], 3, generator=g, device="cuda")
        t = _scene_of(ctx, case, _packed(raw))
        ctx.render_device(t, s.u, w, h, s.target.data_ptr())
        t.close()
    else:
        r = np.random.default_rng(seed)
        s.views = []
        for i, (ww, hh) in enumerate(_view_sizes(case)):
            dl = np.zeros((hh, ww, 4), np.float32)
            dl[..., :3] = 0.1 * r.normal(size=(hh, ww, 3))
            s.views.append((s.scenes[0], _uniforms(case, ww, hh, seed, i), ww, hh, dl))
    return s


def run(s):
    ctx, case = _context(), s.case
    kind, w, h = case["kind"], case["w"], case["h"]
    if kind == "frame":
        if case["out"] in ("queued", "device"):
            ctx.render_device(s.scenes[0], s.u, w, h, s.rgba.data_ptr(), asynchronous=case["out"] == "queued")
            return s.rgba
        return ctx.render(s.scenes[0], s.u, w, h, out=s.rgba)
    if kind == "display":
        for f in range(case["frames"]):
            ctx.render(s.scenes[0], with_fields(s.u, accumulated_frames=f), w, h, out=s.rgba, antialias=True)
            shown = ctx.tonemap(s.rgba, L.GT_TONEMAP_EXPOSURE_GAMMA)
        return {"rgba": s.rgba, "shown": shown}
    if kind == "batch":
        ctx.render_batch(s.views, device_outputs=True)
        return s.images
    if kind == "train":
        ctx.render_device(s.scenes[0], s.u, w, h, s.rgba.data_ptr(), checkpoint=True)
        loss = ctx.l2_loss(s.rgba.data_ptr(), s.target.data_ptr(), w * h, s.dl.data_ptr())
        ctx.backward_device(s.scenes[0], s.u, w, h, s.dl.data_ptr(), s.grad.data_ptr())
        return {"grad": s.grad, "image": s.rgba, "loss": loss}
    if kind == "train_batch":
        grads, _ = ctx.backward_batch(s.views)
        return grads[s.scenes[0]]
    if case["source"] == "ply":
        scene = Scene.from_ply(ctx, s.data, case["alpha_min"], fast_build=case["fast"])
    elif case["source"] == "host":
        scene = Scene(ctx, s.data, case["alpha_min"], fast_build=case["fast"])
    else:
        scene = Scene(ctx, None, case["alpha_min"], device_ptr=s.data.data_ptr(), n=case["n"], stride=320,
                      fast_build=case["fast"])
    ctx.render_device(scene, s.u, w, h, s.rgba.data_ptr())
    kept = scene.info()["n_kept"]
    scene.close()
    return {"image": s.rgba, "kept": kept}


def work(case):
    """Every Gaussian's 59 floats once (for a scene that is loaded, its records
    as they come), every pixel's RGBA once, the gradients once; and some 50
    composited entries a ray at about 100 operations each (ray transform,
    proxy entry, response), three times that with gradients."""
    kind, n = case["kind"], case["n"]
    rays = case["w"] * case["h"]
    scene_bytes = 236 * n
    if kind == "batch":
        rays = sum(a * b for a, b in _view_sizes(case))
        scene_bytes = sum(236 * (n // (i + 1)) for i in range(case["scenes"]))
    nbytes, flops = scene_bytes + 16 * rays, 5000 * rays
    if kind == "display":
        nbytes = scene_bytes + case["frames"] * (16 + 16 + 4) * rays
        flops *= case["frames"]
    elif kind == "train":
        nbytes = 2 * scene_bytes + (16 + 16) * rays
        flops *= 3
    elif kind == "train_batch":
        rays = sum(a * b for a, b in _view_sizes(case))
        nbytes, flops = 2 * scene_bytes + 16 * rays, 15000 * rays
    elif kind == "scene":
        nbytes = (248 if case["source"] == "ply" else 320) * n + 16 * rays
    return {"bytes": nbytes, "flops": flops}


# --------------------------------------------------------- 64-bit reference
_PAIR_LIMIT = 2e10  # (Gaussian, ray) pairs: some seconds on the GPU


def _planes():
    """The 10 slabs of the unit icosahedron (inradius 1): |n . x| <= 1."""
    p = (1.0 + math.sqrt(5.0)) / 2.0
    n = [(1, 1, 1), (1, 1, -1), (1, -1, 1), (-1, 1, 1), (0, 1 / p, p), (0, -1 / p, p), (1 / p, p, 0), (-1 / p, p, 0),
         (p, 0, 1 / p), (p, 0, -1 / p)]
    return torch.tensor(n, dtype=torch.float64, device="cuda") / math.sqrt(3.0)


def _rotation(q):
    w, x, y, z = q.unbind(-1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                        2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], -1).view(-1, 3, 3)


def _rays(u, w, h):
    f = np.frombuffer(bytes(u), dtype=np.float32)
    m = torch.tensor(f[:16].reshape(4, 4).astype(np.float64), device="cuda")
    x = (torch.arange(w, device="cuda", dtype=torch.float64) + 0.5) / w * 2.0 - 1.0
    y = (torch.arange(h, device="cuda", dtype=torch.float64) + 0.5) / h * 2.0 - 1.0
    d = (x * float(f[16]))[None, :, None] * -m[0, :3] + (y * float(f[17]))[:, None, None] * m[1, :3] - m[2, :3]
    d = (d / d.norm(dim=-1, keepdim=True)).reshape(-1, 3)
    return m[3, :3], d, float(f[18]), float(f[19])


def _hits(P, o, d, t_min, t_max, cut):
    """Entry distances of the rays' proxies: per ray its hits in order of t,
    as (index, t) arrays padded with -1 and inf."""
    keep = (P["opacity"].double() > cut).nonzero()[:, 0]
    if keep.numel() == 0:
        return torch.full((d.shape[0], 1), -1, device="cuda"), torch.full((d.shape[0], 1), math.inf, device="cuda")
    size = torch.sqrt(2.0 * torch.log(P["opacity"][keep] / cut))[:, None] * P["scale"][keep]
    inv = _rotation(P["rot"][keep]).transpose(1, 2) / size[:, :, None]  # world to object
    oo = (inv @ (o - P["mu"][keep])[:, :, None])[:, :, 0]
    nrm = _planes()
    nw = torch.einsum("pa,nab->pnb", nrm, inv).contiguous()  # (10, kept, 3)
    no = oo @ nrm.T  # (kept, 10)
    ri, ji, ti = [], [], []
    step = max(1, int(3e8 // keep.numel()))
    for a in range(0, d.shape[0], step):
        dd = d[a:a + step]
        near = far = None
        for p in range(10):
            inv_dn = 1.0 / (dd @ nw[p].T)  # (rays, kept)
            t0 = (-1.0 - no[:, p]) * inv_dn
            t1 = (1.0 - no[:, p]) * inv_dn
            lo, hi = torch.minimum(t0, t1), torch.maximum(t0, t1)
            near = lo if near is None else torch.maximum(near, lo)
            far = hi if far is None else torch.minimum(far, hi)
        r, j = ((near < far) & (near > t_min) & (near < t_max)).nonzero(as_tuple=True)
        ri.append(r + a)
        ji.append(keep[j])
        ti.append(near[r, j])
    ri, ji, ti = torch.cat(ri), torch.cat(ji), torch.cat(ti)
    order = torch.argsort(ti)
    order = order[torch.argsort(ri[order], stable=True)]
    ri, ji, ti = ri[order], ji[order], ti[order]
    count = torch.bincount(ri, minlength=d.shape[0])
    pos = torch.arange(ri.numel(), device="cuda") - (torch.cumsum(count, 0) - count)[ri]
    most = max(1, int(count.max()))
    idx = torch.full((d.shape[0], most), -1, device="cuda")
    t = torch.full((d.shape[0], most), math.inf, dtype=torch.float64, device="cuda")
    idx[ri, pos], t[ri, pos] = ji, ti
    return idx, t


def _sh_colour(sh, d, deg):
    x, y, z = d.unbind(-1)
    xx, yy, zz = x * x, y * y, z * z
    b = [torch.full_like(x, 0.28209479177387814), -0.4886025119029199 * y, 0.4886025119029199 * z,
         -0.4886025119029199 * x, 1.0925484305920792 * x * y, -1.0925484305920792 * y * z,
         0.31539156525252005 * (2 * zz - xx - yy), -1.0925484305920792 * x * z, 0.5462742152960396 * (xx - yy),
         -0.5900435899266435 * y * (3 * xx - yy), 2.890611442640554 * x * y * z,
         -0.4570457994644658 * y * (4 * zz - xx - yy), 0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy),
         -0.4570457994644658 * x * (4 * zz - xx - yy), 1.445305721320277 * z * (xx - yy),
         -0.5900435899266435 * x * (xx - 3 * yy)][:(deg + 1) ** 2]
    return 0.5 + torch.einsum("nk,nkc->nc", torch.stack(b, -1), sh[:, :len(b)])


def _composite(P, case, o, d, idx, t, t_min, t_max):
    """Rounds of k hits each, front to back; differentiable in P."""
    alpha_min, k = float(np.float32(case["alpha_min"])), case["k"]
    t_stop = float(np.float32(case["t_stop"]))
    R = _rotation(P["rot"])
    A = torch.einsum("nij,nj,nkj->nik", R, P["scale"] ** -2, R)
    dirs = P["mu"] - o
    colour = _sh_colour(P["sh"], dirs / dirs.norm(dim=1, keepdim=True), case["deg"]).clamp(min=0.0)
    n_rays, most = idx.shape
    T = torch.ones(n_rays, dtype=torch.float64, device="cuda")
    rgb = torch.zeros(n_rays, 3, dtype=torch.float64, device="cuda")
    t_curr = torch.full((n_rays,), t_min, dtype=torch.float64, device="cuda")
    count = (idx >= 0).sum(1)
    live = torch.arange(n_rays, device="cuda")
    for _ in range(most + 1):
        live = live[(T[live] > t_stop) & (t_curr[live] < t_max)]
        if live.numel() == 0:
            break
        first = (t[live] <= t_curr[live, None]).sum(1)
        n = torch.minimum(count[live] - first, torch.full_like(first, k))
        last = t[live, (first + k - 1).clamp(max=most - 1)] + 1e-4
        for e in range(int(n.max()) if n.numel() else 0):
            on = n > e
            r = live[on]
            p = idx[r, first[on] + e]
            m = P["mu"][p] - o
            Ad = torch.einsum("nij,nj->ni", A[p], d[r])
            tau = (m * Ad).sum(1) / (d[r] * Ad).sum(1)
            q = tau[:, None] * d[r] - m
            a = P["opacity"][p] * torch.exp(-torch.einsum("ni,nij,nj->n", q, A[p], q))
            a = torch.where(a > alpha_min, a, torch.zeros_like(a))
            rgb = rgb.index_add(0, r, (T[r] * a)[:, None] * colour[p])
            T = T.index_put((r,), T[r] * (1.0 - a))
        t_curr = t_curr.index_put((live,), torch.where(n == k, last, torch.full_like(last, t_max)))
    return torch.cat([rgb, torch.ones(n_rays, 1, dtype=torch.float64, device="cuda")], 1)


def _params(raw):
    """Activated parameters: the 32-bit ones of the records in 64 bits."""
    rec = _packed(raw)
    P = {"mu": rec[:, 0:3], "scale": rec[:, 4:7], "rot": rec[:, 8:12], "opacity": rec[:, 12],
         "sh": rec[:, 16:80].view(-1, 16, 4)[:, :, :3]}
    return {k: v.double().clone() for k, v in P.items()}


def _grad_rows(P):
    return torch.cat([P["mu"].grad.T, P["scale"].grad.T, P["rot"].grad.T, P["opacity"].grad[None],
                      P["sh"].grad.reshape(-1, 48).T], 0)


def _exact_image(P, case, u, w, h):
    o, d, t_min, t_max = _rays(u, w, h)
    with torch.no_grad():
        idx, t = _hits(P, o, d, t_min, t_max, float(case["alpha_min"]))
    return _composite(P, case, o, d, idx, t, t_min, t_max).view(h, w, 4)


def exact(case, seed):
    kind, w, h = case["kind"], case["w"], case["h"]
    rays = w * h * (case["views"] if kind in ("train_batch", "batch") else 1)
    if rays * case["n"] > (_PAIR_LIMIT / 4 if kind.startswith("train") else _PAIR_LIMIT):
        return None
    if kind == "frame":
        return _exact_image(_params(_raw(case, seed)), case, _uniforms(case, w, h, seed), w, h)
    if kind == "scene":
        return {"image": _exact_image(_params(_raw(case, seed)), case, _uniforms(case, w, h, seed), w, h),
                "kept": None}
    if kind == "batch":
        P = [_params(_raw(dict(case, n=case["n"] // (i + 1)), seed + 7919 * i)) for i in range(case["scenes"])]
        return [_exact_image(P[i % case["scenes"]], case, _uniforms(case, ww, hh, seed, i), ww, hh)
                for i, (ww, hh) in enumerate(_view_sizes(case))]
    if kind not in ("train", "train_batch"):
        return None
    P = {k: v.requires_grad_() for k, v in _params(_raw(case, seed)).items()}
    s = prepare(case, seed)
    torch.cuda.synchronize()
    if kind == "train":
        img = _exact_image(P, case, s.u, w, h)
        loss = ((img - s.target.double())[..., :3] ** 2).sum()
        loss.backward()
        return {"grad": _grad_rows(P), "image": img.detach(), "loss": float(loss)}
    for _, u, ww, hh, dl in s.views:
        img = _exact_image(P, case, u, ww, hh)
        (img * torch.from_numpy(dl).cuda()).sum().backward()
    return _grad_rows(P)
