"""The work that users of this package have it do, as cases to be timed.

A case is a dict of plain values; ``kind`` says which of the calls below it
is, the rest are sizes and options.  ``listed`` names twelve of them, ``draw``
gives more of the same ranges, ``prepare`` makes what a program has in hand
before the call, ``run`` is one pass, ``work`` its compulsory bytes and
arithmetic, ``exact`` the same outputs in 64 bits by plain torch where the
call is a computation that can be restated (the sampler's descents cannot:
they are draws from its own tree).
"""
import math

import torch

from unbiased_differentiable_splatting_gb300 import proposal, scenes
from unbiased_differentiable_splatting_gb300.cudaExtensions import pixelgather, sampling
from unbiased_differentiable_splatting_gb300.regularizers import NearestSamplesRegularizer
from unbiased_differentiable_splatting_gb300.render import MultiViewSplatting, RenderOptions, Splatting
from unbiased_differentiable_splatting_gb300.training import L1ImageLoss, L2ImageLoss, SplatAdam

DEV = "cuda:0"
ROOM_VIEWS = "16x640x480"
FEATURE_VIEWS = "8x256x256,4x128x128,4x512x512,4x1024x768"


def listed():
    return [
        # shape optimisation of a coarse proxy at thumbnail size: the smallest
        # step, where launches and host work count
        dict(name="step_sphere4k_128", kind="step", scene="sphere", n=4096, w=128, h=128, k=8, shading="forward",
             unit=1.0),
        # one iteration of shape optimisation at the usual working size; the
        # scene in units that leave the EWA weights below their clamp, so that
        # positions and std-devs receive gradients
        dict(name="step_harmonic100k_512", kind="step", scene="harmonic", n=100_000, w=512, h=512, k=8,
             shading="forward", unit=60.0),
        # the size of the benchmark's default workload
        dict(name="step_harmonic500k_1024", kind="step", scene="harmonic", n=500_000, w=1024, h=1024, k=8,
             shading="forward", unit=1.0),
        # deferred shading at an odd size and sample count: the EWA,
        # compositing, interpolation and shading ops one by one
        dict(name="step_deferred20k_403x301", kind="step", scene="harmonic", n=20_011, w=403, h=301, k=13,
             shading="deferred", unit=60.0),
        # pose and scene refinement in a room: 16 views of 2M splats per step
        dict(name="views_room2m_16", kind="views", scene="room", n=2_000_000, views=ROOM_VIEWS, k=8, c=3),
        # feature images of a batch of views of four resolutions, no shading
        dict(name="views_features300k_20", kind="views", scene="features", n=300_000, views=FEATURE_VIEWS, k=8, c=8),
        # the renderer's default number of samples: what a preview or an
        # evaluation draws per pixel
        dict(name="sample_k40_60k_427x320", kind="sample", n=60_000, w=427, h=320, k=40),
        # mass-proportional draws with their path probabilities (importance
        # weighted estimators)
        dict(name="stochastic_500k_1024", kind="stochastic", n=500_000, w=1024, h=1024, k=8),
        # EWA, compositing and interpolation of given sample lists, forward
        # and backward, at a ragged size
        dict(name="render_1001x763", kind="render", n=200_003, w=1001, h=763, k=8, c=3),
        # per-sample attributes and reproducible per-splat sums (visibility
        # and feature accumulation)
        dict(name="gather_1024x768", kind="gather", n=300_000, w=1024, h=768, k=8, c=3),
        # what follows a render in the optimisation loop: neighbour lists and
        # their regulariser, image loss, Adam with its projection
        dict(name="tail_200k_512", kind="tail", n=200_000, w=512, h=512, k=8, m=10),
        # a few training steps of the learned proposal, and its evaluation
        dict(name="proposal_65536", kind="proposal", rows=400_000, batch=65536, steps=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step", "views", "sample", "stochastic", "render", "gather", "tail", "proposal"))
    if kind == "step":
        shading = rng.choice(("forward", "forward", "deferred", "None"))
        k = rng.choice((4, 8, 8, 8, 13, 16))
        side = 1024 if k <= 8 else 512
        scene = rng.choice(("sphere", "harmonic"))
        return dict(kind=kind, scene=scene, n=_log(rng, 4096, 20_000 if scene == "sphere" else 500_000),
                    w=_log(rng, 128, side), h=_log(rng, 128, side), k=k, shading=shading,
                    unit=rng.choice((1.0, 60.0)))
    if kind == "views":
        scene = rng.choice(("room", "features"))
        groups = ["%dx%dx%d" % (rng.randint(1, 4), _log(rng, 128, 640), _log(rng, 128, 480))
                  for _ in range(rng.randint(1, 4))]
        return dict(kind=kind, scene=scene, n=_log(rng, 100_000, 2_000_000) if scene == "room" else
                    _log(rng, 50_000, 300_000), views=",".join(groups), k=rng.choice((4, 8, 8)),
                    c=3 if scene == "room" else rng.choice((3, 8)))
    if kind == "sample":
        k = rng.choice((1, 4, 8, 16, 24, 40))
        side = 1024 if k <= 8 else 400
        return dict(kind=kind, n=_log(rng, 5000, 300_000), w=_log(rng, 128, side), h=_log(rng, 128, side), k=k)
    if kind == "stochastic":
        return dict(kind=kind, n=_log(rng, 10_000, 500_000), w=_log(rng, 128, 1024), h=_log(rng, 128, 1024),
                    k=rng.choice((4, 8, 8)))
    if kind in ("render", "gather", "tail"):
        c = dict(kind=kind, n=_log(rng, 10_000, 400_000), w=_log(rng, 128, 1024), h=_log(rng, 128, 1024),
                 k=rng.choice((4, 8, 8, 11)))
        c.update(dict(m=rng.choice((4, 8, 10))) if kind == "tail" else dict(c=rng.choice((1, 3, 4, 8))))
        return c
    return dict(kind="proposal", rows=_log(rng, 50_000, 1_000_000), batch=_log(rng, 4096, 65536),
                steps=rng.randint(1, 6))


# ------------------------------------------------------------------ scenes
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1_000_003 + 17)


def _rand(g, *shape, lo=0.0, hi=1.0):
    return torch.rand(shape, generator=g, device=DEV) * (hi - lo) + lo


def _directions(g, n):
    d = torch.randn((n, 3), generator=g, device=DEV)
    return d / d.norm(dim=1, keepdim=True)


def _surface(kind, n, g, unit):
    """points, normals, std-devs of a closed surface about the origin: a
    sphere with radial jitter, or a star-shaped surface 0.6 (1 + 0.2 sum of
    low harmonics) with its own normals."""
    d = _directions(g, n)
    if kind == "sphere":
        p = d * (0.5 + 0.01 * torch.randn((n, 1), generator=g, device=DEV))
        return p * unit, d, torch.full((n, 2), 0.005 * unit, device=DEV)
    c = _rand(g, 6, lo=-1.0, hi=1.0)

    def field(q):  # |q| - r(direction): zero on the surface
        r = q.norm(dim=1)
        x, y, z = (q / r[:, None]).unbind(1)
        s = (c[0] * x * y + c[1] * y * z + c[2] * x * z + c[3] * (x * x - y * y) / 2 + c[4] * (3 * z * z - 1) / 2
             + c[5] * 2 * x * y * z)
        return r - 0.6 * (1 + 0.2 * s)

    p = d * (d.norm(dim=1) - field(d))[:, None]
    q = p.clone().requires_grad_(True)
    (grad,) = torch.autograd.grad(field(q).sum(), q)
    sd = _rand(g, n, 2, lo=0.003, hi=0.01)
    return p * unit, grad / grad.norm(dim=1, keepdim=True), sd * unit


def _room(n, g):
    """Splats on the inner walls of a 5 x 5 x 3 room and on 40 boxes, in
    proportion to area."""
    lx, ly, lz = 5.0, 5.0, 3.0
    faces = [((0, 0, 0), (lx, 0, 0), (0, ly, 0), (0, 0, 1)), ((0, 0, lz), (lx, 0, 0), (0, ly, 0), (0, 0, -1)),
             ((0, 0, 0), (lx, 0, 0), (0, 0, lz), (0, 1, 0)), ((0, ly, 0), (lx, 0, 0), (0, 0, lz), (0, -1, 0)),
             ((0, 0, 0), (0, ly, 0), (0, 0, lz), (1, 0, 0)), ((lx, 0, 0), (0, ly, 0), (0, 0, lz), (-1, 0, 0))]
    u = _rand(g, 40, 5).tolist()
    for a, b, e, q, r in u:
        sx, sy, sz = 0.2 + 0.6 * a, 0.2 + 0.6 * b, 0.2 + 0.6 * e
        x, y = 0.2 + q * (lx - 0.4 - sx), 0.2 + r * (ly - 0.4 - sy)
        faces += [((x, y, sz), (sx, 0, 0), (0, sy, 0), (0, 0, 1)), ((x, y, 0), (sx, 0, 0), (0, 0, sz), (0, -1, 0)),
                  ((x, y + sy, 0), (sx, 0, 0), (0, 0, sz), (0, 1, 0)), ((x, y, 0), (0, sy, 0), (0, 0, sz), (-1, 0, 0)),
                  ((x + sx, y, 0), (0, sy, 0), (0, 0, sz), (1, 0, 0))]
    f = torch.tensor(faces, device=DEV)  # (faces, 4, 3): origin, two edges, normal
    area = torch.linalg.cross(f[:, 1], f[:, 2]).norm(dim=1).cumsum(0)
    at = torch.searchsorted(area, _rand(g, n) * area[-1]).clamp_max(len(faces) - 1)
    ab = _rand(g, n, 2)
    p = f[at, 0] + ab[:, :1] * f[at, 1] + ab[:, 1:] * f[at, 2]
    return p, f[at, 3].contiguous(), _rand(g, n, 2, lo=0.005, hi=0.02)


def _views(text):
    out = []
    for group in text.split(","):
        count, w, h = (int(v) for v in group.split("x"))
        out += [(w, h)] * count
    return out


def _front(distance):
    return torch.tensor([[0.0, 0.0, -distance]], device=DEV), torch.tensor([[0.0, 0.0, 0.0, 1.0]], device=DEV)


def _lights(b):
    d = torch.tensor([0.3, 0.4, 1.0], device=DEV)
    d = d / d.norm()
    return dict(ambient=torch.full((1, 1, 3), 0.1, device=DEV), lamps=d.repeat(b, 1, 1),
                power=torch.ones((1, 1, 3), device=DEV))


def _cloud(case, g):
    """One closed surface seen from the front: camera-space points, normals
    facing the camera, std-devs (the sampler's inputs) and focal length."""
    p, n, sd = _surface("harmonic", case["n"], g, 1.0)
    p = p + torch.tensor([0.0, 0.0, -2.0], device=DEV)
    n = torch.where(n[:, 2:] > 0, -n, n)
    return p[None].contiguous(), n[None].contiguous(), sd[None], scenes.focal_from_fov(case["w"])


def _lists(case, seed):
    """A rendered surface as the sampler hands it over, made without it: splats
    on a wavy sheet in front of the camera, in the random order of a point
    cloud, and for each pixel of a disc (the rest is background, all -1) up
    to K distinct splats from its neighbourhood."""
    g = _generator(seed)
    n, w, h, k = case["n"], case["w"], case["h"], case["k"]
    f = scenes.focal_from_fov(w)
    side = max(int(math.sqrt(n)), 8)
    grid_h = max(n // side, 8)
    order = torch.randperm(side * grid_h, generator=g, device=DEV)
    u = torch.arange(side, device=DEV).repeat_interleave(grid_h) + _rand(g, side * grid_h)
    v = torch.arange(grid_h, device=DEV).repeat(side) + _rand(g, side * grid_h)
    sx, sy = u * (w / side), v * (h / grid_h)
    unit = 0.16 * w
    z = -unit * (2.0 + 0.2 * torch.sin(sx * (9.0 / w)) * torch.cos(sy * (7.0 / h))
                 + 0.02 * torch.randn(side * grid_h, generator=g, device=DEV))
    p = torch.stack([(sx - w / 2) * -z / f, -(sy - h / 2) * -z / f, z], 1)
    nrm = torch.tensor([0.0, 0.0, -1.0], device=DEV) + 0.3 * torch.randn((side * grid_h, 3), generator=g, device=DEV)
    nrm[:, 2] = -nrm[:, 2].abs().clamp_min(0.3)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    pts, nn = torch.empty_like(p), torch.empty_like(nrm)
    pts[order], nn[order] = p, nrm
    m = side * grid_h
    sd = _rand(g, m, 2, lo=0.35, hi=0.8)
    # 23 cells around the pixel's own, in a stride of its own per pixel (23 is
    # prime, so the K cells are distinct)
    ring = torch.tensor([(a, b) for a in range(-2, 3) for b in range(-2, 3)][1:24], device=DEV)
    px = torch.arange(w, device=DEV).view(w, 1).expand(w, h)
    py = torch.arange(h, device=DEV).view(1, h).expand(w, h)
    start = torch.randint(0, 23, (w, h), generator=g, device=DEV)
    step = torch.randint(1, 23, (w, h), generator=g, device=DEV)
    at = ring[(start[..., None] + step[..., None] * torch.arange(k, device=DEV)) % 23]
    cx = (px * side // w)[..., None] + at[..., 0]
    cy = (py * grid_h // h)[..., None] + at[..., 1]
    inside = (cx >= 0) & (cx < side) & (cy >= 0) & (cy < grid_h)
    disc = ((px - w / 2) / (0.35 * w)) ** 2 + ((py - h / 2) / (0.35 * h)) ** 2 < 1
    full = torch.randint(0, 8, (w, h), generator=g, device=DEV)  # silhouettes leave lists partly empty
    count = torch.where(full == 0, torch.randint(0, k + 1, (w, h), generator=g, device=DEV), torch.full_like(full, k))
    keep = inside & disc[..., None] & (torch.arange(k, device=DEV) < count[..., None])
    idx = torch.where(keep, order[(cx.clamp(0, side - 1) * grid_h + cy.clamp(0, grid_h - 1))], -1).to(torch.int32)
    return dict(w=w, h=h, k=k, f=f, n=m, idx=idx[None].contiguous(), pts=pts[None], nrm=nn[None], sd=sd[None], g=g)


# ----------------------------------------------------------------- prepare
def _prepare_step(case, seed):
    g = _generator(seed)
    unit = case["unit"]
    p, n, sd = _surface(case["scene"], case["n"], g, unit)
    col = _rand(g, case["n"], 3, lo=0.2, hi=0.9)
    pos, quat = _front(2.0 * unit)
    w, h = case["w"], case["h"]
    opts = RenderOptions(forward="-z", numSamples=case["k"], precision=0.01, shadingMode=case["shading"])
    r = Splatting(opts, None, w, h, scenes.focal_from_fov(w), 0.1, 100.0, 0.0).to(DEV)
    r.sample_kwargs = {"seed": 1000 + int(seed)}
    params = [t.contiguous().requires_grad_(True) for t in (pos, quat, p[None], n[None], sd[None], col[None])]
    return dict(case=case, render=r, params=params, light=_lights(1), loss=L2ImageLoss(),
                target=_rand(g, 1, w, h, 3))


def _prepare_views(case, seed):
    g = _generator(seed)
    sizes = _views(case["views"])
    b = len(sizes)
    room = case["scene"] == "room"
    if room:
        p, n, sd = _room(case["n"], g)
        cams = scenes.room_scene(n=64, views=b, seed=int(seed))
        pos, quat = cams["cam_positions"].to(DEV), cams["cam_orientations"].to(DEV)
        views = [(w, h, 525.0 * w / 640) for w, h in sizes]
        attr = _rand(g, case["n"], case["c"], lo=0.2, hi=0.9)
    else:
        p, n, _ = _surface("harmonic", case["n"], g, 1.0)
        sd = torch.full((case["n"], 2), 0.005, device=DEV)
        pos, quat = (t.to(DEV) for t in scenes.orbit_cameras(b, distance=2.0, seed=int(seed)))
        views = [(w, h, scenes.focal_from_fov(w)) for w, h in sizes]
        attr = torch.randn((case["n"], case["c"]), generator=g, device=DEV)
    opts = RenderOptions(forward="-z", numSamples=case["k"], precision=0.01,
                         shadingMode="forward" if room else "None")
    r = MultiViewSplatting(opts, None, views, 0.1, 100.0, 0.0).to(DEV)
    r.sample_kwargs = {"seed": 1000 + int(seed)}
    params = [t.contiguous().requires_grad_(True) for t in (pos, quat, p[None], n[None], sd[None], attr[None])]
    return dict(case=case, render=r, params=params, light=_lights(b),
                targets=[_rand(g, 1, w, h, case["c"]) for w, h in sizes])


def _prepare_cloud(case, seed):
    g = _generator(seed)
    pts, nrm, sd, f = _cloud(case, g)
    return dict(case=case, pts=pts, nrm=nrm, sd=sd, f=f, seed=1000 + int(seed))


def _prepare_lists(case, seed):
    s = _lists(case, seed)
    g, w, h, k, n = s["g"], s["w"], s["h"], s["k"], s["n"]
    s["case"] = case
    if case["kind"] == "render":
        c = case["c"]
        s["attr"] = _rand(g, 1, n, c, lo=0.2, hi=0.9)
        s["grad"] = torch.randn((1, w, h, c), generator=g, device=DEV)
        s["params"] = [t.contiguous().requires_grad_(True) for t in (s["pts"], s["sd"], s["attr"])]
        s["const"] = s["nrm"].contiguous()
    elif case["kind"] == "gather":
        s["splats"] = torch.randn((1, n, case["c"]), generator=g, device=DEV)
        s["samples"] = torch.randn((1, w, h, k, case["c"]), generator=g, device=DEV)
    else:
        wt = _rand(g, 1, w, h, k)
        s["weights"] = torch.where(s["idx"] >= 0, wt, torch.zeros_like(wt))
        s["params"] = [t.contiguous().clone().requires_grad_(True) for t in
                       (s["pts"], s["nrm"], _rand(g, 1, n, 3), s["sd"])]
        s["grads"] = [torch.randn((1, n, c), generator=g, device=DEV) for c in (3, 2)]
        s["image"] = _rand(g, 1, w, h, 3).requires_grad_(True)
        s["target"] = _rand(g, 1, w, h, 3)
        s["reg"] = NearestSamplesRegularizer(sigma=4.0, num_nearest=case["m"], reduction="mean")
        s["loss"] = L1ImageLoss()
        p = s["params"]
        s["adam"] = SplatAdam(p[0], p[1], p[2], p[3], lr=1e-4, stdDevBound=(0.2, 1.0))
    return s


def _prepare_proposal(case, seed):
    g = _generator(seed)
    x = torch.randn((case["rows"], 16), generator=g, device=DEV).clamp(-4, 4)
    t = torch.sigmoid(2.0 * x[:, 3] - 2.0 * x[:, 9] + 0.5 * torch.randn(case["rows"], generator=g, device=DEV))
    return dict(case=case, x=x, t=t, net=proposal.ProposalNet(DEV, seed=int(seed)))


def prepare(case, seed):
    make = {"step": _prepare_step, "views": _prepare_views, "sample": _prepare_cloud, "stochastic": _prepare_cloud,
            "render": _prepare_lists, "gather": _prepare_lists, "tail": _prepare_lists,
            "proposal": _prepare_proposal}
    return make[case["kind"]](case, seed)


# --------------------------------------------------------------------- run
def _run_step(s):
    pos, quat, pts, nrm, sd, col = s["params"]
    light = s["light"]
    img, idx, depth = s["render"](pos, quat, pts, nrm, sd, col, light["ambient"], light["lamps"], light["power"])
    target = s["target"]
    loss, _ = s["loss"](img, target)
    grads = torch.autograd.grad(loss, s["params"], allow_unused=True)
    return dict(image=img.detach(), indices=idx, depth=depth.detach(), loss=loss.detach(), grads=list(grads))


def _run_views(s):
    pos, quat, pts, nrm, sd, attr = s["params"]
    light = s["light"]
    imgs, idx, _ = s["render"](pos, quat, pts, nrm, sd, attr, light["ambient"], light["lamps"], light["power"])
    loss = sum(((a - b) ** 2).sum() for a, b in zip(imgs, s["targets"]))
    grads = torch.autograd.grad(loss, s["params"], allow_unused=True)
    return dict(images=[i.detach() for i in imgs], indices=idx, loss=loss.detach(), grads=list(grads))


def _run_sample(s):
    c = s["case"]
    return sampling.sample(c["w"], c["h"], s["f"], s["pts"], s["nrm"], None, s["sd"], c["k"], 0.0, 0.01,
                           seed=s["seed"])


def _run_stochastic(s):
    c = s["case"]
    return sampling.sample_stochastic(c["w"], c["h"], s["f"], s["pts"], s["nrm"], s["sd"], c["k"], 0.0, 0.01,
                                      seed=s["seed"])


def _run_render(s):
    pts, sd, attr = s["params"]
    img, depth, ewa = torch.ops.uds.render_splats(s["w"], s["h"], s["f"], s["idx"], pts, s["const"], sd, 0.0, attr)
    grads = torch.autograd.grad(img, s["params"], grad_outputs=s["grad"])
    return dict(image=img.detach(), depth=depth.detach(), ewa=ewa.detach(), grads=list(grads))


def _run_gather(s):
    return dict(scattered=pixelgather.scatter(s["idx"], s["splats"]),
                gathered=pixelgather.gather(s["idx"], s["samples"], s["n"], deterministic=True))


def _run_tail(s):
    pts, nrm, col, sd = s["params"]
    normal, plane = s["reg"](s["idx"], s["weights"], pts, nrm)
    gp, gn = torch.autograd.grad(normal + plane, (pts, nrm))
    loss, _ = s["loss"](s["image"], s["target"])
    (gi,) = torch.autograd.grad(loss, s["image"])
    pts.grad, nrm.grad, col.grad, sd.grad = gp, gn, s["grads"][0], s["grads"][1]
    s["adam"].step()
    return dict(losses=[normal.detach(), plane.detach(), loss.detach()], gi=gi, gp=gp, gn=gn,
                params=[p.detach() for p in s["params"]], moments=[s["adam"].m, s["adam"].v])


def _run_proposal(s):
    losses = s["net"].train(s["x"], s["t"], steps=s["case"]["steps"], batch=s["case"]["batch"])
    return dict(losses=losses, params=s["net"].params, logits=s["net"].logits(s["x"]))


def run(state):
    call = {"step": _run_step, "views": _run_views, "sample": _run_sample, "stochastic": _run_stochastic,
            "render": _run_render, "gather": _run_gather, "tail": _run_tail, "proposal": _run_proposal}
    return call[state["case"]["kind"]](state)


# -------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "proposal":
        macs = 16 * 64 + 2 * 64 * 64 + 64 * 2
        return {"bytes": 4.0 * (case["steps"] * case["batch"] * 17 + case["rows"] * 18),
                "flops": 2.0 * macs * (3 * case["steps"] * case["batch"] + case["rows"])}
    n, k = case["n"], case["k"]
    sizes = _views(case["views"]) if kind == "views" else [(case["w"], case["h"])]
    px = sum(w * h for w, h in sizes)
    b = len(sizes)
    if kind in ("step", "views"):
        c = case.get("c", 3)
        # splat attributes read and their gradients written; per view every
        # splat's position is needed to place it; images, targets, sample
        # lists and depth weights
        per = 4.0 * n * (8 + c) * 2 + 4.0 * b * n * 3 + px * (4.0 * 2 * c + 8.0 * k)
        return {"bytes": per, "flops": px * k * (150.0 + 6 * c) + 200.0 * b * n}
    if kind == "sample":
        return {"bytes": 32.0 * n + 4.0 * px * k, "flops": 200.0 * n + 50.0 * px * k}
    if kind == "stochastic":
        return {"bytes": 32.0 * n + 8.0 * px * k, "flops": 200.0 * n + 50.0 * px * k}
    if kind == "render":
        c = case["c"]
        return {"bytes": px * (4.0 * k * 3 + 8.0 * c) + 4.0 * n * (3 + 3 + 2 + c + 5 + c),
                "flops": px * k * (150.0 + 6 * c) + 200.0 * n}
    if kind == "gather":
        c = case["c"]
        return {"bytes": px * k * (4.0 + 8.0 * c) + 8.0 * n * c, "flops": px * k * float(c)}
    # image and target read, its gradient written; sample lists and weights;
    # points, normals, colours, std-devs with gradients and two moments each
    # read, parameters and moments written
    return {"bytes": px * (36.0 + 8.0 * k) + 4.0 * n * (11 * 7 + case["m"] * 6 + 6), "flops": 60.0 * n * case["m"]}


# ------------------------------------------------------------------- exact
def _exact_render(case, seed):
    s = _prepare_lists(case, seed)
    pts, sd, attr = (t.detach()[0].double().requires_grad_(True) for t in s["params"])
    nrm = s["const"][0].double()
    w, h, f, idx = s["w"], s["h"], s["f"], s["idx"][0].long()
    sx, sy = -pts[:, 0] * f / pts[:, 2] + w / 2, pts[:, 1] * f / pts[:, 2] + h / 2

    def ray(x, y):  # through a screen point, z = 1
        return torch.stack([(w - 2 * x) / (2 * f), -(h - 2 * y) / (2 * f), torch.ones_like(x)], -1)

    def tangent(x):
        return x * ((pts * nrm).sum(-1) / (x * nrm).sum(-1))[:, None] - pts

    t0, t1 = tangent(ray(sx + 1, sy)), tangent(ray(sx, sy + 1))
    al = t0.norm(dim=1)
    u0 = t0 / al[:, None]
    u1 = torch.linalg.cross(u0, nrm)
    be, ga = (t1 * u0).sum(1), (t1 * u1).sum(1)
    j00, j01, j11 = 1 / al, -be / (al * ga), 1 / ga
    a, b = sd[:, 0] ** 2, sd[:, 1] ** 2
    v00, v01, v11 = j00 * j00 * a + j01 * j01 * b, j01 * j11 * b, j11 * j11 * b
    det = v00 * v11 - v01 * v01
    z = 2 * math.pi * det.sqrt() * (al * ga).abs()
    table = torch.stack([sx, sy, v11 / det, -v01 / det, v00 / det, z], 1)
    pn = (pts.detach() * nrm).sum(1)
    px = torch.arange(w, device=DEV, dtype=torch.float64)
    py = torch.arange(h, device=DEV, dtype=torch.float64)
    images, depths, ewas = [], [], []
    total = 0.0
    for i0 in range(0, w, 128):  # columns of pixels at a time
        ids = idx[i0:i0 + 128]
        ok = ids >= 0
        at = ids.clamp_min(0)
        x, y = torch.meshgrid(px[i0:i0 + 128], py, indexing="ij")
        q = table[at]
        dx, dy = x[..., None] - q[..., 0], y[..., None] - q[..., 1]
        e = dx * dx * q[..., 2] + 2 * dx * dy * q[..., 3] + dy * dy * q[..., 4]
        wt = torch.where(ok, (torch.exp(-0.5 * e) / q[..., 5]).clamp_max(1.0), torch.zeros_like(e))
        d = ray(x, y)
        d = -d / d.norm(dim=-1, keepdim=True)
        dist = pn[at] / (d[:, :, None] * nrm[at]).sum(-1)
        dist = torch.where(ok & (dist > 0), dist, torch.full_like(dist, 10000.0))
        order = dist.argsort(dim=-1, stable=True)
        ws = wt.gather(-1, order)
        rem = torch.cat([torch.ones_like(ws[..., :1]), (1 - ws).cumprod(-1)[..., :-1]], -1)
        fw = torch.zeros_like(ws).scatter(-1, order, rem * ws)
        img = (fw[..., None] * attr[at] * ok[..., None]).sum(2)
        images.append(img.detach())
        depths.append(fw.detach())
        ewas.append(wt.detach())
        total = total + (img * s["grad"][0, i0:i0 + 128].double()).sum()
    gp, gs, ga_ = torch.autograd.grad(total, (pts, sd, attr))
    gp, gs = (t / (t.norm(dim=1, keepdim=True) + 1e-4).clamp_min(1.0) for t in (gp, gs))
    return dict(image=torch.cat(images)[None], depth=torch.cat(depths)[None], ewa=torch.cat(ewas)[None],
                grads=[gp[None], gs[None], ga_[None]])


def _exact_gather(case, seed):
    s = _prepare_lists(case, seed)
    at = s["idx"].reshape(-1).long()
    ok = at >= 0
    c = case["c"]
    out = torch.zeros((at.numel(), c), device=DEV, dtype=torch.float64)
    out[ok] = s["splats"][0].double()[at[ok]]
    got = torch.zeros((s["n"], c), device=DEV, dtype=torch.float64)
    got.index_add_(0, at[ok], s["samples"].reshape(-1, c)[ok].double())
    return dict(scattered=out.view(1, s["w"], s["h"], s["k"], c), gathered=got[None])


def _exact_tail(case, seed):
    s = _prepare_lists(case, seed)
    pts, nrm, col, sd = (t.detach()[0].double() for t in s["params"])
    n, m, k = s["n"], case["m"], s["k"]
    ids, wt = s["idx"].reshape(-1, k).long(), s["weights"].reshape(-1, k)
    best = wt.max(1, keepdim=True).values
    first = torch.where(wt == best, torch.arange(k, device=DEV), k).min(1, keepdim=True).values
    top = ids.gather(1, first)
    ok = (ids >= 0) & (top >= 0) & (ids != top)
    pair = torch.unique((top * n + ids)[ok])
    i, j = pair // n, pair % n
    by = (pts[i] - pts[j]).norm(dim=1).argsort(stable=True)
    by = by[i[by].argsort(stable=True)]
    i, j = i[by], j[by]
    rank = torch.arange(i.numel(), device=DEV) - torch.searchsorted(i, i)
    keep = (rank < m) & (j > 0)
    i, j = i[keep], j[keep]
    dp, dn = pts[i] - pts[j], nrm[i] - nrm[j]
    wgt = torch.exp(-((dp * dp).sum(1) + (dn * dn).sum(1)) / 16.0)
    zero = torch.zeros(n, device=DEV, dtype=torch.float64)
    a = zero.index_add(0, i, wgt)
    d = zero.index_add(0, i, wgt * (dp * nrm[j]).sum(1))
    fl = torch.zeros((n, 3), device=DEV, dtype=torch.float64).index_add(0, i, wgt[:, None] * nrm[j])
    some = (zero.index_add(0, i, torch.ones_like(wgt)) > 0).double()
    x = d / (a + 1e-4)
    e = (fl / (fl.norm(dim=1, keepdim=True) + 1e-4) - nrm) * some[:, None]
    gp, gn = 2 * (x / (a + 1e-4))[:, None] * fl / n, -2 * e / n
    diff = s["image"].detach().double() - s["target"].double()
    grads = [gp, gn, s["grads"][0][0].double(), s["grads"][1][0].double()]
    new = [p - 1e-4 * g / (g.abs() + 1e-8) for p, g in zip((pts, nrm, col, sd), grads)]  # Adam's first step
    new[1] = new[1] / (new[1].norm(dim=1, keepdim=True) + 1e-4)
    new[3] = new[3].clamp(0.2, 1.0)
    return dict(losses=[(e * e).sum() / n, (x * x).sum() / n, diff.abs().mean()], gi=diff.sign() / diff.numel(),
                gp=gp[None], gn=gn[None], params=[t[None] for t in new],
                moments=[torch.cat([0.1 * g.reshape(-1) for g in grads]),
                         torch.cat([0.001 * (g * g).reshape(-1) for g in grads])])


def _exact_proposal(case, seed):
    s = _prepare_proposal(case, seed)
    flat = s["net"].params.double().requires_grad_(True)
    x, t = s["x"].double(), s["t"].double()

    def logits(p, rows):
        at, hidden = 0, rows
        for q, (out, inp) in enumerate(((64, 16), (64, 64), (64, 64), (16, 64))):
            wq = p[at:at + out * inp].view(out, inp)
            bq = p[at + out * inp:at + out * inp + out]
            at += out * inp + out
            hidden = hidden @ wq.t() + bq
            hidden = torch.relu(hidden) if q < 3 else hidden
        return hidden[:, :2]

    g = torch.Generator(device=DEV).manual_seed(0)
    m1, m2, losses = torch.zeros_like(flat), torch.zeros_like(flat), []
    for step in range(1, case["steps"] + 1):
        rows = min(case["batch"], x.shape[0])
        sel = torch.randint(0, x.shape[0], (rows,), device=DEV, generator=g)
        lp = torch.log_softmax(logits(flat, x[sel]), dim=1)
        loss = -(t[sel] * lp[:, 0] + (1 - t[sel]) * lp[:, 1]).mean()
        (grad,) = torch.autograd.grad(loss, flat)
        losses.append(loss.detach())
        m1, m2 = 0.9 * m1 + 0.1 * grad, 0.999 * m2 + 0.001 * grad * grad
        new = flat - 3e-3 * (m1 / (1 - 0.9 ** step)) / ((m2 / (1 - 0.999 ** step)).sqrt() + 1e-8)
        flat = new.detach().requires_grad_(True)
    return dict(losses=torch.stack(losses), params=flat.detach(), logits=logits(flat, x).detach())


def exact(case, seed):
    call = {"render": _exact_render, "gather": _exact_gather, "tail": _exact_tail, "proposal": _exact_proposal}
    return call[case["kind"]](case, seed) if case["kind"] in call else None
