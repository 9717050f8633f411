"""Measured work of the rasterizer: the calls that programs make, over the sizes they make them at.

Each case is a dict of plain values; ``prepare`` builds what a program holds before the call (a mesh, its
features, cameras, ray jitter, a batch object), ``run`` makes the call through the package's public entry
points, ``work`` counts the bytes and operations it cannot do without, and ``exact`` gives the same outputs in
64-bit plain torch where that is quick.  The kinds:

  frame     ``render.rasterize`` without gradients: a viewer's or an evaluation's frame.
  step      the drop-in's training step on given cell values: projection, lists, blend, L1 loss, gradients.
  render    the reference's training iteration: ``render()`` with a model whose cell values come from
            ``activate_output``, L1 plus distortion loss, gradients of every parameter.
  views     ``batch.L1Step``: several cameras of one mesh in one captured step, forward and backward.
  serve     ``batch.BatchedRasterizer.forward`` on a resident mesh with packed records: a server's batch.
  err       ``render_err``: the densification statistics of one training view.
  features  ``activate_output`` alone, forward and backward.
  tets      ``orient_tets`` and ``cull_tets``: the GPU part of a Delaunay update.

Points are uniform in a cube (plain renders), uniform in a ball (gradient checks), or a mixture of anisotropic
Gaussians with a uniform background (captured scenes: tile lists with a heavy tail); 30% of a mixture's
tets are nearly empty.  A seed turns the mesh about the vertical axis and draws features, jitter and targets.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from radiance_meshes_b200 import batch as B
from radiance_meshes_b200 import delaunay as D
from radiance_meshes_b200 import features as F
from radiance_meshes_b200 import render as RR
from radiance_meshes_b200 import scenes
from radiance_meshes_b200.camera import tcam_to_struct
from radiance_meshes_b200.delaunay_rasterization.internal.alphablend_tiled_slang_interp import AlphaBlendTiledRender
from radiance_meshes_b200.delaunay_rasterization.internal.render_err import render_err
from radiance_meshes_b200.delaunay_rasterization.internal.render_grid import RenderGrid
from radiance_meshes_b200.delaunay_rasterization.internal.tile_shader_slang import vertex_and_tile_shader

DEV = "cuda"
TETS_PER_POINT = 6.6  # Delaunay tets per vertex of these clouds
MIXED = [(840, 1297), (1080, 1920), (840, 1297), (480, 640)]  # resolutions of a batch, in turn
SERVED = [(480, 640), (720, 1280), (1080, 1920)]


def listed():
    return [
        # the smallest frame a user renders (a viewer's thumbnail, a test): latency and launches
        dict(name="frame_uniform4k_256", kind="frame", cloud="uniform", points=4096, height=256, width=256, tile=16),
        # the smallest training step (gradient checks, toy scenes)
        dict(name="step_ball2k_128", kind="step", cloud="ball", points=2000, height=128, width=128, tile=16, lens=0),
        # an early training iteration of a captured scene, odd image size, SH degree 3, all parameters
        dict(name="render_mix50k_979x545", kind="render", cloud="mix", points=50_000, height=545, width=979, tile=16,
             degree=3),
        # the headline training step: 1.3M tets at 1297x840 with random ray jitter
        dict(name="step_mix200k_1297x840", kind="step", cloud="mix", points=200_000, height=840, width=1297, tile=16,
             lens=0),
        # a full training iteration of the same scene with its SH colours and the distortion loss
        dict(name="render_mix200k_1297x840", kind="render", cloud="mix", points=200_000, height=840, width=1297,
             tile=16, degree=3),
        # a camera with lens distortion on 8x8 tiles (uncorrected photographs)
        dict(name="step_lens30k_640x481", kind="step", cloud="mix", points=30_000, height=481, width=640, tile=8,
             lens=1),
        # a full-HD frame for a viewer or an evaluation
        dict(name="frame_mix200k_1920x1080", kind="frame", cloud="mix", points=200_000, height=1080, width=1920,
             tile=16),
        # the largest step: 16 cameras of a 6.6M-tet mesh in one captured multi-view step
        dict(name="views16_mix1m", kind="views", cloud="mix", points=1_000_000, views=16, tile=16),
        # a server's batch of four requests of mixed resolution
        dict(name="serve4_mix250k", kind="serve", cloud="mix", points=250_000, views=4, tile=16),
        # the densification statistics of one training view
        dict(name="err_mix100k_1297x840", kind="err", cloud="mix", points=100_000, height=840, width=1297, tile=16),
        # the per-tet feature producer alone, forward and backward
        dict(name="features_mix200k_deg3", kind="features", cloud="mix", points=200_000, degree=3),
        # the GPU part of a Delaunay update
        dict(name="tets_mix200k", kind="tets", cloud="mix", points=200_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "step", "step", "step", "render", "render", "views", "serve", "err",
                       "features", "tets"])
    c = dict(kind=kind, cloud="mix", points=_log_int(rng, 4_000, 200_000))
    if kind in ("frame", "step", "render", "err"):
        if kind in ("frame", "step") and rng.random() < 0.4:  # the small clouds and images
            c["cloud"] = rng.choice(["uniform", "ball"])
            c["points"] = _log_int(rng, 1_000, 8_000)
            c["height"], c["width"] = _log_int(rng, 96, 320), _log_int(rng, 96, 320)
        else:
            c["height"] = _log_int(rng, 240, 1080)
            c["width"] = int(c["height"] * rng.uniform(1.0, 1.8))
        c["tile"] = rng.choice([8, 16, 16, 16, 32])
        if kind == "step":
            c["lens"] = rng.choice([0, 0, 0, 1])
        if kind == "render":
            c["degree"] = rng.choice([0, 1, 2, 3])
    elif kind in ("views", "serve"):
        c["views"] = rng.randint(2, 8)
        c["tile"] = 16
    elif kind == "features":
        c["degree"] = rng.choice([0, 1, 2, 3])
    return c


# ------------------------------------------------------------------ inputs --
def _split8(pts, idx):
    """Each tet cut into 8 at its edge midpoints (a conforming refinement)."""
    pts, idx = torch.from_numpy(pts).to(DEV), torch.from_numpy(idx).to(DEV).long()
    ea, eb = (0, 0, 0, 1, 1, 2), (1, 2, 3, 2, 3, 3)
    a, b = idx[:, ea], idx[:, eb]
    lo, hi = torch.minimum(a, b), torch.maximum(a, b)
    uniq, inv = torch.unique((lo * len(pts) + hi).reshape(-1), return_inverse=True)
    mid = 0.5 * (pts[uniq // len(pts)] + pts[uniq % len(pts)])
    m01, m02, m03, m12, m13, m23 = (inv.reshape(-1, 6) + len(pts)).unbind(1)
    v0, v1, v2, v3 = idx.unbind(1)
    kids = [(v0, m01, m02, m03), (m01, v1, m12, m13), (m02, m12, v2, m23), (m03, m13, m23, v3),
            (m01, m02, m03, m13), (m01, m12, m02, m13), (m02, m03, m13, m23), (m02, m13, m12, m23)]
    tets = torch.stack([torch.stack(k, 1) for k in kids], 1).reshape(-1, 4)
    return torch.cat([pts, mid]), tets.int()


@functools.lru_cache(maxsize=6)
def _mesh(cloud, points):
    """Vertices [V,3] and positively oriented tets [T,4] of a cloud, the same for every seed.  Above 200k points
    the Delaunay mesh of an eighth of the points is refined (scipy takes too long there)."""
    n = points if points <= 200_000 else points // 8
    rng = np.random.default_rng(points)
    if cloud == "uniform":
        pts = rng.uniform(-1.0, 1.0, size=(n, 3)).astype(np.float32)
    elif cloud == "ball":
        pts = rng.normal(size=(n, 3))
        pts *= rng.uniform(size=(n, 1)) ** (1.0 / 3.0) / np.linalg.norm(pts, axis=1, keepdims=True)
        pts = pts.astype(np.float32)
    else:
        pts = scenes.mixture_points(n, seed=2)
    idx = scenes.delaunay(pts)
    if n == points:
        return torch.from_numpy(pts).to(DEV), torch.from_numpy(idx).to(DEV)
    v, t = _split8(pts, idx)
    e = v[t.long()]
    neg = (torch.linalg.cross(e[:, 1] - e[:, 0], e[:, 2] - e[:, 0]) * (e[:, 3] - e[:, 0])).sum(1) < 0
    t[neg] = t[neg][:, [1, 0, 2, 3]]
    return v, t.contiguous()


def _gen(seed):
    return torch.Generator(DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _turned(case, seed):
    v, t = _mesh(case["cloud"], case["points"])
    th = 2.0 * math.pi * float(np.random.default_rng(seed).uniform())
    c, s = math.cos(th), math.sin(th)
    rot = torch.tensor([[c, 0.0, s], [0.0, 1.0, 0.0], [-s, 0.0, c]], device=DEV)
    return (v @ rot.T).contiguous(), t.clone()


def _raw(case, n, g):
    """Per-tet density [T,1], colour [T,3] and colour gradient [T,3] with the workloads' distributions."""
    mu, sigma = (0.0, 2.0) if case["cloud"] == "ball" else (-1.0, 1.5)
    density = torch.exp(mu + sigma * torch.randn(n, 1, generator=g, device=DEV))
    if case["cloud"] == "mix":
        density[torch.rand(n, generator=g, device=DEV) < 0.3] = 1e-4
    return density, torch.rand(n, 3, generator=g, device=DEV), 0.1 * torch.randn(n, 3, generator=g, device=DEV)


def _view(case):
    h, w = case["height"], case["width"]
    if case["cloud"] == "uniform":
        return scenes._view((0.0, 0.0, -3.0), (0.0, 0.0, 0.0), h, w, 60.0, case["tile"])
    if case["cloud"] == "ball":
        return scenes._view((0.3, 0.4, -2.9), (0.0, 0.0, 0.0), h, w, 60.0, case["tile"])
    return scenes._view((4.0, 0.5, 0.0), (0.0, 0.0, 0.0), h, w, 60.0, case["tile"])


def _tcam(case):
    tcam = _view(case).tcam(device=DEV)
    if case.get("lens"):
        tcam["distortion_params"] = torch.tensor([0.04, -0.01, 0.001, -0.002], device=DEV)
    return tcam


class _Camera:
    """The attributes of a dataset camera that ``render()`` and ``render_err`` read."""

    def __init__(self, tcam, target):
        keep = ("world_view_transform", "cam_pos", "K", "image_height", "image_width", "fovy", "fovx",
                "distortion_params", "camera_type")
        self._dict = {k: tcam[k] for k in keep}
        self.image_height, self.image_width = tcam["image_height"], tcam["image_width"]
        self.camera_center = tcam["cam_pos"]
        self.original_image = target
        self.gt_alpha_mask = torch.ones((1, self.image_height, self.image_width), device=DEV)

    def to_dict(self, device):
        return dict(self._dict)


class _Model:
    """A per-tet SH model: the fields that ``render()`` and ``render_err`` use."""

    device = DEV
    feature_dim = 7
    mask_values = False

    def __init__(self, vertices, indices, density, rgb, grd, sh, degree):
        self.vertices, self.indices = vertices, indices
        self.density, self.rgb, self.grd, self.sh, self.degree = density, rgb, grd, sh, degree

    def params(self):
        return [self.vertices, self.density, self.rgb, self.grd, self.sh]

    def get_cell_values(self, camera, mask=None, all_circumcenters=None):
        idx, d, c, g, s = self.indices, self.density, self.rgb, self.grd, self.sh
        if mask is not None:
            idx, d, c, g, s = idx[mask], d[mask], c[mask], g[mask], s[mask]
        cc = all_circumcenters
        if cc is None:
            cc = self.vertices[idx.long()].mean(dim=1)
        return s, F.activate_output(camera.camera_center, d, c, g, s, idx, cc, self.vertices, self.degree, 3)


class _State:
    pass


def prepare(case, seed):
    g = _gen(seed)
    s = _State()
    s.kind = kind = case["kind"]
    s.vertices, s.indices = _turned(case, seed)
    T = s.indices.shape[0]
    density, rgb, grd = _raw(case, T, g)
    if kind in ("frame", "step", "render", "err"):
        h, w = case["height"], case["width"]
        s.tcam = _tcam(case)
        s.grid = RenderGrid(h, w, tile_width=case["tile"], tile_height=case["tile"])
        s.target = torch.rand((h, w, 3), generator=g, device=DEV)
        # viewers use the pixel centres, training a random point of each pixel
        s.jitter = None if kind == "frame" else torch.rand((h, w, 2), generator=g, device=DEV)
    if kind in ("frame", "step", "views", "serve"):
        s.values = torch.cat([density, rgb, grd], 1)
    if kind == "step":
        s.vertices.requires_grad_(True)
        s.values.requires_grad_(True)
    if kind in ("render", "features", "err"):
        degree = case.get("degree", 0)
        sh = 0.1 * torch.randn((T, (degree + 1) ** 2 - 1, 3), generator=g, device=DEV)
        s.degree = degree
        s.model = _Model(s.vertices, s.indices, density, rgb, grd, sh, degree)
        if kind != "err":
            for p in s.model.params():
                p.requires_grad_(True)
    if kind in ("render", "err"):
        s.tile = case["tile"]
        s.camera = _Camera(s.tcam, s.target.permute(2, 0, 1).contiguous())
    if kind == "features":
        s.centre = torch.tensor([4.0, 0.5, 0.0], device=DEV)
        s.cc = s.vertices.detach()[s.indices.long()].mean(dim=1).requires_grad_(True)
        s.grad = torch.randn((T, 7), generator=g, device=DEV)
    if kind == "views":
        res = [MIXED[k % 4] for k in range(case["views"])]
        cams = [tcam_to_struct(v.tcam()) for v in scenes.ring_views(case["views"], res, tile_size=case["tile"])]
        batch = B.ViewBatch(cams)
        target = torch.rand((batch.n_pixels, 3), generator=g, device=DEV)
        jitter = torch.rand((batch.n_pixels, 2), generator=g, device=DEV)
        s.rast = B.BatchedRasterizer(s.indices, s.vertices, s.values, batch, jitter=jitter, fine_shift=1)
        s.step = B.L1Step(s.rast, target)
        s.step.capture()
    if kind == "serve":
        rng = np.random.default_rng(seed)
        cams = [tcam_to_struct(scenes.sphere_view(rng, *SERVED[k % 3], tile_size=case["tile"]).tcam())
                for k in range(case["views"])]
        from radiance_meshes_b200.serve import ResidentMesh
        s.mesh = ResidentMesh("mesh", s.indices, s.vertices, s.values, DEV)
        s.rast = B.BatchedRasterizer(s.mesh.indices, s.mesh.vertices, s.mesh.cell_values, B.ViewBatch(cams),
                                     records=s.mesh.records, hit_masks=False, fine_shift=1)
    if kind == "tets":
        flip = torch.rand(T, generator=g, device=DEV) < 0.5  # a tetrahedraliser's mixed orientations
        s.indices[flip] = s.indices[flip][:, [1, 0, 2, 3]]
        hull = torch.randperm(T, generator=g, device=DEV)[:T // 100]  # rows that name the point at infinity
        s.indices[hull, 0] = s.vertices.shape[0]
        s.density = density.reshape(-1)
    return s


# --------------------------------------------------------------------- run --
def run(s):
    if s.kind == "frame":
        with torch.no_grad():
            img, dist, extras = RR.rasterize(s.vertices, s.indices, s.values, s.tcam)
        return dict(img=img, dist=dist, ranges=extras["tile_ranges"], mask=extras["mask"],
                    rect=extras["rect_tile_space"])
    if s.kind == "step":
        ids, ranges, _, _, _, _ = vertex_and_tile_shader(s.indices, s.vertices, s.tcam, s.grid)
        img, dist, _ = AlphaBlendTiledRender.apply(ids, ranges, s.indices, s.vertices, s.values, s.grid, s.tcam,
                                                   s.jitter)
        loss = (img[..., :3] - s.target).abs().mean()
        gv, gc = torch.autograd.grad(loss, [s.vertices, s.values])
        return dict(img=img, dist=dist, loss=loss, grad_vertices=gv, grad_values=gc)
    if s.kind == "render":
        pkg = RR.render(s.camera, s.model, tile_size=s.tile, min_t=0.1, ray_jitter=s.jitter)
        loss = (pkg["render"] - s.camera.original_image).abs().mean() + 1e-3 * pkg["distortion_loss"]
        grads = torch.autograd.grad(loss, s.model.params(), allow_unused=True)
        return dict(render=pkg["render"], alpha=pkg["alpha"], distortion=pkg["distortion_loss"],
                    grads={n: x for n, x in zip(("vertices", "density", "rgb", "grd", "sh"), grads) if x is not None})
    if s.kind == "views":
        loss = s.step.run()
        r = s.rast
        return dict(loss=loss, img=r.img, dist=r.dist, nc=r.nc, grad_vertices=r.grad_vertices,
                    grad_values=r.grad_cell_values)
    if s.kind == "serve":
        img, dist, nc = s.rast.forward()
        return dict(img=img, dist=dist, nc=nc)
    if s.kind == "err":
        err, extras = render_err(s.camera.original_image, s.camera, s.model, tile_size=s.tile, min_t=0.1)
        return dict(err=err, count=extras["tet_count"], pixel=extras["pixel_err"], ssim=extras["ssim_err"],
                    img=extras["render_img"])
    if s.kind == "features":
        m = s.model
        out = F.activate_output(s.centre, m.density, m.rgb, m.grd, m.sh, s.indices, s.cc, s.vertices, s.degree, 3)
        grads = torch.autograd.grad(out, m.params() + [s.cc], s.grad, allow_unused=True)
        return dict(out=out, grads={n: x for n, x in zip(("vertices", "density", "rgb", "grd", "sh", "cc"), grads)
                                    if x is not None})
    if s.kind == "tets":
        idx = D.orient_tets(s.indices, s.vertices)
        kept, empty = D.cull_tets(idx, s.vertices, s.density[:idx.shape[0]], 0.05, 0.01)
        return dict(indices=idx, split=torch.cat([kept, empty]))
    raise ValueError(s.kind)


# -------------------------------------------------------------------- work --
def work(case):
    """Bytes: each input read once, each output and gradient written once.  Operations: a ray crosses about
    T^(1/3) tets before it is opaque or leaves the mesh; a crossing is some 90 operations forward (four planes, two
    quotients, the segment integral, the fold) and 250 backward."""
    V = case["points"]
    T = int(TETS_PER_POINT * V)
    mesh, values = 12 * V + 16 * T, 28 * T
    kind = case["kind"]
    if kind in ("views", "serve"):
        res = MIXED if kind == "views" else SERVED
        px = sum(h * w for h, w in (res[k % len(res)] for k in range(case["views"])))
    else:
        px = case.get("height", 0) * case.get("width", 0)
    crossings = px * T ** (1.0 / 3.0)
    out = 36 * px
    if kind == "frame":
        return dict(bytes=mesh + values + out + 37 * T, flops=90 * crossings)
    if kind == "step":
        return dict(bytes=2 * (mesh + values) + 2 * out + 20 * px, flops=340 * crossings)
    if kind == "render":
        par = 4 * (7 + 3 * ((case["degree"] + 1) ** 2 - 1)) * T
        return dict(bytes=2 * (mesh + par) + 2 * out + 20 * px, flops=340 * crossings + 200 * T)
    if kind == "views":
        return dict(bytes=2 * (mesh + values) + 2 * out + 24 * px, flops=340 * crossings)
    if kind == "serve":
        return dict(bytes=mesh + 128 * T + out + 12 * px, flops=90 * crossings)
    if kind == "err":
        return dict(bytes=mesh + 2 * values + out + 36 * px + 72 * T, flops=250 * crossings)
    if kind == "features":
        par = 4 * (7 + 3 * ((case["degree"] + 1) ** 2 - 1)) * T
        return dict(bytes=3 * par + 2 * (mesh + 12 * T) + 24 * T + 2 * values, flops=400.0 * T)
    return dict(bytes=16 * T * 4 + 12 * V + 4 * T, flops=60.0 * T)


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    kind = case["kind"]
    T = TETS_PER_POINT * case["points"]
    if kind == "features":
        return _exact_features(case, seed)
    if kind not in ("frame", "step", "render") or case.get("lens") or T * case["height"] * case["width"] > 3e9:
        return None
    s = prepare(case, seed)
    idx = s.indices.long()
    grad = kind != "frame"
    leaf = lambda x: x.detach().double().requires_grad_(grad)  # noqa: E731
    v = leaf(s.vertices)
    if kind == "render":
        m = s.model
        raw = [leaf(x) for x in (m.density, m.rgb, m.grd, m.sh)]
        cc = _circumcentres(v[idx])
        values = _activate(s.tcam["cam_pos"].double(), *raw, idx, cc, v, s.degree)
        params = [v] + raw
    else:
        values = leaf(s.values)
        params = [v, values]
    jitter = s.jitter.double() if s.jitter is not None else torch.full((*s.target.shape[:2], 2), 0.5, device=DEV,
                                                                        dtype=torch.float64)
    img, dist = _render64(v, idx, values, s.tcam, jitter)
    if kind == "frame":
        return dict(img=img, dist=dist, ranges=None, mask=None, rect=None)
    target = s.target.double()
    loss = (img[..., :3] - target).abs().mean()
    if kind == "step":
        gv, gc = torch.autograd.grad(loss, params)
        return dict(img=img, dist=dist, loss=loss, grad_vertices=gv, grad_values=gc)
    total = (dist[..., 2] ** 2).clip(min=1e-6)
    dl = (((dist[..., 0] - dist[..., 1]) + dist[..., 4]) / total).clip(min=0).mean()
    grads = torch.autograd.grad(loss + 1e-3 * dl, params, allow_unused=True)
    return dict(render=img[..., :3].permute(2, 0, 1), alpha=img[..., 3], distortion=dl,
                grads={n: x for n, x in zip(("vertices", "density", "rgb", "grd", "sh"), grads) if x is not None})


def _exact_features(case, seed):
    s = prepare(case, seed)
    m = s.model
    leaf = lambda x: x.detach().double().requires_grad_(True)  # noqa: E731
    v, cc = leaf(s.vertices), leaf(s.cc)
    raw = [leaf(x) for x in (m.density, m.rgb, m.grd, m.sh)]
    out = _activate(s.centre.double(), *raw, s.indices.long(), cc, v, s.degree)
    grads = torch.autograd.grad(out, [v] + raw + [cc], s.grad.double(), allow_unused=True)
    return dict(out=out, grads={n: x for n, x in zip(("vertices", "density", "rgb", "grd", "sh", "cc"), grads)
                                if x is not None})


def _basis(d, degree):
    x, y, z = d.unbind(1)
    out = []
    if degree > 0:
        out += [-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x]
    if degree > 1:
        out += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z,
                0.31539156525252005 * (2 * z * z - x * x - y * y), -1.0925484305920792 * x * z,
                0.5462742152960396 * (x * x - y * y)]
    if degree > 2:
        out += [-0.5900435899266435 * y * (3 * x * x - y * y), 2.890611442640554 * x * y * z,
                -0.4570457994644658 * y * (4 * z * z - x * x - y * y),
                0.3731763325901154 * z * (2 * z * z - 3 * x * x - 3 * y * y),
                -0.4570457994644658 * x * (4 * z * z - x * x - y * y), 1.445305721320277 * z * (x * x - y * y),
                -0.5900435899266435 * x * (x * x - 3 * y * y)]
    return out


def _activate(centre, density, rgb, grd, sh, idx, cc, v, degree):
    tets = v[idx]
    ng = grd * rgb.min(dim=1, keepdim=True).values / torch.linalg.norm(tets[:, 0] - cc, dim=1, keepdim=True)
    col = rgb + ((tets[:, 0] - cc).detach() * ng).sum(1, keepdim=True)
    d = torch.nn.functional.normalize(tets.mean(dim=1) - centre.reshape(1, 3), dim=1, eps=1e-8)
    for k, b in enumerate(_basis(d, degree)):
        col = col + b[:, None] * sh[:, k]
    return torch.cat([density, torch.nn.functional.softplus(col, beta=10), ng], 1)


def _circumcentres(t):
    a, b, c = t[:, 1] - t[:, 0], t[:, 2] - t[:, 0], t[:, 3] - t[:, 0]
    bc, ca, ab = torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)
    sq = lambda x: (x * x).sum(1, keepdim=True)  # noqa: E731
    return t[:, 0] + (sq(a) * bc + sq(b) * ca + sq(c) * ab) / (2.0 * (a * bc).sum(1, keepdim=True))


def _normals(t):
    """Outward face normals [n,4,3] and the faces' reference vertices [n,4,3]."""
    faces = ((0, 1, 2, 3), (0, 1, 3, 2), (0, 2, 3, 1), (1, 2, 3, 0))  # corner, two more, the opposite vertex
    n, ref = [], []
    for a, b, c, o in faces:
        x = torch.linalg.cross(t[:, b] - t[:, a], t[:, c] - t[:, a])
        n.append(torch.where(((t[:, o] - t[:, a]) * x).sum(1, keepdim=True) > 0, -x, x))
        ref.append(t[:, a])
    return torch.stack(n, 1), torch.stack(ref, 1)


def _planes(num, den):
    """Entering and exiting distances of rays with plane quotients num / den (last axis: the planes)."""
    t = num / den
    te = torch.where(den < 0, t, torch.full_like(t, -1e30)).amax(-1)
    tx = torch.where(den > 0, t, torch.full_like(t, 1e30)).amin(-1)
    return te, tx


def _render64(v, idx, values, tcam, jitter):
    """Image [H,W,4] and distortion moments [H,W,5] of a pinhole camera: every ray against every tet, the hits
    ordered by the power of the tets' circumspheres, the closed-form integral composited front to back."""
    H, W = jitter.shape[:2]
    M, K, pos = tcam["world_view_transform"].double(), tcam["K"].double(), tcam["cam_pos"].double()
    ys, xs = torch.meshgrid(torch.arange(H, device=DEV), torch.arange(W, device=DEV), indexing="ij")
    d = torch.stack([(xs + jitter[..., 0] - K[0, 2]) / K[0, 0], (ys + jitter[..., 1] - K[1, 2]) / K[1, 1],
                     torch.ones_like(jitter[..., 0])], -1).reshape(-1, 3)
    d = torch.nn.functional.normalize(d @ M[:3, :3], dim=1)
    o = pos + float(tcam["min_t"]) * d
    with torch.no_grad():
        t = v[idx]
        n, ref = _normals(t)
        nu = torch.linalg.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
        flat = (torch.nn.functional.normalize(nu, dim=1) * (t[:, 3] - t[:, 0])).sum(1).abs() < 1e-3
        solid = ~flat & (values[:, 0] > 0)
        cc = _circumcentres(t)
        rank = torch.empty(len(idx), dtype=torch.int64, device=DEV)
        key = ((cc - pos) ** 2).sum(1) - ((cc - t[:, 0]) ** 2).sum(1)
        rank[torch.argsort(key)] = torch.arange(len(idx), device=DEV)
        off = (n * ref).sum(-1)
        px, tet = [], []
        step = max(1, 12_000_000 // len(idx))
        for at in range(0, len(d), step):
            te = torch.full((len(d[at:at + step]), len(idx)), -1e30, device=DEV, dtype=torch.float64)
            tx = -te
            for k in range(4):
                den = d[at:at + step] @ n[:, k].T
                q = (off[:, k] - o[at:at + step] @ n[:, k].T) / den
                te = torch.where((den < 0) & (q > te), q, te)
                tx = torch.where((den > 0) & (q < tx), q, tx)
            p, h = torch.nonzero((te < tx) & (tx > 0) & solid, as_tuple=True)
            px.append(p + at)
            tet.append(h)
        px, tet = torch.cat(px), torch.cat(tet)
        order = torch.argsort(px * len(idx) + rank[tet])
        px, tet = px[order], tet[order]
        first = torch.searchsorted(px, px)  # each hit's pixel's first hit
    before = lambda x: (lambda c: c - x - (c - x)[first])(torch.cumsum(x, 0))  # noqa: E731
    t = v[idx[tet]]
    n, ref = _normals(t)
    dh, oh, val = d[px], o[px], values[tet]
    te, tx = _planes((n * (ref - oh[:, None])).sum(-1), (n * dh[:, None]).sum(-1))
    enter = te.clip(min=0)
    leave = torch.maximum(tx, enter)
    sigma = val[:, 0]
    a = sigma * (leave - enter)
    live = (before(a) <= 5.5).detach().double()
    T = torch.exp(-before(a))
    phi = -torch.expm1(-a) / a
    w0, w1 = phi - torch.exp(-a), 1 - phi
    ce = ((oh + enter[:, None] * dh - t[:, 0]) * val[:, 4:]).sum(1, keepdim=True) + val[:, 1:4]
    cx = ((oh + leave[:, None] * dh - t[:, 0]) * val[:, 4:]).sum(1, keepdim=True) + val[:, 1:4]
    rgb = (w0[:, None] * cx + w1[:, None] * ce) * (T * live)[:, None]
    m0, m1 = sigma * live, sigma * (enter + leave) / 2 * live
    moments = torch.stack([2 * m1 * before(m0), 2 * m0 * before(m1), m0, m1, sigma * sigma * (leave - enter) / 3 * live], 1)
    zero = lambda k: torch.zeros((H * W, k), device=DEV, dtype=torch.float64)  # noqa: E731
    img = zero(4).index_add(0, px, torch.cat([rgb, -(a * live)[:, None]], 1))
    return img.reshape(H, W, 4), zero(5).index_add(0, px, moments).reshape(H, W, 5)
