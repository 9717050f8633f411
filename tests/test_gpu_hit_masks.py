"""What the forward leaves in its workspace for the backward (hit masks and
checkpoints), whichever kind of work item wrote it and whatever else ran on
the workspace in between."""
import ctypes

import numpy as np
import pytest
import torch

from gpu_util import run_gpu_forward, to_dev
from radiance_meshes_b200 import _capi as C
from radiance_meshes_b200 import rasterizer as R
from radiance_meshes_b200.camera import pinhole_tcam
from test_gpu_long_lists import _stack

pytestmark = pytest.mark.gpu


def _scene(n, density, tile=8, H=21, W=18, small=0.0):
    verts, idx, cv = _stack(n, density, n, small)
    tcam = pinhole_tcam((0.1, 0.0, 0.0), (0.0, 0.0, 1.0), H, W, 30.0, tile_size=tile)
    jitter = np.random.default_rng(n).uniform(0, 1, (H, W, 2)).astype(np.float32)
    r = run_gpu_forward(verts, idx, cv, tcam, jitter, keep_debug=False, hit_masks=True)
    g = torch.Generator("cuda").manual_seed(n)
    r["gimg"] = torch.randn(H, W, 4, device="cuda", generator=g)
    r["gdist"] = 1e-3 * torch.randn(H, W, 5, device="cuda", generator=g)
    return r


def _bwd(r, records, hit_masks):
    L = r["lists"]
    out = R.blend_bwd(L.sorted_ids, L.ranges, r["i"], r["v"], r["c"], r["j"], r["cam"], r["img"], r["dist"], r["nc"],
                      r["gimg"], r["gdist"], records, hit_masks=hit_masks)
    torch.cuda.synchronize()
    return out


def _same(a, b):
    """Equal but for the order of the sums."""
    for x, y in zip(a, b):
        assert torch.isfinite(x).all()
        assert float((x - y).norm()) <= 1e-5 * float(y.norm())


@pytest.mark.parametrize("n,density", [(33, 0.3), (400, 0.3), (400, 6.0)])
@pytest.mark.parametrize("own", [False, True])
def test_statistics_keep_the_forwards_masks(cuda, n, density, own):
    """rm_blend_fwd, rm_calc_tet_err and rm_blend_bwd on one workspace, with
    the same flags: the statistics leave the forward's masks as they are.
    Allowed to overwrite them, they leave none that a backward would take."""
    r = _scene(n, density)
    L, cam = r["lists"], r["cam"]
    whole = _bwd(r, r["records"], False)
    before = r["records"].clone()
    rng = np.random.default_rng(n)
    pe, se = (to_dev(rng.uniform(0, 1, (cam.image_height, cam.image_width)).astype(np.float32)) for _ in range(2))
    err = torch.zeros(n, 16, device="cuda")
    cnt = torch.zeros(n, 2, dtype=torch.int32, device="cuda")
    C.check(C.lib().rm_calc_tet_err(
        C.ptr(L.sorted_ids), C.ptr(L.ranges), C.ptr(r["i"]), C.ptr(r["v"]), C.ptr(r["c"]), n, r["v"].shape[0], None,
        ctypes.byref(cam), C.ptr(pe), C.ptr(se), C.ptr(err), C.ptr(cnt), C.ptr(r["records"]), r["records"].numel(),
        C.RM_BLEND_REUSE_RECORDS | C.RM_BLEND_HIT_MASKS | (C.RM_BLEND_OWN_SCRATCH if own else 0),
        C.stream_handle()), "rm_calc_tet_err")
    assert int(cnt[:, 0].sum()) > 0
    base = C.lib().rm_blend_workspace_size(n, cam.grid_width * cam.grid_height)
    assert own or torch.equal(r["records"][base:], before[base:])
    _same(_bwd(r, r["records"], True), whole)


@pytest.mark.parametrize("batch", [16, 32, 64])
@pytest.mark.parametrize("heavy", [0, 1, 15])  # by the lists' lengths, every tile by pair items, by warp items
@pytest.mark.parametrize("n,density", [(33, 0.3), (400, 0.3), (400, 6.0)])
def test_masks_of_every_batch_and_route(cuda, batch, heavy, n, density):
    """Each kind of forward item, with each batch size, leaves masks and
    checkpoints that give the gradients of a backward that tests every entry.
    The pair items of batches of 16 write half a mask word a block.
    (The workspace starts out zeroed: a mask that is not written loses hits.)"""
    r = _scene(n, density)
    whole = _bwd(r, r["records"], False)
    L = r["lists"]
    ws = torch.zeros_like(r["records"])
    old = R.blend_tuning()
    R.set_blend_tuning((heavy << C.RM_BLEND_HEAVY_SHIFT) | ({16: 4, 32: 5, 64: 6}[batch] << C.RM_BLEND_BATCH_SHIFT), 0)
    try:
        img, dist, nc, _ = R.blend_fwd(L.sorted_ids, L.ranges, r["i"], r["v"], r["c"], r["j"], r["cam"],
                                       tiles_touched=r["tiles"], records=ws, hit_masks=True)
    finally:
        R.set_blend_tuning(*old)
    assert torch.equal(img, r["img"]) and torch.equal(dist, r["dist"]) and torch.equal(nc, r["nc"])
    _same(_bwd(r, ws, True), whole)


@pytest.mark.parametrize("tile,heavy", [(4, 0), (8, 1), (8, 15), (16, 0)])
@pytest.mark.parametrize("positive", [1, 5])
def test_nan_ray_ends_at_the_first_entry_it_meets(cuda, tile, heavy, positive):
    """A ray that is not a number counts as a hit of every entry with a
    positive density, whatever the other rays of its strip see; only its own
    pixel shows it."""
    n, size = 160, 32
    verts, idx, cv = _stack(n, 0.3, n, 1.0)
    cv[np.arange(n) % positive != 0, 0] = 0.0
    tcam = pinhole_tcam((0.1, 0.0, 0.0), (0.0, 0.0, 1.0), size, size, 30.0, tile_size=tile)
    jitter = np.random.default_rng(n).uniform(0, 1, (size, size, 2)).astype(np.float32)
    bad = np.zeros((size, size), bool)
    bad[3::16, 5::8] = True
    old = R.blend_tuning()
    R.set_blend_tuning(heavy << C.RM_BLEND_HEAVY_SHIFT, 0)
    try:
        clean = run_gpu_forward(verts, idx, cv, tcam, jitter, keep_debug=False)
        jitter[bad] = np.nan
        r = run_gpu_forward(verts, idx, cv, tcam, jitter, keep_debug=False)
    finally:
        R.set_blend_tuning(*old)
    ids, ranges = r["lists"].sorted_ids.cpu().numpy(), r["lists"].ranges.cpu().numpy()
    nc = r["nc"].cpu().numpy()[..., 0]
    for y, x in zip(*np.nonzero(bad)):
        x0, x1 = ranges[(y // tile) * (size // tile) + x // tile]
        hit = np.flatnonzero(cv[ids[x0:x1], 0] > 0)
        assert nc[y, x] == (hit[0] + 1 if len(hit) else x1 - x0)
    ok = torch.from_numpy(~bad).cuda()
    assert torch.equal(r["nc"][ok], clean["nc"][ok]) and torch.equal(r["img"][ok], clean["img"][ok])


@pytest.mark.parametrize("heavy", [1, 15])  # every tile by pair items, by warp items
@pytest.mark.parametrize("n", [600, 1100])  # 4 and 8 checkpoints
def test_stretches_hold_what_little_is_left(cuda, heavy, n):
    """Bright entries before dark ones: what the dark ones still add to the
    colour is far below the rounding of the colour.  A backward by stretches
    takes it from the checkpoints, one over whole lists adds it up entry by
    entry; each of the n additions rounds by 2^-24 at most, in both, so the
    dark entries' gradients agree to 2n * 2^-24 (1.3e-4 for 1100)."""
    verts, idx, cv = _stack(n, 0.2, n)
    cv[:, 4:] = 0.0
    cv[-100:, 1:4] *= 1e3  # the lists run from the last tets to the first
    cv[:-100, 1:4] *= 1e-2
    H, W = 21, 18
    tcam = pinhole_tcam((0.1, 0.0, 0.0), (0.0, 0.0, 1.0), H, W, 30.0, tile_size=8)
    jitter = np.random.default_rng(n).uniform(0, 1, (H, W, 2)).astype(np.float32)
    old = R.blend_tuning()
    R.set_blend_tuning(heavy << C.RM_BLEND_HEAVY_SHIFT, 0)
    try:
        r = run_gpu_forward(verts, idx, cv, tcam, jitter, keep_debug=False, hit_masks=True)
    finally:
        R.set_blend_tuning(*old)
    g = torch.Generator("cuda").manual_seed(n)
    r["gimg"] = 0.5 + 0.5 * torch.rand(H, W, 4, device="cuda", generator=g)
    r["gimg"][..., 3] = 0.0
    r["gdist"] = None
    (gv0, gc0), (gv1, gc1) = _bwd(r, r["records"], False), _bwd(r, r["records"], True)
    ids, ranges = r["lists"].sorted_ids.cpu().numpy(), r["lists"].ranges.cpu().numpy()
    dark = np.arange(n) < 100
    for x0, x1 in ranges:  # behind every bright one
        bright = np.flatnonzero(ids[x0:x1] >= n - 100)
        assert not dark[ids[x0:x0 + bright[-1] + 1]].any()
    dark = to_dev(dark)
    for a, b in ((gc1[dark, 0], gc0[dark, 0]), (gv1.view(n, 4, 3)[dark], gv0.view(n, 4, 3)[dark])):
        assert float(b.norm()) > 0
        assert float((a.double() - b.double()).norm()) <= 2 * n * 2.0**-24 * float(b.double().norm())
