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


def _room(n_pairs, n_tiles, subs, shift=None):
    """Bytes for the masks of n_pairs entries, and their checkpoints every 1 << shift."""
    words = (n_pairs // 32 + n_tiles + 2) * subs * 64
    return 256 + 4 * (words + (0 if shift is None else ((n_pairs >> shift) + 2) * subs * 8 * 64))


def _header(ws, n_tets, n_tiles):
    base = C.lib().rm_blend_workspace_size(n_tets, n_tiles)
    return ws[base:base + 12].view(torch.int32).tolist()  # state, log2 of the stretch, checkpoint ids


def _fwd_into(r, ws):
    L = r["lists"]
    img, dist, nc, _ = R.blend_fwd(L.sorted_ids, L.ranges, r["i"], r["v"], r["c"], r["j"], r["cam"],
                                   tiles_touched=r["tiles"], records=ws, hit_masks=True)
    assert torch.equal(img, r["img"]) and torch.equal(dist, r["dist"]) and torch.equal(nc, r["nc"])


@pytest.mark.parametrize("million", [0.1, 0.5, 0.6, 1, 9, 17, 55, 65, 100])
def test_stretch_length_is_that_of_the_lists(cuda, million):
    """Short lists are cut every 128 entries, however many the workspace has
    room for."""
    r = _scene(33, 0.3)
    G = r["cam"].grid_width * r["cam"].grid_height
    size = C.lib().rm_blend_workspace_size(33, G) + C.lib().rm_blend_hit_mask_bytes(int(million * 1_000_000), G, 64)
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    _fwd_into(r, ws)
    assert _header(ws, 33, G)[1] == 7


@pytest.mark.parametrize("entries,shift", [(1 << 19, 7), ((1 << 19) + 1, 9), (64 << 20, 9), ((64 << 20) + 1, 12)])
def test_stretch_length_of_long_lists(cuda, entries, shift):
    """Above half a million entries every 512, above 64M every 4096; the size
    that rm_blend_hit_mask_bytes gives has room for them."""
    verts, idx, cv = _stack(1, 400.0, 1)
    tcam = pinhole_tcam((0.1, 0.0, 0.0), (0.0, 0.0, 1.0), 16, 16, 30.0, tile_size=8)
    r = run_gpu_forward(verts, idx, cv, tcam, np.full((16, 16, 2), 0.5, np.float32), keep_debug=False)
    cuts = [0, 1, entries // 2, entries // 2, entries]  # one tet over and over
    ranges = to_dev(np.array(list(zip(cuts[:-1], cuts[1:])), np.int32))
    ids = torch.zeros(entries, dtype=torch.int32, device="cuda")
    _, _, _, ws = R.blend_fwd(ids, ranges, r["i"], r["v"], r["c"], r["j"], r["cam"], hit_masks=True)
    state, got, ids_fit = _header(ws, 1, 4)
    assert got == shift and ids_fit == (entries >> shift) + 2


@pytest.mark.parametrize("shift", [7, 9, 12, None, "half"])
@pytest.mark.parametrize("heavy", [0, 15])
def test_room_for_longer_stretches_or_none(cuda, shift, heavy):
    """A workspace too small for the shortest stretches gets the next longer
    ones, or none where not even the masks all fit: the same image, gradients
    and statistics."""
    n = 9000  # three stretches of 4096
    r = _scene(n, 0.02, H=9, W=14)
    L, cam = r["lists"], r["cam"]
    whole = _bwd(r, r["records"], False)
    G, P = cam.grid_width * cam.grid_height, L.n_pairs
    base = C.lib().rm_blend_workspace_size(n, G)
    room = _room(P, G, 1, shift) if shift != "half" else _room(P // 2, G, 1)
    ws = torch.zeros(base + room, dtype=torch.uint8, device="cuda")
    old = R.blend_tuning()
    R.set_blend_tuning(heavy << C.RM_BLEND_HEAVY_SHIFT, 0)
    try:
        _fwd_into(r, ws)
    finally:
        R.set_blend_tuning(*old)
    assert _header(ws, n, G)[1] == (shift if isinstance(shift, int) else 31)
    _same(_bwd(r, ws, True), whole)
    # the statistics on the same room (and their counts, a pixel each, after it)
    rng = np.random.default_rng(n)
    pe, se = (to_dev(rng.uniform(0, 1, (cam.image_height, cam.image_width)).astype(np.float32)) for _ in range(2))
    out = []
    for size, flags in ((base + room + 512 + 4 * pe.numel(), C.RM_BLEND_OWN_SCRATCH), (base, 0)):
        ws = torch.zeros(size, dtype=torch.uint8, device="cuda")
        err, cnt = torch.zeros(n, 16, device="cuda"), torch.zeros(n, 2, dtype=torch.int32, device="cuda")
        C.check(C.lib().rm_calc_tet_err(
            C.ptr(L.sorted_ids), C.ptr(L.ranges), C.ptr(r["i"]), C.ptr(r["v"]), C.ptr(r["c"]), n, r["v"].shape[0],
            None, ctypes.byref(cam), C.ptr(pe), C.ptr(se), C.ptr(err), C.ptr(cnt), C.ptr(ws), size, flags,
            C.stream_handle()), "rm_calc_tet_err")
        out.append((err, cnt))
    (err, cnt), (err0, cnt0) = out
    assert cnt0[:, 0].sum() > 0 and torch.equal(cnt, cnt0)
    assert float((err - err0).norm()) <= 1e-5 * float(err0.norm())
