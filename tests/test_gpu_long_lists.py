"""Lists around the lengths at which the passes change how they walk them.

The forward takes a list in blocks of 32 entries, drops the entries that no
ray of a strip can hit and fills a batch from as many blocks as that leaves
room for: lists around whole blocks, dense and mostly dropped, are compared
with the oracle bit for bit (log T, distortion, n_contributors).  The backward
takes a list in stretches of 128 entries, each from the state the forward
left there: lists one entry short of, at and past whole stretches are compared
with the oracle's adjoint, with pixels that end before, inside and after a
stretch."""
import ctypes

import numpy as np
import pytest
import torch

from gpu_util import bits, run_gpu_forward, to_dev
from oracle import oracle as O
from radiance_meshes_b200 import _capi as C
from radiance_meshes_b200 import rasterizer as R
from radiance_meshes_b200.camera import pinhole_tcam
from test_gpu_backward import _run

pytestmark = pytest.mark.gpu


def _stack(n, density, seed, small=0.0):
    """n thin tets one behind the other along the view axis, wider than most
    of the image, each shifted sideways a little; a fraction `small` of them a
    few pixels wide."""
    rng = np.random.default_rng(seed)
    z = 2.0 + 0.02 * np.arange(n)[:, None]
    s = z * rng.uniform(0.3, 1.2, size=(n, 1))
    s[rng.uniform(size=n) < small] *= 0.05
    cx, cy = (z * rng.uniform(-0.2, 0.2, size=(n, 1)) for _ in range(2))
    corners = [(-1, -1, 0.0), (1, -1, 0.0), (0, 1.2, 0.0), (0.0, 0.0, 0.015)]
    verts = np.concatenate([np.concatenate([cx + a * s, cy + b * s, z + dz], 1)[:, None] for a, b, dz in corners], 1)
    idx = np.arange(4 * n, dtype=np.int32).reshape(n, 4)[:, [1, 0, 2, 3]]
    cv = np.concatenate([density * rng.uniform(0.5, 1.5, (n, 1)), rng.uniform(0, 1, (n, 3)),
                         rng.normal(0, 0.1, (n, 3))], 1)
    return verts.reshape(-1, 3).astype(np.float32), np.ascontiguousarray(idx), cv.astype(np.float32)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 256, 257, 400])
@pytest.mark.parametrize("density", [0.3, 6.0])  # every pixel reaches the end; most end on the way
def test_backward_over_stretches(cuda, n, density):
    verts, idx, cv = _stack(n, density, n)
    tcam = pinhole_tcam((0.0, 0.0, 0.0), (0.0, 0.0, 1.0), 11, 13, 30.0, tile_size=8)
    jitter = np.random.default_rng(n).uniform(0, 1, (11, 13, 2)).astype(np.float32)
    _run(verts, idx, cv, tcam, jitter, "linear", seed=n, check_f64=False, hit_masks=True)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 191, 193, 420])
@pytest.mark.parametrize("small", [0.0, 0.95])
@pytest.mark.parametrize("density,tile", [(0.3, 8), (6.0, 8), (6.0, 16), (1.0, 4)])
def test_forward_over_blocks(cuda, n, small, density, tile):
    verts, idx, cv = _stack(n, density, n, small)
    cv[::7, 0] = 0.0
    tcam = pinhole_tcam((0.1, 0.0, 0.0), (0.0, 0.0, 1.0), 21, 18, 30.0, tile_size=tile)
    jitter = np.random.default_rng(n).uniform(0, 1, (21, 18, 2)).astype(np.float32)
    L = O.rasterize_lists(idx, verts, tcam)
    img, dist, nc = O.blend_fwd_f32(L, idx, verts, cv, jitter)
    r = run_gpu_forward(verts, idx, cv, tcam, jitter, keep_debug=False, hit_masks=True)
    assert np.array_equal(r["nc"].cpu().numpy()[..., 0], nc)
    assert np.array_equal(bits(r["img"].cpu().numpy()[..., 3]), bits(img[..., 3]))
    assert np.array_equal(bits(r["dist"].cpu().numpy()), bits(dist))
    assert np.abs(r["img"].cpu().numpy() - img).max() <= 1e-4


@pytest.mark.parametrize("n", [1, 32, 33, 127, 128, 129, 400])
@pytest.mark.parametrize("density", [0.3, 6.0])
def test_statistics_over_stretches(cuda, n, density):
    """The statistics by stretches (a workspace with room for the masks) and by
    whole lists (without): equal counts and maxima, sums within 1e-5."""
    verts, idx, cv = _stack(n, density, n, 0.3)
    tcam = pinhole_tcam((0.1, 0.0, 0.0), (0.0, 0.0, 1.0), 21, 18, 30.0, tile_size=8)
    jitter = np.full((21, 18, 2), 0.5, np.float32)
    r = run_gpu_forward(verts, idx, cv, tcam, jitter, keep_debug=False)
    rng = np.random.default_rng(n)
    pe, se = (to_dev(rng.uniform(0, 1, (21, 18)).astype(np.float32)) for _ in range(2))
    L, cam = r["lists"], r["cam"]
    err, cnt = R.calc_tet_err(L.sorted_ids, L.ranges, r["i"], r["v"], r["c"], cam, pe, se)
    err0, cnt0 = torch.zeros_like(err), torch.zeros_like(cnt)
    size = C.lib().rm_blend_workspace_size(n, cam.grid_width * cam.grid_height)
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    C.check(C.lib().rm_calc_tet_err(C.ptr(L.sorted_ids), C.ptr(L.ranges), C.ptr(r["i"]), C.ptr(r["v"]), C.ptr(r["c"]),
                                    n, len(verts), None, ctypes.byref(cam), C.ptr(pe), C.ptr(se), C.ptr(err0),
                                    C.ptr(cnt0), C.ptr(ws), size, 0, C.stream_handle()), "rm_calc_tet_err")
    assert cnt0[:, 0].sum() > 0 and torch.equal(cnt, cnt0)
    scale = err0.abs().amax(dim=0).clamp(min=1e-30)
    assert ((err - err0).abs() / scale).max() <= 1e-5
