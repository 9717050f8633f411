"""The sort, the scan and the ordering of the tiles at the sizes where the way
they split their work changes: the sort's larger tile of pairs, look-backs
over more tiles than one window holds, and tile counts around the ordering's
chunks (1024 tiles a CTA, 8192 a round)."""
import numpy as np
import pytest
import torch

from radiance_meshes_b200 import batch as B
from radiance_meshes_b200 import rasterizer as R
from radiance_meshes_b200 import scenes
from radiance_meshes_b200.camera import tcam_to_struct
from test_gpu_errors import _scan
from test_gpu_sort import gpu_sort, ref_sort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(3 << 20) - 1, 3 << 20, 6144 * 513 - 1, 6144 * 513, 6144 * 513 + 1])
def test_sort_large_tiles(cuda, n):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 2 ** 19, size=n, dtype=np.int64) * 1021  # many equal keys
    vals = np.arange(n, dtype=np.int32)
    for count in (n, 1, 6144, 70_001):  # filled, and all but empty
        ko, vo = gpu_sort(keys, vals, 29, n_dev=count)
        rk, rv = ref_sort(keys[:count], vals[:count], 29)
        assert np.array_equal(ko[:count], rk) and np.array_equal(vo[:count], rv)


@pytest.mark.parametrize("n", [4096 * 32 - 1, 4096 * 33, 4096 * 64 + 1, 4096 * 65, 1_500_007])
def test_scan_windows(cuda, n):
    tiles = torch.from_numpy(np.random.default_rng(n).integers(0, 9, size=n).astype(np.int32)).cuda()
    off, tot, st = _scan(tiles)
    ref = torch.cumsum(tiles, 0)
    assert st == 0 and int(tot.item()) == int(ref[-1].item()) and torch.equal(off.long(), ref)


@pytest.mark.parametrize("n_views,res", [(1, 256), (1, 260), (8, 256), (9, 252)])  # 8x8: 1024 tiles a view and around
def test_every_tile_is_ordered(cuda, n_views, res):
    mesh, _ = scenes.workload_gradient_check()
    i, v, c = (torch.from_numpy(x).cuda() for x in (mesh.indices, mesh.vertices, mesh.cell_values))
    cams = [tcam_to_struct(w.tcam())
            for w in scenes.ring_views(n_views, [(res, res)] * n_views, radius=2.9, height_offset=0.4, tile_size=8)]
    vb = B.ViewBatch(cams)
    jit = torch.full((vb.n_pixels, 2), 0.5, device="cuda")
    br = B.BatchedRasterizer(i, v, c, vb, jitter=jit)
    br.img.fill_(float("nan"))
    br.nc.fill_(-1)
    br.forward()
    br.check()
    assert (br.nc >= 0).all() and torch.isfinite(br.img).all()
    for k in (0, n_views - 1):
        tiles, rect, vs, _ = R.project_fwd(i, v, cams[k])
        lists = R.build_tile_lists(tiles, rect, vs, cams[k])
        img, _, nc, _ = R.blend_fwd(lists.sorted_ids, lists.ranges, i, v, c,
                                    torch.full((res, res, 2), 0.5, device="cuda"), cams[k], tiles_touched=tiles)
        assert torch.equal(vb.split(br.img)[k].reshape(img.shape), img)
        assert torch.equal(vb.split(br.nc)[k].reshape(nc.shape), nc)
