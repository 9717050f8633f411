"""A drop-in frame that nothing can be differentiated through keeps nothing
for a backward, and is the same frame."""
import pytest
import torch

from gpu_util import to_dev
from radiance_meshes_b200 import _capi as C
from radiance_meshes_b200 import rasterizer as R
from radiance_meshes_b200 import render as RR
from radiance_meshes_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [8, 16])
@pytest.mark.parametrize("grads", [(), ("v",), ("c",), ("v", "c")])
def test_room_for_masks_only_where_a_gradient_is_asked_for(cuda, monkeypatch, tile, grads):
    mesh, view = scenes.workload_gradient_check(tile)
    tcam = view.tcam(tile_size=tile)
    i, v, c = to_dev(mesh.indices), to_dev(mesh.vertices), to_dev(mesh.cell_values)
    j = torch.rand(view.height, view.width, 2, device="cuda", generator=torch.Generator("cuda").manual_seed(tile))
    sizes = []
    blend_fwd = R.blend_fwd

    def seen(*args, **kw):
        out = blend_fwd(*args, **kw)
        sizes.append(out[3].numel())
        return out

    monkeypatch.setattr(R, "blend_fwd", seen)
    plain, dist, _ = RR.rasterize(v, i, c, tcam, j)
    G = R.camera(tcam).grid_width * R.camera(tcam).grid_height * (tile // 8) ** 2
    assert sizes == [C.lib().rm_blend_workspace_size(len(mesh.indices), G)]
    leaves = {"v": v, "c": c}
    for name in grads:
        leaves[name].requires_grad_(True)
    img, dist2, _ = RR.rasterize(v, i, c, tcam, j)
    assert torch.equal(img, plain) and torch.equal(dist, dist2)
    assert (sizes[1] > sizes[0]) == bool(grads) and img.requires_grad == bool(grads)
    if grads:
        w = torch.rand(img.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
        got = torch.autograd.grad((img * w).sum(), [leaves[n] for n in grads])
        both = [x.detach().clone().requires_grad_(True) for x in (v, c)]
        want = torch.autograd.grad((RR.rasterize(both[0], i, both[1], tcam, j)[0] * w).sum(), both)
        for name, g in zip(grads, got):
            ref = want["vc".index(name)]
            assert float((g - ref).norm()) <= 1e-5 * float(ref.norm())
