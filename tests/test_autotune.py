"""The autotuner's candidates and its cache, without a GPU."""
import types

import pytest
import torch

from radiance_meshes_b200 import autotune as AT
from radiance_meshes_b200 import scenes


@pytest.mark.parametrize("tile", [4, 8, 16, 32])
def test_no_launch_is_timed_twice(tile):
    """Equal launches would leave the choice to noise; the backward of a batch
    of views has no batch of tets to choose."""
    for cands in (AT.candidates_fwd(tile), AT.candidates_bwd(tile)):
        seen = [AT.flags(**c) for c in cands]
        assert len(set(seen)) == len(seen)
    assert all("batch" not in c for c in AT.candidates_bwd(tile))


def test_cache_entries_belong_to_one_build(tmp_path, monkeypatch):
    props = types.SimpleNamespace(name="gpu", multi_processor_count=148)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda device: props)
    views = scenes.ring_views(1, [(480, 640)])
    keys = []
    for k in (0, 0, 1):
        lib = tmp_path / f"lib{k}.so"
        lib.write_bytes(bytes([k]) * 100)
        monkeypatch.setattr(AT.build, "lib_path", lambda: str(lib))
        keys.append(AT._key(0, 1000, views, (8, 16), True))
    assert keys[0] == keys[1] and keys[0] != keys[2]
