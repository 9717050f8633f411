"""The pair count's way to the host."""
import threading

import pytest
import torch

from radiance_meshes_b200 import rasterizer as R

pytestmark = pytest.mark.gpu


def test_reads_that_overlap_have_buffers_of_their_own(cuda):
    """A frame that failed between the start and the end of its read leaves its
    copy in flight: the next frame's read, on another stream, holds its own
    count, and so does the first one's."""
    first, second = (torch.tensor([n, 0], dtype=torch.int64, device="cuda") for n in (11, 22))
    torch.cuda.synchronize()
    a = R._count_read_start(first)
    with torch.cuda.stream(torch.cuda.Stream()):
        b = R._count_read_start(second)
        assert R._count_read_finish(b) == (22, 0)
    assert R._count_read_finish(a) == (11, 0)


def test_finished_reads_keep_one_buffer(cuda):
    count = torch.tensor([5, 1], dtype=torch.int64, device="cuda")
    for _ in range(3):
        pending = R._count_read_start(count)
        assert R._count_read_finish(pending) == (5, 1)
    held = R._COUNT_READ[(count.device, threading.get_ident())]
    assert R._count_read_start(count)[-1] is held
