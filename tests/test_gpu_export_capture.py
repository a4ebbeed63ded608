"""A tree's exports need nothing of the caller's streams: they give the same words
while the calling thread, or another one, captures a stream -- in every capture
mode, whether or not that stream waits for the legacy one -- and the capture goes
on."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from vitrum_b200 import bvh as vb
from vitrum_b200 import scenes

pytestmark = pytest.mark.gpu


def _stream(flags):
    h = ctypes.c_void_p()
    assert ctypes.CDLL("libcudart.so.12").cudaStreamCreateWithFlags(ctypes.byref(h), flags) == 0
    return torch.cuda.ExternalStream(h.value)


@pytest.mark.parametrize("flags", [0, 1])   # cudaStreamDefault, cudaStreamNonBlocking
@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
@pytest.mark.parametrize("same_thread", [True, False])
@pytest.mark.parametrize("device_build", [True, False])
def test_exports_during_capture(cuda, flags, mode, same_thread, device_build):
    m = scenes.random_triangles(3000, seed=3)
    if device_build:
        pos, idx = torch.from_numpy(m.positions).cuda(), torch.from_numpy(m.indices.view(np.int32)).cuda()
        g = vb.build_compressed_wide_bvh_device(pos.data_ptr(), pos.numel(), idx.data_ptr(), idx.numel())
    else:
        g = vb.build_compressed_wide_bvh(m.positions, m.indices)
    want = [a.tobytes() for a in (*g.export_wide(), *g.export_binary())]
    got, errors = [], []

    def export():
        try:
            got.extend(a.tobytes() for a in (*g.export_wide(), *g.export_binary()))
        except Exception as e:                  # noqa: BLE001 -- handed to the test
            errors.append(e)

    x = torch.arange(1 << 16, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=_stream(flags), capture_error_mode=mode):
        y = x * 2
        if same_thread:
            export()
        else:
            t = threading.Thread(target=export)
            t.start()
            t.join()
        y = y + 1
    graph.replay()
    torch.cuda.synchronize()
    assert not errors, errors
    assert got == want
    assert torch.equal(y, x * 2 + 1)
    g.close()
