"""Creating a renderer reads the blob's header on the host and nothing else: it allocates no device memory for a scene
without split lines, and the blob's bytes have to be there when the first call draws, not before."""

import ctypes

import numpy as np
import pytest
import torch

import __graft_entry__ as entry

entry.load_package()
from gradoom_b200 import native, scene as gdscene, stepper  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _create(blob, device_blob, k):
    handle = ctypes.c_void_p()
    return native.load().gd_renderer_create(blob.ctypes.data, device_blob.data_ptr(), blob.size, 0, k,
                                            ctypes.byref(handle)), handle


def _draw(handle, lanes, things):
    """One step with a scratch buffer and one with the built-in array where the map fits it."""

    lib, n = native.load(), len(lanes)
    scratch = torch.zeros(lib.gd_renderer_scratch_bytes(handle), dtype=torch.uint8, device=DEV)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    dl, dt = torch.from_numpy(lanes).to(DEV), torch.from_numpy(things).to(DEV)
    stacks = [torch.zeros((n, 4, 84, 84), dtype=torch.uint8, device=DEV) for _ in range(2)]
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.gd_render_step(handle, dl.data_ptr(), dt.data_ptr(), n, 0, stacks[0].data_ptr(), scratch.data_ptr(),
                              scratch.numel(), status.data_ptr(), stream) == 0
    rc = lib.gd_render_step_static(handle, dl.data_ptr(), dt.data_ptr(), n, 0, stacks[1].data_ptr(), status.data_ptr(), stream)
    assert rc in (0, -9)
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    if rc == 0:
        assert torch.equal(*stacks)
    return stacks[0][:, 3].cpu().numpy()


# tables on chip, tables in scratch beyond the built-in array's limits, split lines with tables in scratch
@pytest.mark.parametrize("name", ["c1", "c4", "c4s"])
def test_blob_may_arrive_after_creation(name, pkg, oracle, scenes):
    sc, blob = scenes(name)
    lanes, things = stepper.random_lanes(sc, 24, 4, seed=6)
    want = oracle.render(blob, lanes, things, mask_hud=False)["obs"]
    device_blob = torch.zeros(blob.size, dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    rc, handle = _create(blob, device_blob, 4)
    assert rc == 0
    device_blob.copy_(torch.from_numpy(blob))
    assert np.array_equal(_draw(handle, lanes, things), want)
    native.load().gd_renderer_destroy(handle)


@pytest.mark.parametrize("name", ["c1", "c4"])
def test_blob_without_cells_is_drawn_the_same(name, pkg, oracle, scenes):
    sc, blob = scenes(name)
    older = blob.copy()
    older[:gdscene.GD_HDR_WORDS * 4].view(np.int32)[gdscene.GD_HDR_SECTION0 + gdscene.SEC["CELLS"]] = 0
    lanes, things = stepper.random_lanes(sc, 24, 4, seed=7)
    rc, handle = _create(older, torch.from_numpy(older).to(DEV), 4)
    assert rc == 0
    assert np.array_equal(_draw(handle, lanes, things), oracle.render(blob, lanes, things, mask_hud=False)["obs"])
    native.load().gd_renderer_destroy(handle)


def test_creation_and_the_static_step_allocate_nothing(pkg, scenes):
    """Thirty-two renderers of the 800-wall map, then static steps of a small one."""

    _, blob = scenes("c4")
    device_blob = torch.from_numpy(blob).to(DEV)
    small, small_blob = scenes("c1")
    lanes, things = stepper.random_lanes(small, 4, 4, seed=8)
    rc, drawn = _create(small_blob, torch.from_numpy(small_blob).to(DEV), 4)
    assert rc == 0
    _draw(drawn, lanes, things)
    lib = native.load()
    taken = []
    for _ in range(2):                                 # streams and events of the first turn warm the driver up
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        handles = [_create(blob, device_blob, 4) for _ in range(32)]
        assert all(rc == 0 for rc, _ in handles)
        torch.cuda.synchronize()
        taken.append(before - torch.cuda.mem_get_info()[0])
        for _, handle in handles:
            lib.gd_renderer_destroy(handle)
    assert taken[1] == 0
    lib.gd_renderer_destroy(drawn)


def test_creation_while_a_stream_is_captured(pkg, oracle, scenes):
    sc, blob = scenes("c1")
    device_blob = torch.from_numpy(blob).to(DEV)
    lanes, things = stepper.random_lanes(sc, 4, 4, seed=9)
    _, first = _create(blob, device_blob, 4)
    marker = torch.zeros(1, device=DEV)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        rc, handle = _create(blob, device_blob, 4)
        marker += 1
    assert rc == 0
    graph.replay()
    torch.cuda.synchronize()
    assert marker.item() == 1
    assert np.array_equal(_draw(handle, lanes, things), oracle.render(blob, lanes, things, mask_hud=False)["obs"])
    for h in (first, handle):
        native.load().gd_renderer_destroy(h)
