"""Launches of one renderer that overlap on the device, each with a scratch of its own."""

import dataclasses

import pytest
import torch

import __graft_entry__ as entry

entry.load_package()
from gradoom_b200 import native, scene as gdscene, stepper  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# the split-line map of 8 x 8 rooms reads its tables from scratch, the small one from shared memory
@pytest.mark.parametrize("rooms", [None, 3])
def test_split_lines_on_two_streams_and_beside_the_static_step(pkg, rooms):
    spec = gdscene.GRID_CONFIGS["c4s"]
    if rooms:
        spec = dataclasses.replace(spec, rows=rooms, cols=rooms)
    sc = gdscene.make_grid_scene(spec)
    assert sc.meta["fragments"]
    n, k = 100, 4
    r = native.Renderer(gdscene.pack_scene(sc), DEV, k)
    lib = r.lib
    assert sc.num_walls <= lib.gd_static_max_walls()
    batches = [[torch.from_numpy(a).to(DEV) for a in stepper.random_lanes(sc, n, k, seed=seed)] for seed in (1, 2, 3)]
    start = torch.zeros((n, 4, 84, 84), dtype=torch.uint8, device=DEV)
    want = []
    for lanes, things in batches:
        want.append(start.clone())
        r.step(lanes, things, want[-1])
    r.check_status()
    scratches = [torch.zeros(r.scratch_bytes, dtype=torch.uint8, device=DEV) for _ in range(2)]
    streams = [torch.cuda.Stream(DEV) for _ in range(3)]
    for _ in range(4):
        stacks = [start.clone() for _ in range(3)]
        torch.cuda.synchronize()
        for (lanes, things), stack, scratch, stream in zip(batches, stacks, scratches, streams):
            assert lib.gd_render_step(r.handle, lanes.data_ptr(), things.data_ptr(), n, 1, stack.data_ptr(),
                                      scratch.data_ptr(), scratch.numel(), r.status.data_ptr(), stream.cuda_stream) == 0
        lanes, things = batches[2]
        assert lib.gd_render_step_static(r.handle, lanes.data_ptr(), things.data_ptr(), n, 1, stacks[2].data_ptr(),
                                         r.status.data_ptr(), streams[2].cuda_stream) == 0
        torch.cuda.synchronize()
        r.check_status()
        for stack, expected in zip(stacks, want):
            assert torch.equal(stack, expected)
    r.close()
