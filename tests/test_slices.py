"""A lane drawn by several CTAs, each a slice of its columns, against the same lane drawn by one."""

import pytest
import torch

import __graft_entry__ as entry

entry.load_package()
from gradoom_b200 import native, state as gdstate, stepper  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# chips; split lines; grates; unclaimed pixels (half of the lanes on the corners of rooms); the large map; no things
@pytest.mark.parametrize("config,k,hud", [("c1d", 4, False), ("c4s", 7, True), ("c1m", 3, True), ("c2", 12, False),
                                          ("c4", 9, False), ("c3", 0, True)])
def test_slices_equal_whole_lanes(scenes, config, k, hud):
    sc, blob = scenes(config)
    r = native.Renderer(blob, DEV, k)
    n = r.ctas // 4 + 1                      # one lane more than are drawn in slices
    host_lanes, host_things = stepper.random_lanes(sc, n, k, seed=11)
    if config == "c2":
        room = int(sc.meta["spec"].room)
        for lane in range(0, n, 2):
            for fixed, word in ((gdstate.L_X_FIXED, gdstate.L_X), (gdstate.L_Y_FIXED, gdstate.L_Y)):
                host_lanes[lane, fixed] = (1 + lane // 2 % 6) * room << 16
                host_lanes.view("float32")[lane, word] = (1 + lane // 2 % 6) * room
    lanes, things = torch.from_numpy(host_lanes).to(DEV), torch.from_numpy(host_things).to(DEV)
    rings = torch.from_numpy(stepper.random_decals(sc, host_lanes, 20, 64, seed=12)).to(DEV) if config == "c1d" else None
    g = torch.Generator(DEV).manual_seed(7)
    stack = torch.randint(0, 256, (n, 4, 84, 84), dtype=torch.uint8, device=DEV, generator=g)
    ring = torch.randint(0, 256, (n, 8, 84, 84), dtype=torch.uint8, device=DEV, generator=g)
    mask = torch.rand(n, device=DEV, generator=g) < 0.5

    def draw(a, b):
        """Every entry point over lanes a .. b - 1."""

        if rings is not None:
            r.bind_decals(rings[a:b].contiguous())
        part = [t[a:b].contiguous() for t in (lanes, things)]
        out = [stack[a:b].clone() for _ in range(5)] + [ring[a:b].clone() for _ in range(2)]
        rgb = torch.zeros((b - a, 240, 320, 3), dtype=torch.uint8, device=DEV)
        r.step(*part, out[0], mask_hud=not hud)
        r.reset(*part, mask[a:b], out[1], mask_hud=not hud)
        r.step_frames(*part, out[2], rgb=rgb, mask_hud=not hud)
        r.step_reset(*part, *part, mask[a:b], out[3], out[4], mask_hud=not hud)
        r.step_ring(*part, out[5], 2, mask_hud=not hud)
        r.reset_ring(*part, mask[a:b], out[6], mask_hud=not hud)
        return out + [rgb, *r.frames(*part, obs=True, indexed=True, rgb=True, mask_hud=not hud)]

    want = draw(0, n)
    for first, count in ((0, 1), (5, 3), (1, n - 1)):
        for got, expected in zip(draw(first, first + count), want):
            assert torch.equal(got, expected[first:first + count]), count
    r.check_status()
    r.close()


def test_static_step_in_slices(scenes):
    sc, blob = scenes("c1")
    r = native.Renderer(blob, DEV, 4)
    lanes, things = (torch.from_numpy(a).to(DEV) for a in stepper.random_lanes(sc, 100, 4, seed=2))
    whole = torch.zeros((100, 4, 84, 84), dtype=torch.uint8, device=DEV)
    r.step(lanes, things, whole)
    for n in (1, 8, 9, 33):
        got = torch.zeros((n, 4, 84, 84), dtype=torch.uint8, device=DEV)
        r.step_static(lanes[:n], things[:n], got)
        assert torch.equal(got, whole[:n])
    r.close()
