"""Views and maps at the edges of the render kernel's short cuts, against the oracle."""

import dataclasses

import numpy as np
import pytest
import torch

import __graft_entry__ as entry

entry.load_package()
from gradoom_b200 import native, scene as gdscene, state as gdstate, stepper  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
FIXED = 1 << 16


def _equal(oracle, sc, lanes, things, k):
    blob = gdscene.pack_scene(sc)
    want = oracle.render(blob, lanes, things, mask_hud=False)
    renderer = native.Renderer(blob, DEV, k)
    obs, indexed, _ = renderer.frames(torch.from_numpy(lanes).to(DEV), torch.from_numpy(things).to(DEV), obs=True,
                                      indexed=True, mask_hud=False)
    renderer.check_status()
    assert np.array_equal(indexed.cpu().numpy(), want["indexed"])
    assert np.array_equal(obs.cpu().numpy(), want["obs"])
    renderer.close()


def _place(lanes, rows, x, y):
    lf = lanes.view(np.float32)
    lanes[rows, gdstate.L_X_FIXED] = np.round(np.asarray(x) * FIXED).astype(np.int32)
    lanes[rows, gdstate.L_Y_FIXED] = np.round(np.asarray(y) * FIXED).astype(np.int32)
    lf[rows, gdstate.L_X] = lanes[rows, gdstate.L_X_FIXED].astype(np.float32) / np.float32(FIXED)
    lf[rows, gdstate.L_Y] = lanes[rows, gdstate.L_Y_FIXED].astype(np.float32) / np.float32(FIXED)


# 2 x 300 rooms: a cell of the sector grid meets ten rooms, more than it lists (the players look across the rows,
# so that no column crosses more lines than its scratch holds); 16 x 16: one to four; 1 x 1: all the same room
@pytest.mark.parametrize("rows,cols,room", [(2, 300, 96.0), (16, 16, 128.0), (1, 1, 512.0)])
def test_views_from_outside_rooms_and_close_to_walls(pkg, oracle, rows, cols, room):
    """Players outside the map (every pixel is searched for a sector), on lines, and within 8 units of walls (where
    the columns of a wall are not taken from its projected ends)."""

    spec = dataclasses.replace(gdscene.GRID_CONFIGS["c2"], rows=rows, cols=cols, room=room, seed=91)
    sc = gdscene.make_grid_scene(spec)
    n, k = 24, 6
    lanes, things = stepper.random_lanes(sc, n, k, seed=rows)
    rng = np.random.default_rng(cols)
    wide, high = cols * room, rows * room
    _place(lanes, slice(0, 4), [-40.0, wide + 300.0, wide / 2, -2000.0], [high / 2, high / 2, -64.5, high + 1000.0])
    _place(lanes, slice(4, 14), rng.integers(0, cols, 10) * room + rng.uniform(0.0, 7.0, 10),
           rng.integers(0, rows, 10) * room + rng.uniform(1.0, room - 1.0, 10))
    _place(lanes, slice(14, 16), [room, room / 2], [room / 2, room])
    if cols > 100:
        quarter = np.where(np.arange(n) % 2, 1 << 30, 3 << 30) + rng.integers(-(1 << 26), 1 << 26, n)
        lanes[:, gdstate.L_ANGLE_BAM] = quarter.astype(np.uint32).view(np.int32)
        lanes.view(np.float32)[:, gdstate.L_ANGLE] = quarter.astype(np.float32) * np.float32(gdstate.BAM_TO_RADIANS)
    # things right in front of some players: sprites that fill the view, some beyond the floor's edge
    tf = things.view(np.float32)
    lf = lanes.view(np.float32)
    for lane in range(10, 24):
        for slot, distance in enumerate((6.0, 20.0, 45.0)):
            tf[lane, slot, 0] = lf[lane, gdstate.L_X] + distance * np.cos(lf[lane, gdstate.L_ANGLE])
            tf[lane, slot, 1] = lf[lane, gdstate.L_Y] + distance * np.sin(lf[lane, gdstate.L_ANGLE])
            tf[lane, slot, 2] = lf[lane, gdstate.L_VIEW_Z] - 41.0 - 30.0 * slot
    _equal(oracle, sc, lanes, things, k)


def test_wall_light_below_the_range_of_the_shade(pkg, oracle, scenes):
    """A viewer outside every room sees a wall of another sector from its far side: the light of the first column is
    -2 147 316 498, which the shade's base less it does not fit 32 bits.  The column is the darkest, not the brightest."""

    sc, _ = scenes("c2")
    lanes, things = stepper.random_lanes(sc, 3, 0, seed=3)
    _place(lanes, slice(0, 3), [302.71452, 302.71452, 303.0], [-24.25008, -24.2, -24.25008])
    lanes[:, gdstate.L_ANGLE_BAM] = 770460205
    lanes.view(np.float32)[:, gdstate.L_ANGLE] = np.float32(770460205) * np.float32(gdstate.BAM_TO_RADIANS)
    lanes.view(np.float32)[:, gdstate.L_VIEW_Z] = 150.0
    _equal(oracle, sc, lanes, things, 0)


def test_status_bar_numbers(pkg, oracle, scenes):
    """One, two and three digits, the sign that is not drawn, and values past the bar's range."""

    sc, _ = scenes("c1")
    values = np.asarray([-500, -100, -99, -10, -1, 0, 1, 9, 10, 99, 100, 101, 999, 1000, 5000], dtype=np.float32)
    lanes, things = stepper.random_lanes(sc, len(values), 0, seed=8)
    lf = lanes.view(np.float32)
    lanes[:, gdstate.L_WEAPON] = np.arange(len(values)) % 8
    for word in (gdstate.L_HEALTH, gdstate.L_ARMOR, gdstate.L_READY_AMMO):
        lf[:, word] = np.roll(values, word)
    for word in range(gdstate.L_AMMO0, gdstate.L_AMMO3 + 1):
        lf[:, word] = np.roll(values, 3 * word)
    _equal(oracle, sc, lanes, things, 0)


@pytest.mark.parametrize("config,things,seed,rows", [("c4s", 24, 5, (2, 83, 224, 275)), ("c2", 12, 5, (2, 99, 100))])
def test_planes_on_both_sides_of_the_horizon(pkg, oracle, scenes, config, things, seed, rows):
    """Views whose whole columns are one floor or ceiling: its span has rows at the horizon, which need 64 bits."""

    sc, _ = scenes(config)
    lanes, records = (a[list(rows)] for a in stepper.random_lanes(sc, 300, things, seed=seed))
    _equal(oracle, sc, np.ascontiguousarray(lanes), np.ascontiguousarray(records), things)


@pytest.mark.parametrize("config,things,rows", [("c4s", 24, (292,)), ("c2", 12, (95, 113)), ("c2", 12, ())])
def test_unclaimed_pixels_far_from_their_anchors(pkg, oracle, scenes, config, things, rows):
    """Unclaimed pixels that the columns near them do not decide, so that all 320 are repaired; without `rows`, viewers
    outside the map at many headings, of whose columns none to all find a resolved row below."""

    sc, _ = scenes(config)
    lanes, records = stepper.random_lanes(sc, 300, things, seed=5)
    lanes, records = (np.ascontiguousarray(a[list(rows)] if rows else a[:16]) for a in (lanes, records))
    if not rows:
        _place(lanes, slice(0, 16), np.tile([-20.0, -90.0, 700.0, 1500.0], 4), np.repeat([-15.0, -200.0, 2060.0, 2300.0], 4))
    _equal(oracle, sc, lanes, records, things)          # slices of a lane
    blob = gdscene.pack_scene(sc)
    want = oracle.render(blob, lanes, records, mask_hud=False)["indexed"]
    renderer = native.Renderer(blob, DEV, things)       # as many copies as are drawn whole
    copies = renderer.ctas // 4 // len(lanes) + 1
    many = [torch.from_numpy(np.tile(a, (copies,) + (1,) * (a.ndim - 1))).to(DEV) for a in (lanes, records)]
    _, indexed, _ = renderer.frames(*many, indexed=True, mask_hud=False)
    renderer.check_status()
    assert np.array_equal(indexed.cpu().numpy(), np.tile(want, (copies, 1, 1)))
    renderer.close()
