"""Columns whose claims do not continue one another (crossings behind projected solids, tiers that overlap, rows nothing
claims) next to those whose claims do, against the oracle: viewers on lines, on corners, beside them and outside."""

import dataclasses

import numpy as np
import pytest
import torch

import __graft_entry__ as entry

entry.load_package()
from gradoom_b200 import native, scene as gdscene, state as gdstate, stepper  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("config,changes", [
    ("c1", {}), ("c1", {"diagonals": True, "floor_max": 128, "seed": 31}), ("c1m", {"mid_textures": 0.9}),
    ("c4s", {"rows": 4, "cols": 4, "diagonals": True, "seed": 9}), ("c2", {"room": 64.0, "floor_max": 96, "seed": 5})])
def test_views_from_lines_and_corners(oracle, config, changes):
    spec = dataclasses.replace(gdscene.GRID_CONFIGS[config], **changes)
    sc = gdscene.make_grid_scene(spec)
    blob = gdscene.pack_scene(sc)
    n, k = 128, 5
    lanes, things = stepper.random_lanes(sc, n, k, seed=3)
    rng = np.random.default_rng(8)
    kind = rng.integers(0, 4, n)
    for axis, count, fixed, word in ((0, spec.cols, gdstate.L_X_FIXED, gdstate.L_X), (1, spec.rows, gdstate.L_Y_FIXED, gdstate.L_Y)):
        line = rng.integers(0, count + 1, n) * spec.room
        place = np.where(kind == 0, line, np.where(kind == 1, line + rng.integers(-2, 3, n),
                         np.where((kind == 2) & (axis == 0), line + rng.uniform(-1, 1, n), rng.uniform(-64, count * spec.room + 64, n))))
        lanes[:, fixed] = np.round(place * 65536).astype(np.int64).astype(np.int32)
        lanes.view(np.float32)[:, word] = lanes[:, fixed].astype(np.float32) / np.float32(65536)
    lanes.view(np.float32)[:, gdstate.L_VIEW_Z] += rng.choice([0.0, 0.0, -30.0, 60.0], n).astype(np.float32)
    r = native.Renderer(blob, DEV, k)
    for count in (n, 20):                    # whole lanes, and few enough for slices of them
        part = [np.ascontiguousarray(a[:count]) for a in (lanes, things)]
        want = oracle.render(blob, *part, mask_hud=True)
        obs, indexed, _ = r.frames(*(torch.from_numpy(a).to(DEV) for a in part), obs=True, indexed=True, mask_hud=True, include_hud=False)
        rows = np.nonzero((indexed.cpu().numpy()[:, :208] != want["indexed"][:, :208]).any(axis=(1, 2)))[0]
        assert rows.size == 0, (rows, kind[rows])
        assert np.array_equal(obs.cpu().numpy(), want["obs"])
    r.check_status()
    r.close()


@pytest.mark.parametrize("lower", ["as packed", "on some lines", "on no line"])
@pytest.mark.parametrize("config,changes", [
    ("c1", {"floor_max": 160, "ceil_lo": 96}), ("c2", {"ceil_lo": 96}), ("c1m", {"floor_max": 160, "ceil_lo": 96}),
    ("c4s", {"rows": 4, "cols": 4, "floor_max": 160, "ceil_lo": 96})])
def test_tiers_of_a_line_that_share_rows(oracle, config, changes, lower):
    """Sectors whose ceiling lies below their floor, seen from rooms that reach farther down and up: the line between has
    an upper and a lower tier in the same rows.  Those are the lower tier's, or nobody's where it has no texture."""

    spec = dataclasses.replace(gdscene.GRID_CONFIGS[config], **changes)
    sc = gdscene.make_grid_scene(spec)
    rng = np.random.default_rng(4)
    if lower != "as packed":
        bare = rng.random(sc.side_textures.shape[:2]) < (0.5 if lower == "on some lines" else 1.0)
        sc.side_textures[..., 1][bare] = -1
    blob = gdscene.pack_scene(sc)
    sides = []                               # of lines with such a sector beyond: line, side, lowest and highest shared height
    for wall, pair in enumerate(sc.wall_sectors):
        for side in range(2):
            if pair[1] < 0 or pair[0] == pair[1]:
                continue
            (floor, ceil), (floor2, ceil2) = sc.sector_heights[pair[side]], sc.sector_heights[pair[1 - side]]
            if ceil - floor >= 56 and floor < floor2 and ceil > ceil2 and max(floor, ceil2) < min(floor2, ceil):
                sides.append((wall, side, max(floor, ceil2), min(floor2, ceil)))
    assert sides
    n, k = 96, 5
    lanes, things = stepper.random_lanes(sc, n, k, seed=6)
    lf, shared = lanes.view(np.float32), 0
    for lane in range(n):
        wall, side, low, high = sides[lane % len(sides)]
        x1, y1, x2, y2 = (float(c) for c in sc.walls[wall])
        nx, ny = np.array([y2 - y1, x1 - x2]) / np.hypot(x2 - x1, y2 - y1) * (1 if side == 0 else -1)
        away, along = rng.uniform(24, spec.room - 24), rng.uniform(0.2, 0.8)
        bam = int((np.arctan2(-ny, -nx) + rng.uniform(-0.4, 0.4)) / (2 * np.pi) * 2 ** 32) % 2 ** 32
        for place, fixed, word in ((x1 + along * (x2 - x1) + away * nx, gdstate.L_X_FIXED, gdstate.L_X),
                                   (y1 + along * (y2 - y1) + away * ny, gdstate.L_Y_FIXED, gdstate.L_Y)):
            lanes[lane, fixed] = round(place * 65536)
            lf[lane, word] = np.float32(lanes[lane, fixed]) / np.float32(65536)
        lanes[lane, gdstate.L_ANGLE_BAM] = np.uint32(bam).view(np.int32)
        lf[lane, gdstate.L_ANGLE] = np.float32(bam) * np.float32(gdstate.BAM_TO_RADIANS)
        lf[lane, gdstate.L_VIEW_Z] = sc.sector_heights[sc.wall_sectors[wall, side], 0] + stepper.VIEW_HEIGHT
        rows = np.clip(104 - (np.array([high, low]) - lf[lane, gdstate.L_VIEW_Z]) * 192 / away, 0, 208)
        shared += bool(rows[1] - rows[0] >= 2)
    assert shared >= n // 3, shared          # the tiers do meet in the middle of the view
    r = native.Renderer(blob, DEV, k)
    for count in (n, 20):                    # whole lanes, and few enough for slices of them
        part = [np.ascontiguousarray(a[:count]) for a in (lanes, things)]
        want = oracle.render(blob, *part, mask_hud=True)
        obs, indexed, _ = r.frames(*(torch.from_numpy(a).to(DEV) for a in part), obs=True, indexed=True, mask_hud=True, include_hud=False)
        wrong = (indexed.cpu().numpy()[:, :208] != want["indexed"][:, :208]).any(axis=(1, 2))
        assert not wrong.any(), (np.nonzero(wrong)[0], shared)
        assert np.array_equal(obs.cpu().numpy(), want["obs"])
    r.check_status()
    r.close()
