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
