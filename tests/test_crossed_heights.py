"""The campaign's specifications once more, on maps where some ceilings lie below floors and some sides have no lower or
upper texture, so that two tiers of a line share rows.  Every indexed frame and observation must be equal to the oracle's."""

import numpy as np
import pytest

import test_gpu_campaign as campaign

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trial", range(campaign.FIRST, campaign.FIRST + campaign.SPECS, 4))
def test_random_scene_specification_with_ceilings_below_floors(trial, pkg, oracle, monkeypatch):
    from gradoom_b200 import scene as gdscene

    plain = gdscene.make_grid_scene

    def crossed(spec):
        sc = plain(spec)
        rng = np.random.default_rng(9900 + trial)
        low = rng.random(len(sc.sector_heights)) < 0.25
        low[rng.integers(0, low.size)] = True
        floor = sc.sector_heights[low, 0] + rng.integers(4, 9, size=low.sum()) * 8
        sc.sector_heights[low] = np.stack((floor, floor - rng.integers(1, 9, size=low.sum()) * 8), axis=1)
        bare = rng.random((len(sc.walls), 2, 2)) < rng.choice([0.0, 0.2, 0.6])
        sc.side_textures[..., 1:][bare & (sc.wall_sectors[:, 1] >= 0)[:, None, None]] = -1
        return sc

    monkeypatch.setattr(gdscene, "make_grid_scene", crossed)
    monkeypatch.delenv("GD_CAMPAIGN_LOG", raising=False)      # its lines tell of the plain maps
    campaign.test_random_scene_specification(trial, pkg, oracle)
