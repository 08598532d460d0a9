"""The lane stepper's fused kernels against the same rules as tensor operations."""

import pytest
import torch

import __graft_entry__ as entry

entry.load_package()
from gradoom_b200 import native, scene as gdscene, stepper  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TIMEOUT = 9


def _pair(config, n, k, max_things, frame_skip=2):
    """Two steppers in the same state; the first one is bound to a renderer."""

    sc = gdscene.make_grid_scene(gdscene.GRID_CONFIGS[config])
    a, b = (stepper.LaneStepper(sc, n, device=DEV, k_things=k, max_things=max_things, frame_skip=frame_skip,
                                episode_timeout=TIMEOUT, seed=5) for _ in range(2))
    a.bind_renderer(native.Renderer(gdscene.pack_scene(sc), DEV, max_things))
    return a, b


def _same(a, b):
    for name in ("lanes", "players", "things", "signal_buffer", "pending_reset"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name


@pytest.mark.parametrize("config,n,k,max_things,columns", [
    ("c1", 1, 0, 0, 20), ("c1", 3, 1, 4, 1), ("c2", 4099, 12, 12, 20),
    ("c4", 130, 64, 64, 20), ("c3", 257, 5, 16, 40)])
def test_step_and_reset_kernels(config, n, k, max_things, columns):
    a, b = _pair(config, n, k, max_things)
    g = torch.Generator(DEV).manual_seed(n)
    kills = 0
    for tick in range(7):
        seeds = torch.randint(-(1 << 62), 1 << 62, (n,), device=DEV, generator=g)
        mask = torch.rand(n, device=DEV, generator=g) < (1.0 if tick == 0 else 0.3)
        a.reset(mask, seeds)
        b.reset(mask, seeds)                          # without a renderer: tensor operations
        _same(a, b)
        buttons = torch.rand((n, columns), device=DEV, generator=g) < 0.5
        got = a.step(buttons)
        b.renderer, b._tick = a.renderer, b._tick + 1
        want = b._step_tensors(buttons)
        b.renderer = None
        for x, y in zip(got, want):
            assert x.dtype == y.dtype and torch.equal(x, y)
        kills += int(got[0].sum())
        _same(a, b)
    assert bool(a.pending_reset.any()) or n < 100
    assert kills > 0 or n * k < 1000


def test_replaced_buffers_and_other_buttons_still_step():
    a, b = _pair("c1", 40, 2, 2)
    b.bind_renderer(a.renderer)
    seeds = torch.arange(40, device=DEV)
    a.reset(seeds >= 0, seeds)
    b.reset(seeds >= 0, seeds)
    b.signal_buffer = torch.zeros((40, 40), device=DEV)[:, :27].copy_(b.signal_buffer)
    buttons = (seeds[:, None] >> torch.arange(5, device=DEV)) & 1
    for x, y in zip(a.step(buttons != 0), b.step(buttons)):
        assert torch.equal(x, y)
    _same(a, b)
