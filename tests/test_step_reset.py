"""A step and the restarted lanes' first frames drawn by one launch, against the step, the copy and the reset one by one."""

import pytest
import torch

import __graft_entry__ as entry

entry.load_package()
from gradoom_b200 import env as gdenv, native, state as gdstate, stepper  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# one lane; fewer frames than CTAs; more lanes than CTAs; tables in scratch and split lines; no things
@pytest.mark.parametrize("config,n,k,share,hud", [
    ("c1", 1, 4, 1.0, False), ("c1", 1, 0, 0.0, True), ("c2", 130, 12, 0.2, True), ("c3", 700, 5, 0.05, False),
    ("c4s", 37, 3, 1.0, False), ("c1m", 300, 2, 0.5, True)])
def test_one_launch_equals_three_calls(scenes, config, n, k, share, hud):
    sc, blob = scenes(config)
    r = native.Renderer(blob, DEV, k)
    (lanes, things), (fresh, fresh_things) = ([torch.from_numpy(a).to(DEV) for a in stepper.random_lanes(sc, n, k, seed=s)]
                                              for s in (3, 4))
    g = torch.Generator(DEV).manual_seed(n)
    stack = torch.randint(0, 256, (n, 4, 84, 84), dtype=torch.uint8, device=DEV, generator=g)
    mask = torch.rand(n, device=DEV, generator=g) < share
    want = stack.clone()
    r.step(lanes, things, want, mask_hud=not hud)
    want_final = want.clone()
    r.reset(fresh, fresh_things, mask, want, mask_hud=not hud)
    final = torch.full_like(stack, 7)
    for _ in range(2):                       # the queue is left as it was found
        got = stack.clone()
        r.step_reset(lanes, things, fresh, fresh_things, mask, got, final, mask_hud=not hud)
        assert torch.equal(got, want) and torch.equal(final, want_final)
    r.check_status()
    r.close()


def _env(sc, kind, **options):
    return kind(compiled_scenario=sc, num_envs=23, device=DEV, max_things=6, vizdoom_config={"episode_timeout": 9},
                obs_crop=(0, 32, 0, 0), obs_crop_mode="mask", **options)


@pytest.mark.parametrize("options", [{}, {"obs_layout": "hwc"}, {"stack_policy": "ring"}])
def test_environment_takes_either_route(scenes, options):
    class TwoCalls(gdenv.GraDoomVecEnv):
        def step_device(self, actions):      # a step of one's own
            return super().step_device(actions)

    sc, _ = scenes("c1")
    a, b = _env(sc, gdenv.GraDoomVecEnv, **options), _env(sc, TwoCalls, **options)
    everyone, g = torch.ones(23, dtype=torch.bool, device=DEV), torch.Generator(DEV).manual_seed(1)
    seeds = torch.arange(23, device=DEV)
    assert a._one_launch(seeds) == ("stack_policy" not in options) and not b._one_launch(seeds)
    for env in (a, b):
        env.reset_device(everyone, seeds)
        times = torch.arange(23, device=DEV, dtype=torch.int32) % 8 + 1
        env._producer.lanes[:, gdstate.L_EPISODE_TIME] = times
        env._producer.players[:, gdstate.P_EPISODE_TIME] = times
    ended = 0
    for _ in range(9):
        actions = torch.randint(0, 17, (23,), device=DEV, generator=g)
        seeds = torch.randint(0, 1 << 31, (23,), device=DEV, generator=g)
        x, y = (env.step_and_reset_device(actions, seeds) for env in (a, b))
        for name in ("observations", "rewards", "terminated", "truncated", "signals", "info_histories",
                     "final_observations", "final_signals", "final_info_histories"):
            p, q = getattr(x, name), getattr(y, name)
            assert p.dtype == q.dtype and p.stride() == q.stride() and torch.equal(p, q), name
        assert x.observations.data_ptr() == a._device_observations().data_ptr()
        ended += int(x.truncated.sum())
    assert ended > 23
    for wrong in (seeds.cpu(), seeds[:5], seeds.to(torch.float32)):
        with pytest.raises((TypeError, ValueError)):
            a.step_and_reset_device(actions, wrong)
    a.close()
    b.close()
    with pytest.raises(RuntimeError):
        a.step_and_reset_device(actions, seeds)


def test_final_stack_over_the_stack_is_refused(scenes):
    sc, blob = scenes("c1")
    n = 5
    r = native.Renderer(blob, DEV, 0)
    part = [torch.from_numpy(a).to(DEV) for a in stepper.random_lanes(sc, n, 0, seed=1)]
    mask = torch.tensor([True, False, True, False, False], device=DEV)
    both = torch.full((2 * n, 4, 84, 84), 9, dtype=torch.uint8, device=DEV)
    for a, b in ((0, 0), (0, 1), (0, n - 1), (n - 1, 0), (n, 1)):
        with pytest.raises(native.NativeError, match="overlap"):
            r.step_reset(*part, *part, mask, both[a:a + n], both[b:b + n])
    assert bool((both == 9).all())
    for a, b in ((0, n), (n, 0)):            # one behind the other is accepted
        want = both[a:a + n].clone()
        r.step(*part, want)
        final = want.clone()
        r.reset(*part, mask, want)
        r.step_reset(*part, *part, mask, both[a:a + n], both[b:b + n])
        assert torch.equal(both[a:a + n], want) and torch.equal(both[b:b + n], final)
    r.close()
