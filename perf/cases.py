"""The calls this framework is used for, as cases that can be timed and compared.

A case is a dict of plain values:

``call``    which public entry point one pass goes through
            ``env``       ``GraDoomVecEnv.step_and_reset_device``: a learner on the device (actions in,
                          observations, rewards and signals out, finished lanes restarted)
            ``gym``       ``GraDoomVecEnv.step`` and, when lanes ended, ``reset`` with a mask: a gym-style loop
            ``image``     ``GraDoomVecEnv.render_lane``: one 320x240 RGB frame on the host (a viewer)
            ``engine``    ``GraDoomVecEnv.step_device`` over ``EngineStateProducer``: an engine that keeps
                          its own lane tensors (packed every step) and bullet-chip rings
            ``step``      ``native.Renderer.step``: lane records in, four-frame stack rolled
            ``ring``      ``native.Renderer.step_ring``: the same on the mirrored eight-slot ring
            ``frames``    ``native.Renderer.step_frames``: the stack and every lane's RGB24 frame
            ``reset``     ``native.Renderer.reset``: masked refill of the stack at episode starts
            ``host``      ``native.Renderer.step_host``: records and newest frames in pinned host memory
``map``     a seeded grid map of ``scene.GRID_CONFIGS``
``lanes``, ``things``   environment lanes of the call, drawable things per lane
``hud``     whether the observation shows the status bar or the masked profile's black rows

States are made from the seed on the GPU: poses uniform over the rooms, weapons and status
values in their ranges, things at uniform positions.  Lanes of the environment cases are at
different times of their episodes, as they are in a program that has run for a while.
"""

import dataclasses
import importlib
import math

import numpy as np
import torch

gradoom = importlib.import_module("env-gradoom-turbo-torch_b200")
env_api = importlib.import_module("env-gradoom-turbo-torch_b200.env")
native = importlib.import_module("env-gradoom-turbo-torch_b200.native")
gdscene, gdstate, stepper = gradoom.scene, gradoom.state, gradoom.stepper

FIXED = 1 << 16
SLOT = 84 * 84                  # bytes of one observation frame
RGB = 240 * 320 * 3
BANK = 32                       # prepared action (and seed) batches a state cycles through
EPISODE_TICS = 1050             # thirty seconds of game time
FRAME_SKIP = 4
ENGINE_ITEMS = 12
ENGINE_SLOTS = {"enemy_slots": 64, "projectile_slots": 32, "enemy_projectile_slots": 64, "puff_slots": 20,
                "items": ENGINE_ITEMS}
DECAL_SLOTS = 64
DECALS = 24
STEP_CALLS = ("step", "ring", "frames", "reset", "host")


def listed():
    def case(name, call, map_, lanes, things, hud=False):
        return {"name": name, "call": call, "map": map_, "lanes": lanes, "things": things, "hud": hud}

    return [
        # the smallest training or evaluation run: the 16-sector map with four lanes
        case("env 4 lanes", "env", "c1", 4, 4),
        # a learner that collects rollouts on one GPU with 256 lanes
        case("env 256 lanes", "env", "c2", 256, 12),
        # the same loop at a batch that fills the GPU several times over
        case("env 1024 lanes", "env", "c2", 1024, 12),
        # a gym-style loop with an odd number of lanes and the status bar in view
        case("gym 333 lanes", "gym", "c3", 333, 12, hud=True),
        # a viewer that shows one lane of a small run
        case("image of one lane", "image", "c2", 16, 12),
        # a full game engine behind the environment: state packing, map items, bullet chips
        case("engine 512 lanes", "engine", "c2", 512, 56),
        # the throughput configuration: 64 sectors, 12 things, 4096 lanes
        case("step 4096 lanes", "step", "c2", 4096, 12),
        # frames recorded with the observations: the status bar and RGB24 of every lane every step
        case("frames 1024 lanes", "frames", "c3", 1024, 12, hud=True),
        # the large map (256 sectors, 800 lines with diagonals) at 8192 lanes and 32 things
        case("step 8192 lanes, large map", "step", "c4", 8192, 32),
        # lines that a node builder split, as every compiled map has them, on the mirrored ring
        case("ring 1501 lanes, split lines", "ring", "c4s", 1501, 24),
        # masked middle textures (grates, fences) with the status bar in view
        case("step 700 lanes, grates", "step", "c1m", 700, 8, hud=True),
        # a learner on the host: records up, newest frames down, every step
        case("host 4096 lanes", "host", "c2", 4096, 12),
    ]


# call -> (maps, fewest lanes, most lanes, most things)
RANGES = {
    "env": (("c1", "c2", "c3", "c1m", "c4s"), 1, 1024, 32),
    "gym": (("c1", "c2", "c3", "c1m"), 1, 512, 32),
    "image": (("c1", "c2", "c3", "c1m", "c4s"), 1, 64, 32),
    "engine": (("c1", "c2", "c3", "c1m"), 1, 1024, 56),
    "step": (("c1", "c2", "c3", "c4", "c1m", "c4s"), 1, 4096, 64),
    "ring": (("c1", "c2", "c3", "c4", "c1m", "c4s"), 1, 4096, 64),
    "frames": (("c1", "c2", "c3", "c1m"), 1, 2048, 32),
    "reset": (("c1", "c2", "c3", "c4", "c1m", "c4s"), 1, 4096, 32),
    "host": (("c1", "c2", "c3", "c4s"), 1, 4096, 32),
}


def draw(rng):
    call = rng.choice(sorted(RANGES))
    maps, low, high, most = RANGES[call]
    lanes = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    things = 56 if call == "engine" else rng.randint(0, most)
    return {"call": call, "map": rng.choice(maps), "lanes": lanes, "things": things, "hud": rng.random() < 0.3}


# -- scenes: immutable, packed once per map --------------------------------------

_scenes = {}


def _scene(name, engine=False):
    if (name, engine) not in _scenes:
        spec = gdscene.GRID_CONFIGS[name]
        if engine:
            spec = dataclasses.replace(spec, items=ENGINE_ITEMS, decals=True)
        sc = gdscene.make_grid_scene(spec)
        _scenes[name, engine] = sc, gdscene.pack_scene(sc)
    return _scenes[name, engine]


# -- lane states -------------------------------------------------------------------


class _Draw:
    """Seeded draws on the GPU."""

    def __init__(self, seed):
        self.device = torch.device("cuda", torch.cuda.current_device())
        self.g = torch.Generator(self.device).manual_seed(int(seed))

    def uniform(self, low, high, *shape):
        return torch.rand(shape, generator=self.g, device=self.device) * (high - low) + low

    def whole(self, low, high, *shape, dtype=torch.int32):
        return torch.randint(low, high, shape, generator=self.g, device=self.device).to(dtype)

    def chance(self, p, *shape):
        return torch.rand(shape, generator=self.g, device=self.device) < p


def _bits(t):
    return t.to(torch.float32).contiguous().view(torch.int32)


def _rooms(sc, x, y):
    """Sector of points of a grid map: its rooms are the sectors, row by row."""

    spec = sc.meta["spec"]
    col = (x / spec.room).floor().clamp(0, spec.cols - 1).to(torch.int64)
    row = (y / spec.room).floor().clamp(0, spec.rows - 1).to(torch.int64)
    return row * spec.cols + col


def _coordinate(d, count, room, n):
    """Fixed-point positions in uniformly drawn rooms, at least 20 units away from the room's edges."""

    inside = d.uniform(20.0, room - 20.0, n)
    return d.whole(0, count, n, dtype=torch.int64) * int(room * FIXED) + (inside * FIXED).to(torch.int64)


def _poses(d, sc, n):
    spec = sc.meta["spec"]
    xf, yf = _coordinate(d, spec.cols, spec.room, n), _coordinate(d, spec.rows, spec.room, n)
    bam = torch.randint(0, 1 << 32, (n,), generator=d.g, device=d.device)
    x, y = xf.to(torch.float32) / FIXED, yf.to(torch.float32) / FIXED
    floors = torch.as_tensor(sc.sector_heights[:, 0].astype(np.float32), device=d.device)
    return xf, yf, bam, x, y, bam.to(torch.float32) * gdstate.BAM_TO_RADIANS, floors[_rooms(sc, x, y)]


def _lane_records(d, sc, n, things):
    """``(n,32)`` lane records and ``(n,K,4)`` thing records."""

    S = gdstate
    xf, yf, bam, x, y, angle, floor = _poses(d, sc, n)
    lanes = torch.zeros((n, S.LANE_WORDS), dtype=torch.int32, device=d.device)
    for word, value in ((S.L_X, x), (S.L_Y, y), (S.L_ANGLE, angle), (S.L_VIEW_Z, floor + 41.0),
                        (S.L_HEALTH, d.whole(0, 201, n)), (S.L_ARMOR, d.whole(0, 201, n)),
                        (S.L_READY_AMMO, d.whole(0, 301, n))):
        lanes[:, word] = _bits(value)
    for word in range(S.L_AMMO0, S.L_AMMO3 + 1):
        lanes[:, word] = _bits(d.whole(0, 301, n))
    zero = torch.zeros(n, dtype=torch.int32, device=d.device)
    for word, value in (
            (S.L_X_FIXED, xf), (S.L_Y_FIXED, yf), (S.L_ANGLE_BAM, torch.where(bam >= 1 << 31, bam - (1 << 32), bam)),
            (S.L_EPISODE_TIME, d.whole(1, EPISODE_TICS, n)), (S.L_BOB_FIXED, d.whole(0, 16 * FIXED, n)),
            (S.L_WEAPON, d.whole(0, 8, n)), (S.L_WPN_COOLDOWN, torch.where(d.chance(0.5, n), zero, d.whole(0, 20, n))),
            (S.L_WPN_FIRE_COUNT, d.whole(0, 9, n)), (S.L_WPN_READY_TICS, d.whole(0, 40, n)),
            (S.L_WPN_RAISE, torch.where(d.chance(0.8, n), zero, d.whole(0, 15, n))), (S.L_WPN_LOWER, d.whole(0, 17, n)),
            (S.L_WPN_PENDING, torch.where(d.chance(0.9, n), zero - 1, d.whole(0, 8, n))),
            (S.L_WEAPONS_OWNED, d.whole(0, 64, n) | 3), (S.L_FACE_INDEX, d.whole(0, 3, n)),
            (S.L_PAIN_DIRECTION, d.whole(0, 3, n)),
            (S.L_PAIN_TICS, torch.where(d.chance(0.8, n), zero, d.whole(1, 35, n))),
            (S.L_GRIN_TICS, torch.where(d.chance(0.9, n), zero, d.whole(1, 71, n))),
            (S.L_ATTACK_HELD, torch.where(d.chance(0.9, n), zero, d.whole(70, 100, n))),
            (S.L_FLAGS, d.chance(0.03, n).to(torch.int32) | (d.chance(0.1, n).to(torch.int32) << 1)),
            (S.L_THINGS, zero + things)):
        lanes[:, word] = value.to(torch.int32)
    records = torch.zeros((n, max(things, 1), 4), dtype=torch.int32, device=d.device)
    if things:
        spec = sc.meta["spec"]
        tx = d.uniform(8.0, spec.cols * spec.room - 8.0, n, things)
        ty = d.uniform(8.0, spec.rows * spec.room - 8.0, n, things)
        floors = torch.as_tensor(sc.sector_heights[:, 0].astype(np.float32), device=d.device)
        styles = torch.tensor([-1, -1, -1, -1, 0, 1, -2], device=d.device)[d.whole(0, 7, n, things, dtype=torch.int64)]
        records = gdstate.pack_things(tx, ty, floors[_rooms(sc, tx, ty)], d.whole(0, len(sc.spr_atlas), n, things),
                                      d.chance(0.95, n, things), d.chance(0.1, n, things), styles)
    return lanes, records


class _Engine:
    """What a game engine behind the environment looks like to it: the lane tensors under the
    reference engine's names and dtypes, with every class of actors in use, and bullet-chip
    rings.  Its own step only turns the players and lets time pass."""

    def __init__(self, d, sc, n):
        spec, counts = sc.meta["spec"], ENGINE_SLOTS
        wide, high = spec.cols * spec.room, spec.rows * spec.room
        floors = torch.as_tensor(sc.sector_heights[:, 0].astype(np.float32), device=d.device)
        shapes = {}
        for _field, name, dtype, shape in gdstate.ENGINE_STATE_POINTERS:
            dims = (n,) if shape is None else (n, shape if isinstance(shape, int) else counts[shape])
            shapes[name] = dims
            if dtype == torch.float32:
                t = d.uniform(0.0, 200.0, *dims)
            elif dtype == torch.uint8:
                t = d.chance(0.15, *dims)
            elif dtype == torch.int64:
                t = d.whole(0, 6, *dims, dtype=torch.int64)
            else:
                t = d.whole(0, 40, *dims) * d.chance(0.2, *dims)
            setattr(self, name, t)
        for stem in ("enemy", "teleport_fog", "drop", "projectile", "enemy_projectile", "hitscan_puff"):
            x = d.uniform(20.0, wide - 20.0, *shapes[stem + "_x"])
            y = d.uniform(20.0, high - 20.0, *shapes[stem + "_y"])
            setattr(self, stem + "_x", x)
            setattr(self, stem + "_y", y)
            lift = 32.0 if "proj" in stem or "puff" in stem else 0.0
            setattr(self, stem + "_z", floors[_rooms(sc, x, y)] + lift)
        for stem in ("projectile", "enemy_projectile"):
            for axis in "xy":
                setattr(self, f"{stem}_velocity_{axis}", d.uniform(-20.0, 20.0, *shapes[stem + "_x"]))
        self._x_fixed, self._y_fixed, self._angle_bam, self.x, self.y, self.angle, floor = _poses(d, sc, n)
        self.view_z = floor + 41.0
        self._pitch_bam = torch.zeros(n, dtype=torch.int64, device=d.device)
        self._player_bob_fixed = d.whole(0, 16 * FIXED, n, dtype=torch.int64)
        self.health = d.whole(1, 201, n).to(torch.float32)
        self.episode_time = d.whole(1, EPISODE_TICS, n)
        self.selected_weapon = d.whole(0, 7, n, dtype=torch.int64)
        self.pending_weapon = torch.where(d.chance(0.9, n), -1, d.whole(0, 7, n, dtype=torch.int64))
        self.player_dead = d.chance(0.03, n)
        self.weapons = d.chance(0.5, n, 6).to(torch.float32)
        self.enemy_angle = d.uniform(-3.14, 3.14, *shapes["enemy_x"])
        self.enemy_target_slot = d.whole(-2, 4, *shapes["enemy_x"], dtype=torch.int64)
        self.enemy_attack_phase = d.whole(0, 5, *shapes["enemy_x"])
        self.enemy_animation_tics = d.whole(0, 300, *shapes["enemy_x"])
        self.enemy_death_elapsed = d.whole(0, 80, *shapes["enemy_x"])
        kinds = torch.tensor([-1, 2007, 2002, 2001], device=d.device)
        self.drop_type = kinds[d.whole(0, 4, *shapes["drop_x"], dtype=torch.int64)]
        self.projectile_type = d.whole(-1, 2, *shapes["projectile_x"], dtype=torch.int64)
        self.projectile_impact_type = d.whole(-1, 3, *shapes["projectile_x"], dtype=torch.int64)
        self.item_available = d.chance(0.8, n, ENGINE_ITEMS)
        self.item_animation_initial_tics = d.whole(1, 7, n, ENGINE_ITEMS)
        # a handful of slots of every class are in use
        for name, keep in (("enemy_alive", 6), ("enemy_death_tics", 5), ("teleport_fog_tics", 4), ("drop_spawned", 4),
                           ("projectile_alive", 4), ("projectile_impact_tics", 3), ("enemy_projectile_alive", 4),
                           ("enemy_projectile_impact_tics", 3), ("hitscan_puff_tics", 4)):
            getattr(self, name)[:, keep:] = 0
        self._chips(d, sc, n)
        self.signal_buffer = torch.zeros((n, len(env_api.DEVICE_SIGNAL_NAMES)), device=d.device)
        self.pending_reset = torch.zeros(n, dtype=torch.bool, device=d.device)
        self._none = torch.zeros(n, dtype=torch.bool, device=d.device)
        self._nothing = torch.zeros(n, device=d.device)
        self.turn = d.whole(-3, 4, n, dtype=torch.int64) * (640 << 16)

    def _chips(self, d, sc, n):
        """Chips where rays through the view meet the nearest line, on the viewer's side of it."""

        walls = torch.as_tensor(sc.walls.astype(np.float32), device=d.device)
        sx, sy = walls[:, 0], walls[:, 1]
        ex, ey = walls[:, 2] - sx, walls[:, 3] - sy
        free = DECAL_SLOTS - DECALS

        def ring(values, fill):
            return torch.cat((values, torch.full((n, free), fill, dtype=values.dtype, device=d.device)), dim=1)

        ray = self.angle[:, None] + d.uniform(-0.75, 0.75, n, DECALS)
        rx, ry = torch.cos(ray)[..., None], torch.sin(ray)[..., None]
        px, py = self.x[:, None, None], self.y[:, None, None]
        den = rx * ey - ry * ex
        den = torch.where(den.abs() > 1e-6, den, torch.full_like(den, 1e-6))
        dist = ((sx - px) * ey - (sy - py) * ex) / den
        along = ((sx - px) * ry - (sy - py) * rx) / den
        wall = torch.where((dist > 1e-3) & (along >= 0) & (along <= 1), dist, torch.inf).argmin(dim=2)
        along = along.gather(2, wall[..., None])[..., 0].clamp(0.0, 1.0)
        side = (ex[wall] * (self.y[:, None] - sy[wall]) - ey[wall] * (self.x[:, None] - sx[wall]) > 0).to(torch.int32)
        style = d.whole(0, 5, n, DECALS) + 5 * d.whole(0, 2, n, DECALS) + 10 * d.whole(0, 2, n, DECALS) + 20 * side
        serial = 1000 + torch.arange(DECALS, dtype=torch.int32, device=d.device).expand(n, DECALS)
        self.hitscan_decal_serial = ring(serial, -1)
        self.hitscan_decal_wall = ring(wall.to(torch.int32), -1)
        self.hitscan_decal_style = ring(style.to(torch.uint8), 0)
        self.hitscan_decal_along = ring(along, 0.0)
        self.hitscan_decal_z = ring(self.view_z[:, None] + d.uniform(-40.0, 60.0, n, DECALS), 0.0)

    def render_frame(self, active=None):
        return None                 # the environment draws; an engine's own renderer stays idle

    def reset(self, mask, seeds):
        self.pending_reset &= ~mask

    def step(self, buttons):
        self._angle_bam.add_(self.turn).bitwise_and_(0xFFFFFFFF)
        torch.mul(self._angle_bam, gdstate.BAM_TO_RADIANS, out=self.angle)
        self.episode_time += FRAME_SKIP
        return None, self._nothing, self._none, self._none


# -- states --------------------------------------------------------------------------


class _State:
    """What a program keeps between passes, and a counter into its bank of action batches."""

    def __init__(self, call, **things):
        self.call, self.passes = call, 0
        vars(self).update(things)

    def next(self):
        self.passes += 1
        return self.passes % BANK


def _environment(case, d, sc, producer=None, **options):
    crop = {} if case["hud"] else {"obs_crop": (0, 32, 0, 0), "obs_crop_mode": "mask"}
    return env_api.GraDoomVecEnv(compiled_scenario=sc, num_envs=case["lanes"], device=d.device, frame_skip=FRAME_SKIP,
                                 vizdoom_config={"episode_timeout": EPISODE_TICS}, producer=producer,
                                 render_mode="rgb_array", **crop, **options)


def prepare(case, seed):
    d = _Draw(seed)
    n, things, call = case["lanes"], case["things"], case["call"]
    sc, blob = _scene(case["map"], call == "engine")
    if call in STEP_CALLS:
        lanes, records = _lane_records(d, sc, n, things)
        state = _State(call, lanes=lanes, things=records, hud=case["hud"], renderer=native.Renderer(blob, d.device, things))
        slots = 8 if call == "ring" else 4
        state.stack = d.whole(0, 256, n, slots, 84, 84, dtype=torch.uint8)
        if call == "ring":
            state.stack[:, 4:] = state.stack[:, :4]
        if call == "frames":
            state.rgb = torch.empty((n, 240, 320, 3), dtype=torch.uint8, device=d.device)
        if call == "reset":
            state.mask = d.chance(0.25, n)
        if call == "host":
            state.host_lanes, state.host_things = lanes.cpu().pin_memory(), records.cpu().pin_memory()
            state.host_frames = torch.zeros((n, 84, 84), dtype=torch.uint8).pin_memory()
        return state
    everyone = torch.ones(n, dtype=torch.bool, device=d.device)
    seeds = d.whole(0, 1 << 31, BANK, n, dtype=torch.int64)
    actions = d.whole(0, len(env_api.DEATHMATCH_ACTIONS), BANK, n, dtype=torch.int64)
    if call == "engine":
        env = _environment(case, d, sc, env_api.EngineStateProducer(_Engine(d, sc, n), sc, things), max_things=things)
        env.reset_device(everyone, seeds[0])
        return _State(call, env=env, actions=actions)
    # the built-in producer, its lanes spread over their episodes
    producer = stepper.LaneStepper(sc, n, device=d.device, k_things=things, frame_skip=FRAME_SKIP,
                                   episode_timeout=EPISODE_TICS, seed=int(seed))
    env = _environment(case, d, sc, producer, max_things=things)
    if call == "gym":
        env.reset(seed=int(seed))
    else:
        env.reset_device(everyone, seeds[0])
    started = d.whole(8, EPISODE_TICS, n)
    producer.lanes[:, gdstate.L_EPISODE_TIME] = started
    producer.players[:, gdstate.P_EPISODE_TIME] = started
    return _State(call, env=env, actions=actions, seeds=seeds)


def run(state):
    call = state.call
    if call == "env":
        k = state.next()
        t = state.env.step_and_reset_device(state.actions[k], state.seeds[k])
        return (t.observations, t.rewards, t.terminated, t.truncated, t.signals, t.final_observations, t.final_signals)
    if call == "gym":
        observations, rewards, terminated, truncated, infos = state.env.step(state.actions[state.next()])
        done = terminated | truncated
        first = observations
        if bool(done.any()):
            first, _ = state.env.reset(options={"reset_mask": done})
        return observations, rewards, terminated, truncated, infos, first
    if call == "image":
        return state.env.render_lane(state.next() % state.env.num_envs)
    if call == "engine":
        t = state.env.step_device(state.actions[state.next()])
        return t.observations, t.rewards, t.terminated, t.truncated, t.signals
    r, lanes, things, mask_hud = state.renderer, state.lanes, state.things, not state.hud
    if call == "step":
        r.step(lanes, things, state.stack, mask_hud=mask_hud)
    elif call == "ring":
        r.step_ring(lanes, things, state.stack, state.next() & 3, mask_hud=mask_hud)
    elif call == "frames":
        r.step_frames(lanes, things, state.stack, rgb=state.rgb, mask_hud=mask_hud)
        return state.stack, state.rgb
    elif call == "reset":
        r.reset(lanes, things, state.mask, state.stack, mask_hud=mask_hud)
    else:
        r.step_host(state.host_lanes, state.host_things, lanes, things, state.stack, state.host_frames, mask_hud=mask_hud)
        torch.cuda.current_stream().synchronize()       # the learner reads the frames now
        return state.stack, state.host_frames
    return state.stack


def work(case):
    """Records and old frames read once, frames and results written once; the scene (2 to 5 MB,
    shared by all lanes and all calls) is left out.  The path has no floating-point contraction:
    its arithmetic is whole-number work of one texel and one light lookup for each of the 66,560
    pixels of a view, which no rate in FLOP/s describes."""

    n, things, call = case["lanes"], case["things"], case["call"]
    records = 128 + 16 * things
    rolled = 3 * SLOT + 4 * SLOT
    signals = 27 * 4
    if call == "image":
        return {"bytes": records + RGB, "flops": 0}
    if call == "env":
        return {"bytes": n * (records + rolled + 2 * 96 + 4 * SLOT + 3 * signals + 8 + 8 + 6), "flops": 0}
    if call == "gym":
        return {"bytes": n * (records + rolled + 2 * 96 + 4 * SLOT + 2 * signals + 27 * 9 + 8 + 6), "flops": 0}
    if call == "engine":
        engine = sum(torch.empty((), dtype=dtype).element_size()
                     * (1 if shape is None else shape if isinstance(shape, int) else ENGINE_SLOTS[shape])
                     for _field, _name, dtype, shape in gdstate.ENGINE_STATE_POINTERS)
        return {"bytes": n * (engine + 17 * DECAL_SLOTS + rolled + signals + 8 + 6), "flops": 0}
    if call == "reset":
        return {"bytes": n + n * 0.25 * (records + 4 * SLOT), "flops": 0}
    written = {"step": rolled, "ring": 2 * SLOT, "frames": rolled + RGB, "host": rolled + SLOT}[call]
    return {"bytes": n * (records + written), "flops": 0}


def tolerance(case):
    """Palette indices, frames, rewards and counters are whole-number results."""

    return "exact"
