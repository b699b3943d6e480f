"""The work a user has this framework do, as cases to be timed and compared: batched arena ticks through BatchSim and
the serving loop, from one match to the 16,384-arena training batch.

A case is one of four kinds of program:

  train   An RL training loop on the device. Controls lie in HBM, a pass is `ticks` ticks of every arena
          (step_with_device_commands), then the resets for the next pass are chosen on the device (episode_commands:
          a goal, or 300 ticks without a touch). The first tick of the next pass applies them.
  host    A loop with its policy on the host: upload_controls, step, download the cars, the balls and the envs.
  balls   Ball trajectories: every arena's ball is put back to its start, in place on the device, and rolled out.
  serve   Clients of a Server: each submits a request with its controls and polls for its states.

Keys: arenas (serve: all clients' together), cars (2, 4 or 6 in every arena; 0: the 55 / 27 / 18 % mix of 1v1, 2v2 and
3v3), ticks (per pass), bodies (0: the default body everywhere, 1: the six hitbox presets drawn per car), graphs (1:
steps replayed as CUDA graphs), events (event records per arena; 0: no stream), meshes (2: every other arena on the
64-segment geometry), drive (0: controls drawn at random and held, 1: everybody drives, full throttle and boost, which
brings pile-ups, bumps and demolitions), clients (serve).

Outputs are the state arrays as the public structs' bytes: the framework's contract is that every bit of them is
reproduced, so nothing in them is compared by a distance.
"""
from __future__ import annotations

import numpy as np
import torch

from rocketgpu_b200 import abi, arena, autotune
from rocketgpu_b200.batch_sim import (BALL_BYTES, CAR_BYTES, CONTROLS_BYTES, ENV_BYTES, ENV_COMMAND_BYTES, PAD_BYTES,
                                      PHYSICS_EVENT_DTYPE, PHYSICS_EVENT_WINDOW_DTYPE, BatchSim, SimConfig, car_preset)
from rocketgpu_b200.server import Server

MAX_CARS = 6
RING_TICKS = 64        # ticks of controls that a state holds; passes go round
SETTLE_TICKS = 320     # from kickoff into play before the first pass
NO_TOUCH_TICKS = 300
WHEELS_BYTES = 292
PADS = 34


def _case(name, kind, arenas, cars, ticks, bodies=0, graphs=0, events=0, meshes=1, drive=0, clients=0):
    c = {"kind": kind, "arenas": arenas, "cars": cars, "ticks": ticks, "bodies": bodies, "graphs": graphs,
         "events": events, "meshes": meshes, "drive": drive, "clients": clients}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one live 3v3 match driven tick by tick from the host: a bot in the loop, latency only
        _case("match_3v3_host", "host", 1, 6, 1),
        # one 1v1 match on the device, 8 ticks per decision: evaluation of an agent
        _case("match_1v1", "train", 1, 2, 8),
        # a small vectorised environment, steps replayed as CUDA graphs as the launch config offers for such sizes
        _case("vec_2v2_graphs", "train", 96, 4, 8, graphs=1),
        # a policy on the host with an odd number of arenas: controls up, 8 ticks, states down
        _case("host_mix", "host", 333, 0, 8, bodies=1),
        # one launch sequence per tick at the size of the plain batched workload
        _case("mix_1k_per_tick", "train", 1024, 0, 1),
        # physics events recorded for rewards and analysis
        _case("mix_1k_events", "train", 1000, 0, 8, bodies=1, events=64),
        # two geometries in one batch, everybody driving: many contacts
        _case("contacts_3v3", "train", 4095, 6, 8, meshes=2, drive=1),
        # the 1v1 training batch
        _case("duel_8k", "train", 8192, 2, 8),
        # the headline: 16,384 mixed arenas, six hitbox presets, 8 ticks per step
        _case("mix_16k", "train", 16384, 0, 8, bodies=1),
        # ball prediction: half a second of 16,384 balls
        _case("balls_16k", "balls", 16384, 0, 60),
        # clients sharing one GPU through the serving loop
        _case("serve", "serve", 1024, 0, 8, clients=8),
    ]


def draw(rng):
    kind = rng.choice(["train", "train", "train", "train", "host", "balls", "serve"])

    def size(lo, hi):
        return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))

    if kind == "balls":
        return _case(None, "balls", size(1, 16384), 0, rng.choice([8, 15, 30, 60]))
    if kind == "serve":
        return _case(None, "serve", size(64, 2048), rng.choice([0, 2, 4, 6]), rng.choice([1, 4, 8]),
                     clients=rng.choice([1, 2, 5, 8]))
    cars = rng.choice([0, 0, 2, 4, 6])
    if kind == "host":
        return _case(None, "host", size(1, 2048), cars, rng.choice([1, 2, 4, 8]), bodies=rng.choice([0, 1]))
    arenas = size(1, {0: 16000, 2: 16000, 4: 12000, 6: 8000}[cars])
    return _case(None, "train", arenas, cars, rng.choice([1, 4, 8]), bodies=rng.choice([0, 1]),
                 graphs=rng.choice([0, 0, 1]), events=rng.choice([0, 0, 32]) if arenas <= 4096 else 0,
                 meshes=rng.choice([1, 1, 2]), drive=rng.choice([0, 0, 1]))


_geometry = {}


def _mesh(fine=False):
    if fine not in _geometry:
        _geometry[fine] = arena.generate_fine() if fine else arena.generate()
    return _geometry[fine]


def _car_counts(case, rng):
    n = case["arenas"]
    if case["kind"] == "balls":
        return np.zeros(n, np.int32)
    if case["cars"]:
        return np.full(n, case["cars"], np.int32)
    return rng.choice(np.array([2, 4, 6], np.int32), size=n, p=[0.55, 0.27, 0.18]).astype(np.int32)


def _teams(counts):
    """The first half of an arena's cars plays blue, the second orange."""
    slot = np.arange(MAX_CARS)[None, :]
    half = (counts // 2)[:, None]
    return ((slot >= half) & (slot < counts[:, None])).astype(np.uint8).reshape(-1)


def _controls(rows, ticks, drive, seed):
    """[ticks, rows, CONTROLS_BYTES] on the GPU: throttle, steer, pitch, yaw, roll uniform in [-1, 1], jump, boost and
    handbrake with probability 0.1, 0.3 and 0.1, each sample held for about 15 ticks. With `drive`, throttle and boost
    are full, the others small, jumps rare."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def sample():
        axes = torch.rand((rows, 5), generator=g, device="cuda") * 2 - 1
        chance = torch.rand((rows, 3), generator=g, device="cuda")
        if drive:
            axes = axes * 0.3
            axes[:, 0] = 1.0
        buttons = torch.zeros((rows, 4), dtype=torch.uint8, device="cuda")
        for k, p in enumerate((0.01, 1.0, 0.02) if drive else (0.1, 0.3, 0.1)):
            buttons[:, k] = chance[:, k] < p
        return torch.cat([axes.view(torch.uint8), buttons], 1)

    out = torch.empty((ticks, rows, CONTROLS_BYTES), dtype=torch.uint8, device="cuda")
    now = sample()
    for t in range(ticks):
        renew = torch.rand((rows, 1), generator=g, device="cuda") < 1.0 / 15.5
        now = torch.where(renew, sample(), now)
        out[t] = now
    return out


class _View:
    """Bytes of one of the batch's device arrays; it keeps the batch alive."""

    def __init__(self, sim, entry):
        self.sim = sim
        ptr = entry["__cuda_array_interface__"]["data"][0]
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (entry["count"], entry["itemsize"]),
                                         "typestr": "|u1", "strides": None, "version": 3}


def _views(sim, names):
    arrays = sim.device_arrays()
    return {n: torch.as_tensor(_View(sim, arrays[n]), device="cuda") for n in names}


class _State:
    pass


def _batch(case, rng, seed):
    n = case["arenas"]
    counts = _car_counts(case, rng)
    v, i = _mesh()
    sim = BatchSim(SimConfig(kickoff_settled=0, env_count=n, max_cars_per_env=MAX_CARS), v, i)
    if case["meshes"] == 2:
        sim.add_mesh(*_mesh(fine=True))
        sim.set_arena_meshes(np.arange(n) % 2)
    sim.set_env_car_count(counts)
    if case["kind"] != "balls":
        sim.set_teams(_teams(counts))
        if case["bodies"]:
            presets = np.stack([car_preset(k) for k in range(6)])
            sim.set_car_configs(presets[rng.integers(0, 6, n * MAX_CARS)])
        sim.reset_to_kickoff(seed)
    if case["graphs"]:
        c = autotune.get_config(sim)
        autotune.set_config(sim, c["arena_threads"], c["car_threads"], True)
    return sim


def _ball_starts(n, rng):
    """Seeded positions inside the arena, velocities up to 6000 uu/s in any direction, some spin."""
    out = np.zeros(BALL_BYTES, np.uint8)
    abi.lib().rg_default_ball_state(out.ctypes.data)
    out = np.tile(out, (n, 1))
    pos = np.stack([rng.uniform(-3000, 3000, n), rng.uniform(-4000, 4000, n), rng.uniform(150, 1800, n)], 1)
    d = rng.normal(size=(n, 3))
    vel = d / np.linalg.norm(d, axis=1, keepdims=True) * rng.uniform(0, 6000, (n, 1))
    for at, x in ((40, pos), (68, vel), (80, rng.uniform(-4, 4, (n, 3)))):
        out[:, at:at + 12] = np.ascontiguousarray(x, np.float32).view(np.uint8)
    return out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    s = _State()
    s.case, s.at = case, 0
    n, ticks, kind = case["arenas"], case["ticks"], case["kind"]
    if kind == "serve":
        share = [n // case["clients"] + (k < n % case["clients"]) for k in range(case["clients"])]
        v, i = _mesh()
        s.server = Server(v, i, max_arenas=n, max_cars_per_env=MAX_CARS)
        s.clients = []
        for k, m in enumerate(share):
            counts = _car_counts({**case, "arenas": m}, rng)
            client = s.server.open_client(counts, _teams(counts), kickoff_seed=seed * 100 + k)
            block = _controls(m * MAX_CARS, RING_TICKS, 0, seed * 100 + k).cpu().numpy()
            s.clients.append((client, [np.ascontiguousarray(block[t:t + ticks]) for t in range(0, RING_TICKS, ticks)],
                              block))
        for t in range(0, SETTLE_TICKS, 8):
            sent = [(s.server.submit(c, np.ascontiguousarray(b[t % RING_TICKS:t % RING_TICKS + 8])), c)
                    for c, _, b in s.clients]
            for request, _ in sent:
                while s.server.poll(request, wait_ms=1000) is None:
                    pass
        return s
    s.sim = _batch(case, rng, seed)
    if kind == "balls":
        s.sim.upload_ball_states(_ball_starts(n, rng))
        s.out = _views(s.sim, ("ball_states", "env_states"))
        s.start = s.out["ball_states"].clone()
        return s
    rows = n * MAX_CARS
    ring = _controls(rows, RING_TICKS, case["drive"], seed)
    commands = torch.zeros((8, n, ENV_COMMAND_BYTES), dtype=torch.uint8, device="cuda")
    s.sim.episode_commands(NO_TOUCH_TICKS, commands.data_ptr(), stagger_seed=seed + 1, init=True)
    s.ring, s.commands = ring, commands
    s.windows = None
    for t in range(0, SETTLE_TICKS, 8):
        s.sim.step_with_device_commands(ring[t % RING_TICKS].data_ptr(), rows, commands.data_ptr(), n, 8)
        s.sim.episode_commands(NO_TOUCH_TICKS, commands.data_ptr())
    if kind == "host":
        host = ring[::ticks].cpu().numpy()
        s.ring = [host[k] for k in range(len(host))]
        return s
    s.out = _views(s.sim, ("car_states", "ball_states", "env_states", "boost_pad_states"))
    if case["events"]:
        s.records = torch.zeros((n, case["events"] * PHYSICS_EVENT_DTYPE.itemsize), dtype=torch.uint8, device="cuda")
        s.windows = torch.zeros((n, PHYSICS_EVENT_WINDOW_DTYPE.itemsize), dtype=torch.uint8, device="cuda")
        s.sim.set_physics_event_stream(s.records.data_ptr(), s.windows.data_ptr(), case["events"])
        s.out = {**s.out, "events": s.records, "event_windows": s.windows}
    return s


def run(s):
    c = s.case
    n, ticks, kind = c["arenas"], c["ticks"], c["kind"]
    at, s.at = s.at, s.at + 1
    if kind == "balls":
        s.out["ball_states"].copy_(s.start)
        s.sim.step(ticks)
        return s.out
    if kind == "host":
        s.sim.upload_controls(s.ring[at % len(s.ring)])
        s.sim.step(ticks)
        return {"cars": s.sim.download_car_states(), "balls": s.sim.download_ball_states(),
                "envs": s.sim.download_env_states()}
    if kind == "serve":
        sent = [(s.server.submit(client, blocks[at % len(blocks)]), client) for client, blocks, _ in s.clients]
        out = {}
        for k, (request, client) in enumerate(sent):
            while (got := s.server.poll(request, client, wait_ms=1000)) is None:
                pass
            out["client%d" % k] = {"cars": got[1], "balls": got[2], "envs": got[3]}
        return out
    if s.windows is not None:
        s.windows.zero_()
    block = s.ring[at * ticks % RING_TICKS]
    s.sim.step_with_device_commands(block.data_ptr(), n * MAX_CARS, s.commands.data_ptr(), n, ticks)
    s.sim.episode_commands(NO_TOUCH_TICKS, s.commands.data_ptr())
    return s.out


def work(case):
    """State read and written once per pass, controls read once; FP32 operations per car-tick and ball-tick as counted
    on the mixed workload (16,294 thread-instructions per arena-tick) and on ball-only arenas (388)."""
    n = case["arenas"]
    if case["kind"] == "balls":
        return {"bytes": n * 2 * (BALL_BYTES + ENV_BYTES), "flops": n * case["ticks"] * 388}
    cars = n * (case["cars"] or 3.26)
    state = n * (BALL_BYTES + ENV_BYTES + PADS * PAD_BYTES) + cars * (CAR_BYTES + WHEELS_BYTES)
    return {"bytes": 2 * state + case["ticks"] * cars * CONTROLS_BYTES + n * ENV_COMMAND_BYTES
            + n * case["events"] * PHYSICS_EVENT_DTYPE.itemsize,
            "flops": case["ticks"] * (cars * 4880 + n * 388)}
