"""What a turn does with states that are not the tick's own: visit orders that name inactive slots or leave slots out, pads
that the layout does not have, launches captured for other car counts. The headers run on the CPU, with an arena's active cars in a copy of their own as the turn
keeps them, against the batch's array; on a GPU, the kernels against the headers."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from rocketgpu_b200 import build
from tests.test_host_paths import CSRC, MC, ROOT, _build, _same, host_step

OFF_MODE, OFF_ORDER = 17, 20  # env state: the visit order's mode and its slots, four bits each
OFF_DEMOED, OFF_RESPAWN = 135, 108  # car state


@pytest.fixture(scope="module")
def turn(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("turn_paths") / "turn.so")
    cuda = os.path.dirname(os.path.dirname(build.nvcc()))
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-ffp-contract=off", "-w", "-I", CSRC, "-I",
                    os.path.join(ROOT, "include"), "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "turn_paths.cpp"), "-o", out], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize("command", [0, 1], ids=["tail", "kickoff command"])
@pytest.mark.parametrize("mode,order", [(1, 0x76543210), (1, 0x76103245), (3, 0x76043215), (1, 0xFFFFFFFF), (2, 0)])
def test_visit_order_past_the_active_cars(turn, command, mode, order):
    for count in range(1, MC + 1):
        for seed in range(40):
            assert turn.tp_visit_order(command, mode, ctypes.c_uint32(order), count, seed) == 0, (count, seed)


def test_visited_slots_that_the_arena_does_not_have(turn):
    """The places visited read as the last slot where they name none of the arena's; all else stays."""
    rng = np.random.default_rng(4)
    for order in rng.integers(0, 16, (400, 8)).tolist() + [list(range(8)), [15] * 8]:
        packed = sum(s << 4 * k for k, s in enumerate(order))
        for mode in range(4):
            for max_cars in range(1, MC + 1):
                for count in range(max_cars + 1):
                    want = packed if mode in (0, 2) else sum(
                        (min(s, max_cars - 1) if k < count else s) << 4 * k for k, s in enumerate(order))
                    got = turn.tp_bound(mode, ctypes.c_uint32(packed), count, max_cars)
                    assert got & 0xFFFFFFFF == want, (order, mode, count, max_cars)


@pytest.mark.parametrize("touching", [0, 1, 20, 21, 64, 65, 128, 255])
def test_touched_pad_past_the_layout(turn, touching):
    """The layout has 20 pads."""
    for seed in range(60):
        assert turn.tp_touching(touching, seed) == 0, seed


def _game_order(order, present, demoed):
    """The game's order by its rule: a car that is back takes the place after the last car present, a demolished one trades
    places with the last one present. Slots that the order leaves out stay out."""
    count = len(demoed)

    def last(order):
        return max((k for k, s in enumerate(order) if s < count and present[s]), default=-1)

    for s in range(count):
        if not present[s] and not demoed[s] and s in order:
            p, to = order.index(s), last(order) + 1
            order.insert(min(p, to), order.pop(p))
            present[s] = 1
    for s in range(count):
        if present[s] and demoed[s] and s in order:
            p, q = order.index(s), last(order)
            order[p], order[q] = order[q], s
            present[s] = 0
    return order, present


def test_game_order_of_slots_in_it_and_left_out(turn):
    """Whole orders and uploaded ones that leave slots out (mode 3 is accepted with any order), every demolition."""
    rng = np.random.default_rng(2)
    orders = [list(rng.permutation(8)) for _ in range(60)] + [list(rng.integers(0, 16, 8)) for _ in range(60)] + \
        [[0] * 8, [7] * 8, [15] * 8]
    for order in orders:
        order = [int(s) for s in order]
        if len(set(order)) != 8:  # the rule for a slot that stands twice is the first place's; keep to left-out ones
            order = [s if s not in order[:k] else 8 + k % 8 for k, s in enumerate(order)]
        for count in range(1, MC + 1):
            for mask in (0xFF, 0, 0x15):
                demoed = rng.integers(0, 2, count).astype(np.uint8)
                present = ctypes.c_uint8(mask)
                got = turn.tp_update_order(ctypes.c_uint32(sum(s << 4 * k for k, s in enumerate(order))),
                                           ctypes.byref(present), count, demoed.ctypes.data_as(ctypes.c_void_p))
                want, bits = _game_order(list(order), [mask >> s & 1 for s in range(16)], demoed)
                assert got & 0xFFFFFFFF == sum(s << 4 * k for k, s in enumerate(want)), (order, count, mask, demoed)
                assert present.value == sum(b << s for s, b in enumerate(bits[:8]))


def test_resident_warps_by_block_size(turn):
    """168 registers: twelve warps of an SM, but one block of 256 threads; 255: eight, in blocks of any size."""
    assert [turn.tp_resident_warps(168, t) for t in (32, 64, 128, 256)] == [12, 12, 12, 8]
    assert [turn.tp_resident_warps(255, t) for t in (32, 64, 128, 256)] == [8, 8, 8, 8]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 37, 5000, 40000])
def test_ball_batches_by_block_size(arena_mesh, n):
    """A ball-only batch's arenas are spread over more warps at some block sizes than at others, with the same results."""
    from rocketgpu_b200 import abi, autotune
    from rocketgpu_b200.batch_sim import BatchSim, SimConfig
    from tests import scenarios
    ball = np.zeros(288, np.uint8)
    abi.lib().rg_default_ball_state(ball.ctypes.data)
    start = scenarios.ball_states(ball, n, seed=n)
    out = []
    for threads in (32, 64, 128, 256):
        sim = BatchSim(SimConfig(kickoff_settled=0, env_count=n, max_cars_per_env=0), *arena_mesh)
        autotune.set_config(sim, threads, 64, False)
        sim.upload_ball_states(start)
        sim.step(24)
        out.append((sim.download_ball_states(), sim.download_env_states()))
        sim.close()
    assert not np.array_equal(out[0][0], start)
    for balls, envs in out[1:]:
        assert np.array_equal(balls, out[0][0]) and np.array_equal(envs, out[0][1])


@pytest.mark.parametrize("n,sms,pads", [(1, 148, 34), (37, 4, 34), (700, 4, 64), (5000, 148, 34)])
def test_turn_plans_one_after_another(turn, n, sms, pads):
    """Car counts raised, lowered, set to none and mixed: a launch captured for any earlier plan finds no arena twice."""
    rng = np.random.default_rng(n)
    counts = [np.full(n, MC), rng.integers(0, MC + 1, n), np.full(n, 2), np.zeros(n), rng.integers(0, 2, n),
              np.arange(n) % 3 * 2, np.full(n, 1), rng.integers(0, MC + 1, n)]
    counts = np.ascontiguousarray(counts, np.int32)
    assert turn.tp_plans(counts.ctypes.data_as(ctypes.c_void_p), len(counts), n, sms, pads) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("old,new", [((6, 6, 6, 6), (2, 4, 1, 6)), ((2, 4, 6, 2), (6, 2, 2, 4)), ((1, 1, 2, 2), (6, 0, 3, 4)),
                                     ((6, 2, 4, 0), (0, 0, 1, 0))])
def test_replay_of_a_capture_after_car_counts_change(arena_mesh, old, new):
    """A caller's own capture of a step, replayed after the car counts change. The counts of the first two cases, lowered or
    traded between arenas, fit what was captured, and it steps them as a new launch would; otherwise it only has to end,
    and a new launch steps on."""
    import torch

    from rocketgpu_b200.batch_sim import BatchSim, SimConfig
    n = 600
    old, new = (np.array(c, np.int32).repeat(n // 4) for c in (old, new))
    controls = torch.zeros((4 * n * MC, 24), dtype=torch.uint8, device="cuda")
    controls.view(torch.float32)[:, 0] = 1.0

    def batch():
        sim = BatchSim(SimConfig(kickoff_settled=0, env_count=n, max_cars_per_env=MC), *arena_mesh)
        sim.set_env_car_count(old)
        sim.set_teams(np.tile((np.arange(MC) % 2).astype(np.uint8), n))
        sim.reset_to_kickoff(3)
        return sim

    def state(sim):
        torch.cuda.synchronize()
        cars = sim.download_car_states().reshape(n, MC, -1)[np.arange(MC)[None] < new[:, None]]
        return cars, sim.download_ball_states(), sim.download_env_states(), sim.download_boost_pad_states()

    sim, ref = batch(), batch()
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        sim.step_with_device_controls(controls.data_ptr(), 4, n * MC, side.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    ref.step_with_device_controls(controls.data_ptr(), 4, n * MC)
    for s in (sim, ref):
        s.set_env_car_count(new)
    graph.replay()
    torch.cuda.synchronize()
    if (new >= 1).all() and new.sum() <= old.sum():
        ref.step_with_device_controls(controls.data_ptr(), 4, n * MC)
        for a, b in zip(state(sim), state(ref)):
            assert np.array_equal(a, b)
    for s in (sim, ref):
        s.reset_to_kickoff(8)
        s.step_with_device_controls(controls.data_ptr(), 4, n * MC)
    state(sim)
    sim.close()
    ref.close()


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["kept", "uploaded"])
def test_car_count_lowered_after_play_matches_the_headers(tmp_path_factory, arena_mesh, order):
    """Six cars, of which the first is demolished and comes back, so that the game's vehicle order ends with it, and is
    demolished again; then two or three cars without a kickoff: the order visits inactive slots, and the first car, which
    does nothing, not at all. Or an uploaded order that does so and names a slot that the arena does not have. Bitwise
    as the headers step it on the host."""
    import torch

    from rocketgpu_b200.batch_sim import BatchSim, SimConfig, car_preset
    lib = _build(str(tmp_path_factory.mktemp("host")), "as_is")
    n, seed = 37, 5
    rng = np.random.default_rng(seed)
    sim = BatchSim(SimConfig(kickoff_settled=0, env_count=n, max_cars_per_env=MC), *arena_mesh)
    sim.set_env_car_count(np.full(n, MC, np.int32))
    teams = np.tile((np.arange(MC) >= 3).astype(np.uint8), n)
    cfgs = np.tile(car_preset(0), (n * MC, 1))
    sim.set_teams(teams)
    sim.set_car_configs(cfgs)
    sim.reset_to_kickoff(seed)
    sim.step(4)

    def demolish_first(seconds):
        cars = sim.download_car_states()
        cars[::MC, OFF_DEMOED] = 1
        cars[::MC, OFF_RESPAWN:OFF_RESPAWN + 4] = np.frombuffer(np.float32(seconds).tobytes(), np.uint8)
        sim.upload_car_states(cars)

    demolish_first(3 / 120)
    sim.step(8)
    assert not sim.download_car_states()[::MC, OFF_DEMOED].any()
    demolish_first(3.0)
    sim.step(1)
    want = 0x76043215
    if order == "uploaded":
        envs, want = sim.download_env_states(), 0x70643215
        envs[:, OFF_MODE] = 1
        envs[:, OFF_ORDER:OFF_ORDER + 4] = np.frombuffer(np.uint32(want).tobytes(), np.uint8)
        sim.upload_env_states(envs)
    assert (sim.download_env_states()[:, OFF_ORDER:OFF_ORDER + 4].copy().view(np.uint32) == want).all()
    counts = (2 + np.arange(n) % 2).astype(np.int32)
    sim.set_env_car_count(counts)
    active = (np.arange(MC)[None, :] < counts[:, None]).reshape(-1)
    for k in range(10):
        controls = np.zeros((4, n * MC, 24), np.uint8)
        axes = rng.uniform(-1, 1, (4, n * MC, 5)).astype(np.float32)
        axes[..., 0] = 1.0
        controls[..., :20] = axes.view(np.uint8)
        want = host_step(lib, sim, arena_mesh, counts, teams, cfgs, seed, controls)
        dev = torch.from_numpy(controls.reshape(-1)).cuda()
        sim.step_with_device_controls(dev.data_ptr(), 4, n * MC)
        sim.synchronize()
        got = (sim.download_car_states(), sim.download_ball_states(), sim.download_env_states(),
               sim.download_boost_pad_states())
        for name, g, w in zip(("cars", "balls", "envs", "pads"), got, want):
            if name == "cars":
                g, w = g[active], w[active]
            assert _same(np.ascontiguousarray(g).view(np.float32), np.ascontiguousarray(w).view(np.float32)), (name, k)
    sim.close()
