"""Shortcuts in the tick's headers against the general path they stand for, on the CPU: the headers are host code too,
so they are compiled as they are and, for the general path, with the shortcut's line taken out."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from rocketgpu_b200 import build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "rocketgpu_b200", "csrc")
MC = 6


def _build(tmp, name, edits=()):
    """The headers with `edits` [(file, line to take out)] as a shared library."""
    src = os.path.join(tmp, name)
    shutil.copytree(CSRC, src)
    for f, line in edits:
        path = os.path.join(src, f)
        with open(path) as h:
            text = h.read()
        assert text.count(line) == 1, (f, line)
        with open(path, "w") as h:
            h.write(text.replace(line, ""))
    out = os.path.join(tmp, name + ".so")
    cuda = os.path.dirname(os.path.dirname(build.nvcc()))  # rg_mesh.cpp holds the mesh upload too
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-ffp-contract=off", "-w", "-I", src, "-I",
                    os.path.join(ROOT, "include"), "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "host_paths.cpp"), os.path.join(src, "rg_mesh.cpp"), "-o", out,
                    "-L", os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath," + os.path.join(cuda, "lib64")],
                   check=True)
    return ctypes.CDLL(out)


def _same(a, b):
    """Bitwise, a NaN equal to any NaN."""
    return bool(((a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))).all())


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    tmp = str(tmp_path_factory.mktemp("host_paths"))
    return (_build(tmp, "as_is"),
            _build(tmp, "general", [("rg_gjk.cuh", "    if (any_nan(xa.o) || any_nan(xb.o)) return false;\n")]))


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 3.0e38])
def test_pair_detector_of_a_body_without_a_position(libs, bad):
    """Boxes, triangles and spheres with a bad value at each place of the box's position, basis, offset and of the
    other shape, and with none: the same contacts with the shortcut as through the whole loop."""
    rng = np.random.default_rng(11)
    n = 9 + 3 + 3 + 9 + 24
    q = np.linalg.qr(rng.normal(size=(n, 3, 3)))[0]
    basis = np.ascontiguousarray(q, np.float32)
    pos = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    offset = np.tile(np.float32([0.27, 0.0, 0.41]), (n, 1))
    half = np.tile(np.float32([1.18, 0.84, 0.36]), (n, 1))
    tri = rng.uniform(-3, 3, (n, 3, 3)).astype(np.float32)
    ball = rng.uniform(-2, 2, (n, 3)).astype(np.float32)
    places = [(basis, k) for k in range(9)] + [(pos, k) for k in range(3)] + [(offset, k) for k in range(3)] + \
        [(tri, k) for k in range(9)]
    for case, (a, k) in enumerate(places):
        a.reshape(n, -1)[case, k] = bad
        ball[case, k % 3] = bad if a is tri else ball[case, k % 3]
    ptr = [x.ctypes.data_as(ctypes.c_void_p) for x in (basis, pos, offset, half)]
    got = {}
    for name, fn, other, width in (("triangle", "hp_box_triangle", tri, 5), ("ball", "hp_ball_box", ball, 17)):
        for k, lib in enumerate(libs):
            out = np.zeros((n, width), np.float32)
            getattr(lib, fn)(*ptr, other.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p), n)
            got[name, k] = out
        assert _same(got[name, 0], got[name, 1]), name
        assert got[name, 0][len(places):, 0].any(), name  # some of the sound cases touch


def _boxes(rng, v, n):
    """Boxes around mesh vertices and anywhere, from a point to the largest that one cell serves and past it, on cell
    and quantization edges, and a few that are not finite."""
    bt = v * np.float32(1 / 50)
    at = bt[rng.integers(0, len(bt), n)] + rng.normal(0, 1, (n, 3)) * rng.choice([0.0, 0.01, 1.0, 5.0], (n, 1))
    at[: n // 8] = np.round(at[: n // 8] / 2) * 2
    lo, hi = bt.min(0) - 3, bt.max(0) + 3
    at[n // 8: n // 4] = rng.uniform(lo, hi, (n // 4 - n // 8, 3))
    size = rng.choice([0.0, 0.002, 0.5, 3.9999, 4.0, 4.001, 9.0], (n, 3))
    out = np.concatenate([at, at + size], 1).astype(np.float32)
    out[-3:] = [[np.nan] * 6, [np.inf] * 3 + [np.nan] * 3, [-np.inf] * 3 + [np.inf] * 3]
    return out


@pytest.mark.parametrize("mesh", ["arena", "fine", "coarse box", "largest coordinates", "many large triangles"])
def test_query_grid_visits_what_a_scan_of_all_triangles_does(libs, mesh, arena_mesh):
    from rocketgpu_b200 import arena
    rng = np.random.default_rng(5)
    if mesh == "arena":
        v, i = arena_mesh
    elif mesh == "fine":
        v, i = arena.generate_fine()
    else:  # triangles across the whole range: 2 bt cells until their lists would grow too long
        n, scale = {"coarse box": (12, 4000.0), "largest coordinates": (4, 11500.0),
                    "many large triangles": (60, 6000.0)}[mesh]
        v = (rng.uniform(-1, 1, (3 * n, 3)) * scale).astype(np.float32)
        i = np.arange(3 * n, dtype=np.int32)
    v, i = np.ascontiguousarray(v, np.float32), np.ascontiguousarray(i, np.int32)
    boxes = _boxes(rng, v, 1500)
    cell = ctypes.c_float()
    ptr = [x.ctypes.data_as(ctypes.c_void_p) for x in (v, i, boxes)]
    wrong = libs[0].hp_query_boxes(ptr[0], ctypes.c_longlong(len(v)), ptr[1], ctypes.c_longlong(len(i)), ptr[2],
                                   len(boxes), ctypes.byref(cell))
    assert wrong == 0
    assert cell.value == (4.0 if mesh in ("largest coordinates", "many large triangles") else 2.0)


PADS = [(0, -4240, 70), (-1792, -4184, 70), (1792, -4184, 70), (-940, -3308, 70), (940, -3308, 70), (0, -2816, 70),
        (-3584, -2484, 70), (3584, -2484, 70), (-1788, -2302, 70), (1788, -2302, 70), (-2048, -1036, 70),
        (0, -1024, 70), (2048, -1036, 70), (-1024, 0, 70), (1024, 0, 70), (-2048, 1036, 70), (0, 1024, 70),
        (2048, 1036, 70), (-1788, 2302, 70), (1788, 2302, 70), (-3584, 2484, 70), (3584, 2484, 70), (0, 2816, 70),
        (-940, 3308, 70), (940, 3308, 70), (-1792, 4184, 70), (1792, 4184, 70), (0, 4240, 70), (-3584, 0, 73),
        (3584, 0, 73), (-3072, 4096, 73), (3072, 4096, 73), (-3072, -4096, 73), (3072, -4096, 73)]


class HostBatch(ctypes.Structure):
    ARRAYS = ("counts", "teams", "cfgs", "cars", "balls", "env_states", "pads", "wheels", "ball_world", "broadphase",
              "car_world", "ball_car", "pairs", "pad_pos", "pad_big")
    _fields_ = [("envs", ctypes.c_int32), ("max_cars", ctypes.c_int32), ("pad_count", ctypes.c_int32)] + \
        [(a, ctypes.c_void_p) for a in ARRAYS] + [("kickoff_seed", ctypes.c_uint64)]


def host_step(lib, sim, mesh, counts, teams, cfgs, seed, controls):
    """The batch's state as it stands, stepped on the host: (cars, balls, envs, pads) after the ticks of `controls`
    [ticks, envs * MC, 24]."""
    arrays = {"counts": np.ascontiguousarray(counts, np.int32), "teams": teams, "cfgs": cfgs,
              "cars": sim.download_car_states(), "balls": sim.download_ball_states(),
              "env_states": sim.download_env_states(), "pads": sim.download_boost_pad_states(),
              "pad_pos": np.array(PADS, np.float32), "pad_big": np.array([k >= 28 for k in range(34)], np.uint8)}
    blob, at = sim.download_internal_state(), 0
    names = {"wheel_runtime": "wheels", "car_pairs": "pairs"}
    for name, size in sim.internal_state_layout():
        if name != "car_stages":
            arrays[names.get(name, name)] = np.concatenate([blob[at:at + size], np.zeros(16, np.uint8)])
        at += size
    arrays = {k: _aligned(x) for k, x in arrays.items()}
    b = HostBatch(len(counts), MC, 34, *[arrays[a].ctypes.data for a in HostBatch.ARRAYS], seed)
    v, i = (np.ascontiguousarray(mesh[0], np.float32), np.ascontiguousarray(mesh[1], np.int32))
    lib.hp_step(ctypes.byref(b), ctypes.byref(sim.config.c), v.ctypes.data_as(ctypes.c_void_p),
                ctypes.c_longlong(len(v)), i.ctypes.data_as(ctypes.c_void_p), ctypes.c_longlong(len(i)),
                controls.ctypes.data_as(ctypes.c_void_p), len(controls))
    return arrays["cars"], arrays["balls"], arrays["env_states"], arrays["pads"]


def _aligned(a):
    """A copy at a 16-byte boundary, as the structs' host build expects."""
    raw = np.zeros(a.nbytes + 16, np.uint8)
    off = -raw.ctypes.data % 16
    out = raw[off:off + a.nbytes].view(a.dtype).reshape(a.shape)
    out[...] = a
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("mix", ["one car", "odd mix", "six cars in contact", "centre of the floor",
                                 "groups of arenas"])
def test_ticks_match_the_headers_on_the_host(libs, arena_mesh, mix):
    """The tick's kernels against the same headers stepped on the host, arena after arena, one lane per car and every
    vehicle update in the arena's order: bitwise over play with landings, wheels on cars, bumps and ball touches. Car
    totals leave partly filled warps and blocks; at the centre of the floor, where a hundred slivers meet, a car lying low
    touches more triangles than the narrowphase notes at a time; one arena has a car without a position (NaN); 2,511
    arenas of none to four cars, more than the chip holds warps for, take the turn in groups."""
    import torch

    from rocketgpu_b200.batch_sim import BatchSim, SimConfig, car_preset
    from tests import scenarios
    n, ticks, rounds, seed = {"one car": (1, 4, 40, 3), "odd mix": (67, 8, 30, 5),
                              "six cars in contact": (41, 8, 30, 7), "centre of the floor": (9, 2, 6, 9),
                              "groups of arenas": (2511, 4, 4, 13)}[mix]
    rng = np.random.default_rng(seed)
    counts = {"one car": np.array([1]), "odd mix": rng.integers(0, MC + 1, n),
              "six cars in contact": np.full(n, MC), "centre of the floor": np.full(n, 2),
              "groups of arenas": np.arange(n) % 5}[mix].astype(np.int32)
    slot = np.arange(MC)[None, :]
    teams = ((slot >= (counts // 2)[:, None]) & (slot < counts[:, None])).astype(np.uint8).reshape(-1)
    cfgs = np.stack([car_preset(k) for k in range(6)])[rng.integers(0, 6, n * MC)]
    sim = BatchSim(SimConfig(kickoff_settled=0, env_count=n, max_cars_per_env=MC), *arena_mesh)
    sim.set_env_car_count(counts)
    sim.set_teams(teams)
    sim.set_car_configs(cfgs)
    sim.reset_to_kickoff(seed)
    if mix == "six cars in contact":
        cars, balls = scenarios.contact_heavy(sim.download_car_states(), sim.download_ball_states(), counts, MC, seed)
        sim.upload_car_states(cars)
        sim.upload_ball_states(balls)
    if mix == "centre of the floor":
        cars = sim.download_car_states()
        at = np.stack([rng.uniform(-60, 60, n), rng.uniform(-60, 60, n), rng.uniform(-9, 1, n)], 1)
        at[0] = np.nan
        cars[::MC, 0:12] = at.astype(np.float32).view(np.uint8)
        sim.upload_car_states(cars)
    stream = scenarios.ControlStream(n * MC, seed, p_jump=0.1, hold_max=30)
    active = (slot < counts[:, None]).reshape(-1)
    for k in range(rounds):
        controls = np.ascontiguousarray(np.stack([stream.next() for _ in range(ticks)]))
        if mix == "six cars in contact":
            chase = scenarios.chase_ball_controls(sim.download_car_states(), sim.download_ball_states(), MC, rng)
            controls[:] = chase
        want = host_step(libs[0], sim, arena_mesh, counts, teams, cfgs, seed, controls)
        dev = torch.from_numpy(controls.reshape(-1)).cuda()
        sim.step_with_device_controls(dev.data_ptr(), ticks, n * MC)
        sim.synchronize()
        got = (sim.download_car_states(), sim.download_ball_states(), sim.download_env_states(),
               sim.download_boost_pad_states())
        for name, g, w in zip(("cars", "balls", "envs", "pads"), got, want):
            if name == "cars":
                g, w = g[active], w[active]
            assert _same(np.ascontiguousarray(g).view(np.float32), np.ascontiguousarray(w).view(np.float32)), (name, k)
    moved = sim.download_car_states()[active][:, 28:40].copy().view(np.float32)
    assert np.abs(moved[np.isfinite(moved)]).max() > 100.0
    sim.close()
