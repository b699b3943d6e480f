"""rg_batch_phase_timing: six parts of a tick under enable = 1, five launches under 2, the same states under both."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_parts_and_launches(arena_mesh):
    import torch

    from rocketgpu_b200 import abi
    from rocketgpu_b200.batch_sim import BatchSim, SimConfig
    n, ticks, steps = 300, 8, 6
    counts = (np.arange(n) % 4).astype(np.int32) + 1
    lib = abi.lib()
    states = []
    for enable in (0, 1, 2):
        sim = BatchSim(SimConfig(kickoff_settled=0, env_count=n, max_cars_per_env=6), *arena_mesh)
        sim.set_env_car_count(counts)
        sim.set_teams(np.tile((np.arange(6) % 2).astype(np.uint8), n))
        sim.reset_to_kickoff(4)
        g = torch.Generator().manual_seed(1)
        rows = torch.zeros((ticks, n * 6, 24), dtype=torch.uint8)
        rows.view(torch.float32)[..., 0:5] = torch.rand((ticks, n * 6, 5), generator=g) * 2 - 0.5
        rows[..., 20:22] = 1
        controls = rows.cuda()
        commands = torch.zeros((ticks, n, 16), dtype=torch.uint8, device="cuda")
        sim.episode_commands(20, commands.data_ptr(), stagger_seed=2, init=True)
        assert lib.rg_batch_phase_timing(sim._h, enable) == 0
        for _ in range(steps):
            sim.step_with_device_commands(controls.data_ptr(), n * 6, commands.data_ptr(), n, ticks)
            sim.episode_commands(20, commands.data_ptr())
        ms, count = (ctypes.c_float * 6)(*[-1.0] * 6), ctypes.c_int64(-1)
        assert lib.rg_batch_phase_times(sim._h, ms, ctypes.byref(count)) == 0
        assert count.value == (ticks * steps if enable else 0)
        assert [m > 0 for m in ms] == [enable > 0] * 5 + [enable == 1], list(ms)
        assert lib.rg_batch_phase_timing(sim._h, 0) == 0
        states.append((sim.download_car_states(), sim.download_ball_states(), sim.download_env_states(),
                       sim.download_boost_pad_states()))
        sim.close()
    for other in states[1:]:
        for a, b in zip(states[0], other):
            assert np.array_equal(a, b)
