"""bench.py's times per launch: the turn that starts a step is launched once a step, the other kernels once a tick."""
import bench


def test_kernel_times_per_launch_and_step():
    steps, ticks = 5, 5 * bench.TICKS_PER_STEP
    each = {"turn_start": 0.02, "car_geometry": 0.3, "car_vehicle": 0.2, "arena_finish": 0.25, "arena_turn": 0.15}
    total = [each[n] * (steps if n == "turn_start" else ticks) for n in bench.KERNEL_NAMES]
    launch, step = bench.kernel_times(total + [0.0], ticks)
    assert all(abs(launch[n] - each[n]) < 1e-9 for n in each)
    assert all(abs(step[n] - each[n] * (1 if n == "turn_start" else bench.TICKS_PER_STEP)) < 1e-9 for n in each)
    start, turn = bench.KERNEL_BYTES["turn_start"], bench.KERNEL_BYTES["arena_turn"]
    # seven of eight turns of a step end and start a tick, the last only ends one
    ends = (2 * (288 + 44 + 34 * 16), 2 * (880 + 292) + 120 + 24 + 56)
    both = (ends[0] + 24 + 16, ends[1] + 24 + 136)
    assert all(abs(8 * turn[k] - (7 * both[k] + ends[k])) < 1e-6 for k in range(2)) and turn[2] == 0
    assert start[0] == both[0] and start[1] == both[1] - 24 - 56
