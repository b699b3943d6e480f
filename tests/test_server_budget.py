"""The device memory of a serving pool against the bytes per slot that size it by hbm_budget_bytes."""
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def test_pool_takes_no_more_than_its_slots_are_counted_for(arena_mesh):
    """A pool of 2^19 slots of one car less a pool of one slot: the mesh and what a process allocates once cancel. Every
    array but the teams' bytes then fills whole 2 MiB pages; the teams' half MiB may take one."""
    import torch

    from rocketgpu_b200.server import Server

    def used(slots):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        server = Server(*arena_mesh, max_arenas=slots, max_cars_per_env=1)
        torch.cuda.synchronize()
        taken, stats = before - torch.cuda.mem_get_info()[0], server.stats()
        server.close()
        return taken, stats

    used(1)
    one, _ = used(1)
    many, stats = used(1 << 19)
    assert stats["capacity"] == 1 << 19
    assert many - one <= stats["capacity"] * stats["slot_bytes"] + 2 * MIB, (many - one, stats)
