"""Where the four-lane cell loop hands over to the lane-per-cell loop (1,200 cells per
SM), with the population known to the device only: one loop, and the schedule kernel
with it, must take over exactly where the other returns, in ticks above the limit,
across it and below it."""
import numpy as np
import pytest

from helpers import random_cells, random_field
from test_gpu_batch import assert_run_equal

pytestmark = pytest.mark.gpu


def limit() -> int:
    import torch

    return 1200 * torch.cuda.get_device_properties(0).multi_processor_count


def run(marl, field, cells, dims, plan):
    """Ticks with the given cells per warp (32: by the limit; 31: a lane per cell throughout)."""
    ctx = marl.Context(dims, marl.default_params(), cell_capacity=1 << 18)
    ctx.upload_field(field)
    ctx.upload_cells(cells)
    ctx.fate_init(5, 0)
    seen = []
    for lanes, ticks in plan:
        assert marl.load().marl_ctx_set_cell_lanes(ctx.h, lanes) == 0
        for _ in range(ticks):
            seen.append(ctx.fate_stats()["population"])
            ctx.run_ticks(1)
    out = ctx.download_field().tobytes(), ctx.download_cells().tobytes(), ctx.download_light().tobytes()
    ctx.close()
    return out, seen


def test_context_with_device_fate(marl):
    dims, n = (128, 128, 64), limit() + 37_400  # cells starve: the population falls through the limit
    rng = np.random.default_rng(1)
    cells, field = random_cells(dims, n, rng), random_field(dims, rng, 2.0)
    want, seen = run(marl, field, cells, dims, [(31, 6)])
    assert seen[1] > limit() > seen[-1], seen
    for plan in ([(32, 6)], [(32, 3), (31, 3)], [(31, 2), (32, 4)]):
        assert run(marl, field, cells, dims, plan)[0] == want, plan


@pytest.mark.parametrize("device_fate", [False, True])
def test_batch(marl, device_fate):
    """Seven runs of 25,000 cells, together above the limit for the first ticks; the
    engines they are compared with stay below it."""
    runs = [((96, 96, 48), seed, 9000, 1 << 16) for seed in range(21, 28)]
    p = marl.default_params()
    b = marl.Batch(runs, p)
    b.set_device_fate(device_fate)

    def total():
        return sum(b.stats(r)["population"] for r in range(len(runs)))

    first = total()
    b.step(6)
    assert first > limit() and total() > limit()
    b.step(18)
    assert total() < limit()
    for r, (dims, seed, count, cap) in enumerate(runs):
        e = marl.Engine(dims, p, rng_seed=seed, seed_count=count, cell_capacity=cap)
        e.set_device_fate(device_fate)
        e.step(24)
        assert_run_equal(b, r, e)
        e.close()
    b.close()
