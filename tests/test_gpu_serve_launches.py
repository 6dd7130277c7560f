"""The serving engine counts the launches that the device sees, replayed ticks included: one for a tick
of the resident 2D kernel, the priming pass and two passes a stage otherwise."""

import pytest
import torch

from test_gpu_serve_engine import DEV, _drain, _half, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch,chunk,per_tick", [(64, 4, 8, 1), (256, 16, 4, 1 + 4 * 8)], ids=["resident", "passes"])
def test_launches_of_replayed_ticks(n, batch, chunk, per_tick):
    _, _, plan, pool = _setup("burgers2d", n, batch, chunk, True)
    half = _half(plan, "burgers2d", n, batch, 5)
    pool.submit(1, 5 * chunk, 0.01, half)
    assert _drain(pool) == [1]
    torch.cuda.synchronize(DEV)
    st = pool.stats()
    assert st["ticks"] == 5 and st["graph_replays"] == 4  # the first tick of a shape runs directly
    assert st["launches"] == 5 * per_tick
