"""Every candidate of the island-scheduling autotuner is a schedule of its own:
in a step that tries a limit other than the default, the islands go to the
kernels that the limit names.  (The default follows the step's islands: a small
step gives small islands a warp each, and its few large ones a CTA each.)"""
import pytest

import worldio
from reactphysics3d_b200 import engine, scenes

pytestmark = pytest.mark.gpu
DT = float(worldio.DT)


def _settled(ctx, sc, steps):
    sc.settings["sleeping_enabled"] = 0
    w = engine.World(ctx, sc)
    w.update(DT, steps)
    return w


def test_small_limits_are_the_ones_that_run(cuda_lib):
    ctx = engine.Context(0)
    w = _settled(ctx, scenes.box_pile(6, 1, 6, seed=3, spacing=3.0), 60)   # boxes that lie apart: one manifold an island
    w.update(DT)
    assert ctx.dynamics_routes() == {"thread": 0, "warp": 36, "cta": 0, "streamed": 0}
    w.autotune(rounds=1)
    seen = []
    for _ in range(9):
        w.update(DT)
        seen.append(ctx.dynamics_routes())
    assert not w.tuning()["tuning"]
    # the default, then 4, 16, 32 manifolds
    assert [r["thread"] for r in seen[:4]] == [0, 36, 36, 36], seen
    assert [r["warp"] for r in seen[:4]] == [36, 0, 0, 0], seen
    w.close()
    ctx.close()


def test_cta_limits_are_the_ones_that_run(cuda_lib):
    ctx = engine.Context(0)
    w = _settled(ctx, scenes.box_pile(6, 6, 6, seed=3), 100)
    w.update(DT)
    assert ctx.dynamics_routes()["cta"] >= 1
    w.autotune(rounds=1)
    seen = []
    for _ in range(9):
        w.update(DT)
        r = ctx.dynamics_routes()
        seen.append((r["cta"], r["warp"]))
    assert len(w.contacts()[0]) <= 512
    # the default (256, which a few large islands do not wait for), 128, 512
    assert seen[4][0] >= 1 and seen[5][0] >= 1 and seen[6][0] == 0 and seen[6][1] >= 1, seen
    w.close()
    ctx.close()
