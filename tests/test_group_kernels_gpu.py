"""World groups at the sizes where a group's kernels change their route: trees
of the size that still fits the reinsertion kernel's shared memory, one leaf
more and a single leaf (against the same group with host trees), and more
islands with joints than the joint kernels give a warp each (against the worlds
stepped alone)."""
import numpy as np
import pytest
import torch

import worldio
from reactphysics3d_b200 import engine, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cuda_lib):
    c = engine.Context(0)
    yield c
    c.close()


def _same(a, ka, b, kb, what):
    assert np.array_equal(a.pairs(ka), b.pairs(kb)), what
    for x, y in zip(a.bodies(ka), b.bodies(kb)):
        assert np.array_equal(x, y), what


def test_trees_around_the_shared_memory_limit(ctx):
    # n colliders make 2 n nodes with the free one: 1,024 fit
    raw = [scenes.box_pile(7, 73, 1, seed=1, spacing=1.1, jitter=0.3), scenes.box_pile(8, 64, 1, seed=2, spacing=1.1, jitter=0.3),
           scenes.box_pile(1, 1, 1, seed=3), scenes.box_pile(4, 4, 4, seed=4, spacing=1.2)]
    shapes, scs = scenes.merge_shapes(raw)
    a = engine.WorldGroup(ctx, scs, shapes, threads=2)
    b = engine.WorldGroup(ctx, scs, shapes, threads=2)
    b.set_device_trees(False)
    assert a.device_trees and not b.device_trees
    for step in range(40):
        a.update(float(worldio.DT))
        b.update(float(worldio.DT))
        if step % 8 == 7:
            for k in range(len(scs)):
                _same(a, k, b, k, (step, k))
    assert a.stats()["overlapping_pairs"] > 0
    a.close()
    b.close()


def test_more_joint_islands_than_warps(ctx):
    per_world = 4 * torch.cuda.get_device_properties(0).multi_processor_count + 7
    raw = [scenes.ragdoll_world(per_world, seed=5), scenes.ragdoll_world(per_world, seed=6)]
    shapes, scs = scenes.merge_shapes(raw)
    g = engine.WorldGroup(ctx, scs, shapes, threads=2)
    g.update(float(worldio.DT), 12)
    for k, sc in enumerate(raw):
        sh, one = scenes.merge_shapes([sc])
        w = engine.WorldGroup(ctx, one, sh, threads=2)
        w.update(float(worldio.DT), 12)
        _same(g, k, w, 0, k)
        w.close()
    g.close()
