"""Colliders with more partners than a walk of their own is kept up for: warps
with many such colliders (walked together), with one or three (walked alone),
at the number of partners where the walk is given up, with groups, filters that
drop partners, and a capacity smaller than the number of pairs.  The pairs and
their order are exact."""
import numpy as np
import pytest

import bpio
from reactphysics3d_b200 import engine
from test_broadphase_sizes_gpu import _ordered, _positions, _search

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cuda_lib):
    c = engine.Context(0)
    yield c
    c.close()


def _clumps(sizes, rng, bodies):
    """Boxes that all overlap inside a clump, clumps apart."""
    mn = np.zeros((sum(sizes), 4), np.float32)
    at = 0
    for k, m in enumerate(sizes):
        mn[at:at + m, :3] = (20.0 * k, 0.0, 0.0) + rng.uniform(-0.4, 0.4, (m, 3))
        at += m
    mx = mn.copy()
    mx[:, :3] += 1.0
    return mn, mx, (rng.integers(0, bodies, len(mn)) if bodies else np.arange(len(mn))).astype(np.int32)


# (clump sizes, bodies to share or 0, groups, boxes that span everything)
CASES = {
    "at the limit": ([64, 65, 66, 67, 68], 0, 0, 0),
    "few dense lanes": ([66] * 12, 0, 0, 0),
    "all": ([700], 0, 0, 0),
    "a warp and more": ([33, 130, 31, 96, 1, 1, 300], 0, 0, 0),
    "shared bodies": ([400, 150], 60, 0, 0),
    "grounds": ([2] * 150, 0, 0, 3),
    "groups": ([500], 0, 3, 0),
}


@pytest.mark.parametrize("name", CASES)
def test_dense_pairs_and_their_order(ctx, port, name):
    sizes, bodies, groups, grounds = CASES[name]
    rng = np.random.default_rng(len(name))
    mn, mx, body = _clumps(sizes, rng, bodies)
    if grounds:
        g = np.zeros((grounds, 4), np.float32)
        g[:, :3] = (-1.0, -2.0, -1.0)
        top = g.copy()
        top[:, :3] = (20.0 * len(sizes), 2.0, 1.0)
        mn, mx = np.concatenate([mn, g]), np.concatenate([mx, top])
        body = np.arange(len(mn), dtype=np.int32)
    n = len(mn)
    order = rng.permutation(n)
    mn, mx = mn[order], mx[order]
    grp = rng.integers(0, groups, n).astype(np.int32) if groups else None
    ref = []
    for g in range(max(groups, 1)):
        idx = np.arange(n) if not groups else np.flatnonzero(grp == g)
        ref.append(idx[bpio.oracle_pairs(port.lib, mn[idx], mx[idx], body[idx])])
    ref = np.sort(np.concatenate(ref), axis=1)
    exp = _ordered(ref, _positions(mn, mx, grp))
    assert len(exp) > 100
    cnt, got = _search(ctx, mn, mx, body, grp, len(exp) + 5)
    assert cnt == len(exp)
    assert np.array_equal(got[:cnt], exp)
    cnt2, got2 = _search(ctx, mn, mx, body, grp, cnt // 2)
    assert cnt2 == cnt and np.array_equal(got2[:cnt // 2], exp[:cnt // 2])
