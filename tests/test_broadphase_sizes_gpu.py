"""The LBVH pair search at the sizes where its kernels change shape (one and
two colliders, the edges of a warp, of a block and of a sort tile, more blocks
than add up their own offsets, more tiles than add up their own counts), with
coincident colliders (equal Morton keys), more partners than a collider keeps
between the kernels, groups, and a capacity smaller than the number of pairs.
The pairs and their order are exact: by sorted position of the first collider,
then of the second, positions by Morton key of the box centres (stable)."""
import numpy as np
import pytest

import bpio
from reactphysics3d_b200 import broadphase as BP
from reactphysics3d_b200 import engine

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cuda_lib):
    c = engine.Context(0)
    yield c
    c.close()


def _spread(v):
    r = np.zeros_like(v)
    for b in range(10):
        r |= ((v >> b) & 1) << (3 * b)
    return r


def _positions(mn, mx, group):
    """Sorted position of each collider."""
    f = np.float32
    c = f(0.5) * (mn[:, :3] + mx[:, :3])
    lo, hi = c.min(0), c.max(0)
    ext = hi - lo
    inv = np.where(ext > 0, f(1023.0) / np.where(ext > 0, ext, f(1.0)), f(0.0)).astype(f)
    q = np.clip((c - lo) * inv, f(0.0), f(1023.0)).astype(np.uint64)
    key = (_spread(q[:, 0]) << np.uint64(2)) | (_spread(q[:, 1]) << np.uint64(1)) | _spread(q[:, 2])
    if group is not None:
        key |= group.astype(np.uint64) << np.uint64(30)
    pos = np.empty(len(key), np.int64)
    pos[np.argsort(key, kind="stable")] = np.arange(len(key))
    return pos


def _search(ctx, mn, mx, body, group, capacity, axis=-1):
    import torch
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (mn, mx, body)]
    g = None if group is None else torch.from_numpy(group).cuda()
    bp = BP.make(len(mn), 0, 0 if group is None else int(group.max()) + 1, body=t[2], group=g, fat_min=t[0], fat_max=t[1])
    cnt, pairs = ctx.broadphase_pairs(bp, capacity, axis=axis, device=True)
    ctx.synchronize()
    assert ctx.device_errors(clear=True) & 24 == 0
    return int(cnt.item()), pairs.cpu().numpy()


def _ordered(pairs, pos):
    p = np.sort(pos[pairs], axis=1)
    return pairs[np.lexsort((p[:, 1], p[:, 0]))]


@pytest.mark.parametrize("n,groups", [(2, 0), (3, 0), (31, 0), (33, 0), (127, 0), (129, 3), (2047, 0), (2049, 5), (6000, 40)])
@pytest.mark.parametrize("kind", ["spread", "dense", "coincident"])
def test_pairs_and_their_order(ctx, port, n, groups, kind):
    rng = np.random.default_rng(n)
    mn, mx, body, grp = bpio.random_aabbs(n, rng, world={"spread": 1.2 * n ** (1 / 3), "dense": 0.4 * n ** (1 / 3) + 0.5,
                                                         "coincident": 4.0}[kind], groups=groups, nbodies=max(2, int(0.9 * n)))
    if kind == "coincident":                     # boxes in a few places: equal keys, long partner lists
        k = rng.integers(0, max(1, n // 12), n)
        mn, mx = mn[k].copy(), mx[k].copy()
    ref = []
    for g in range(max(groups, 1)):
        idx = np.arange(n) if not groups else np.flatnonzero(grp == g)
        if len(idx) > 1:
            ref.append(idx[bpio.oracle_pairs(port.lib, mn[idx], mx[idx], body[idx])])
    ref = np.sort(np.concatenate(ref), axis=1) if ref else np.zeros((0, 2), np.int64)
    exp = _ordered(ref, _positions(mn, mx, grp if groups > 1 else None))
    cnt, got = _search(ctx, mn, mx, body, grp if groups > 1 else None, len(exp) + 5)
    assert cnt == len(exp)
    assert np.array_equal(got[:cnt], exp)
    if cnt > 3:                                  # a small array: the count is whole, the array's part too
        cnt2, got2 = _search(ctx, mn, mx, body, grp if groups > 1 else None, cnt // 2)
        assert cnt2 == cnt and np.array_equal(got2[:cnt // 2], exp[:cnt // 2])


@pytest.mark.parametrize("n", [128 * 2048 + 1, 2048 * 512 + 1])
def test_many_colliders(ctx, n):
    """Above the sizes at which blocks and tiles add up what comes before
    them; the sweep along x finds the same pairs."""
    rng = np.random.default_rng(n)
    mn, mx, body, _ = bpio.random_aabbs(n, rng, world=n ** (1 / 3), size=(0.1, 0.5))
    cnt, got = _search(ctx, mn, mx, body, None, 2 * n)
    cnt2, ref = _search(ctx, mn, mx, body, None, 2 * n, axis=0)
    assert n // 32 < cnt == cnt2 <= 2 * n
    assert np.array_equal(got[:cnt], _ordered(ref[:cnt], _positions(mn, mx, None)))
