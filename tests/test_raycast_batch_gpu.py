"""World raycasts against themselves where the batch kernel changes shape: the
rays of a batch cast together, in small batches (one ray a warp) and one by
one give the same hits; the closest hit of a ray is the nearest of all its
hits and ANY returns the first of them (the nearest: for rays that hit no
convex mesh, whose hits the reference places on planes through the unscaled
vertices, so that a scaled mesh's hit can lie outside the bounds that a clipped
ray is tested against).  Terrain rays include near-vertical
ones along grid lines and corners, rays starting far away, ending inside the
field, level with it, of zero length and with a small maxFraction; every
height-field hit is also checked against a float64 test of all triangles.

Tolerance of that check: the reference's hit fraction comes from float
products of coordinates up to D from the ray's origin, off by about
10 * 2^-24 * D^2 cells; rays within twice that of missing or of a second hit
are left out."""
import numpy as np
import pytest

from reactphysics3d_b200 import _abi as A
from reactphysics3d_b200 import engine, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cuda_lib):
    c = engine.Context(0)
    yield c
    c.close()


def _field_rays(n, cols, rng):
    half = 0.5 * (cols - 1)
    r = A.rays(n)
    p1, p2 = rng.uniform(-half, half, (n, 3)), rng.uniform(-half, half, (n, 3))
    p1[:, 1], p2[:, 1] = rng.uniform(3.0, 30.0, n), rng.uniform(-30.0, -3.0, n)
    k = np.arange(n) % 10
    p2[k == 0] = p1[k == 0] + (0.0, -40.0, 0.0)                            # vertical
    g = np.round(p1[:, [0, 2]] - half) + half                              # grid lines and corners
    p1[k == 1, 0] = p2[k == 1, 0] = g[k == 1, 0]
    on = k == 2
    p1[on, 0], p1[on, 2] = g[on, 0], g[on, 1]
    p2[on] = p1[on] + rng.uniform(-1e-3, 1e-3, (int(on.sum()), 3)) + (0.0, -40.0, 0.0)
    far = k == 3
    d = p2[far] - p1[far]
    p1[far] -= 20.0 * d                                                    # far origin
    p2[k == 4, 1] = p1[k == 4, 1] = rng.uniform(-2.0, 2.0, int((k == 4).sum()))   # level
    p2[k == 5, 1] = rng.uniform(-2.0, 2.0, int((k == 5).sum()))            # ends at the surface
    p2[k == 6] = p1[k == 6] + rng.uniform(-2.0, 2.0, (int((k == 6).sum()), 3)) + (0.0, -40.0, 0.0)   # steep
    p2[(k == 7) & (np.arange(n) % 100 == 7)] = p1[(k == 7) & (np.arange(n) % 100 == 7)]  # zero length
    r["point1"], r["point2"] = p1.astype(np.float32), p2.astype(np.float32)
    r["max_fraction"][k == 8] = rng.uniform(0.05, 1.0, int((k == 8).sum())).astype(np.float32)
    r["max_fraction"][k == 9] = 3.0
    return r


def _same(a, b):
    assert np.array_equal(a[1], b[1])
    hit = a[1] > 0
    assert np.array_equal(a[0][hit].view(np.uint8), b[0][hit].view(np.uint8))


def _check_modes_and_batches(w, rays, sc):
    n = len(rays)
    closest = w.raycast(rays, A.RAYCAST_CLOSEST)
    for size in (1, 31, 33, 4736, 4737):
        if size <= n:
            _same((closest[0][:size], closest[1][:size]), w.raycast(rays[:size], A.RAYCAST_CLOSEST))
    for k in range(0, n, max(1, n // 40)):
        _same((closest[0][k:k + 1], closest[1][k:k + 1]), w.raycast(rays[k:k + 1], A.RAYCAST_CLOSEST))
    every, counts = w.raycast(rays, A.RAYCAST_ALL, 16)
    first, any_counts = w.raycast(rays, A.RAYCAST_ANY)
    # ALL never clips the ray below 1, so it is compared where maxFraction is 1
    for i in np.flatnonzero((rays["max_fraction"] == 1.0) & (counts <= 16)):
        assert (any_counts[i] > 0) == (counts[i] > 0) == (closest[1][i] > 0), i
        if counts[i]:
            f = every[i, :counts[i]]["hit_fraction"]
            if not np.any(sc.shapes["kind"][every[i, :counts[i]]["collider"]] == A.SHAPE_CONVEX_MESH):
                assert closest[0][i, 0]["hit_fraction"] == f.min(), i
            assert first[i, 0]["collider"] == every[i, 0]["collider"] and first[i, 0]["hit_fraction"] == f[0], i


def test_terrain_batches(ctx):
    sc = scenes.heightfield_world(n_bodies=1500, cols=60, rows=60, seed=12)
    w = engine.World(ctx, sc)
    w.update(1.0 / 60.0, 30)
    _check_modes_and_batches(w, np.concatenate([_field_rays(3000, 60, np.random.default_rng(1)),
                                                scenes.terrain_rays(sc, 3000, seed=2)]), sc)
    w.close()


def test_hull_batches(ctx):
    sc = scenes.hull_world(6, 6, 6, seed=13)
    w = engine.World(ctx, sc)
    w.update(1.0 / 60.0, 40)
    p = sc.bodies["position"][1:]
    _check_modes_and_batches(w, scenes.world_rays(6000, p.min(0) - 1.0, p.max(0) + 1.0, seed=3), sc)
    w.close()


@pytest.mark.parametrize("scale", [(1.0, 1.0, 1.0), (0.5, 2.0, 1.5)])
def test_height_field_hits_against_every_triangle(ctx, scale):
    cols = rows = 40
    heights = scenes.sine_heights(cols, rows, seed=77, k_range=(0.2, 1.2))
    shapes = np.zeros(1, A.SHAPE_DTYPE)
    shapes[0]["kind"], shapes[0]["mesh"] = A.SHAPE_HEIGHTFIELD, 0
    bodies, colliders = A.body_descs(1), A.collider_descs(1)
    bodies[0]["type"] = A.BODY_STATIC
    sc = scenes.WorldScene(A.default_world_settings(), shapes, bodies, colliders, heightfields=[(heights, scale)])
    w = engine.World(ctx, sc)
    w.update(1.0 / 60.0)
    rays = _field_rays(4000, cols, np.random.default_rng(5))
    s = np.array(scale)
    for f in ("point1", "point2"):
        rays[f] = (rays[f] * s).astype(np.float32)
    hits, counts = w.raycast(rays)
    w.close()
    h = heights.astype(np.float64)
    origin = -0.5 * (h.max() + h.min())
    x, z = np.meshgrid(np.arange(cols) - 0.5 * (cols - 1), np.arange(rows) - 0.5 * (rows - 1))
    v = np.stack([x, h + origin, z], -1)                                   # [row][column]
    q1, q2, q3, q4 = v[:-1, :-1], v[1:, :-1], v[:-1, 1:], v[1:, 1:]
    tri = np.concatenate([np.stack(t, -2).reshape(-1, 3, 3) for t in ((q1, q2, q3), (q3, q2, q4))])
    checked = 0
    for i in range(0, len(rays), 3):
        p1, p2 = rays[i]["point1"] / s, rays[i]["point2"] / s
        d = (p2 - p1).astype(np.float64)
        if not np.any(d):
            assert counts[i] == 0
            continue
        a, b, c = (tri[:, k] - p1 for k in range(3))
        m = np.linalg.norm(d)
        vol = np.stack([np.einsum("ij,ij->i", b, np.cross(d, c)), -np.einsum("ij,ij->i", a, np.cross(d, c)),
                        np.einsum("ij,ij->i", a, np.cross(d, b))]) / m
        low = vol.min(0)
        slack = 2.0 * 10.0 * 2.0 ** -24 * max(1.0, float((np.linalg.norm(tri - p1, axis=2) ** 2).max()))
        if np.any(np.abs(low) <= slack):
            continue                                                       # an edge, a corner or a plane: rounding decides
        ok = np.flatnonzero(low > slack)
        wsum = vol[:, ok].sum(0)
        lp = (vol[:, ok] / wsum).T[:, :, None] * tri[ok]
        t = (lp.sum(1) - p1) @ d / (d @ d)
        mf = float(rays[i]["max_fraction"])
        if np.any(np.abs(t) < 1e-4) or np.any(np.abs(t - mf) < 1e-4):
            continue
        t = t[(t >= 0.0) & (t <= mf)]
        assert (counts[i] > 0) == (len(t) > 0), (i, t)
        if len(t):
            assert abs(hits[i, 0]["hit_fraction"] - t.min()) < 1e-3, (i, t, hits[i, 0])
        checked += 1
    assert checked > 700
