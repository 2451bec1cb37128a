"""The contact solver's island kernels at the sizes where an island changes
kernel or layout, bit for bit against the C restatement of the reference's
stage (which is pinned to the reference elsewhere): synthetic islands of
random manifolds (1-4 points, random body order, fixed bodies among them)
around the thread-per-island limit, the warp's stage (512 manifolds, 320
bodies), one level wider than the staged ring, one long chain, islands of
several CTA-sized schedules, and more such islands than CTAs."""
import ctypes as C

import numpy as np
import pytest

import dynio
import reflib
from reactphysics3d_b200 import dynamics as D
from reactphysics3d_b200 import engine

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cuda_lib):
    c = engine.Context(0)
    yield c
    c.close()


def _pairs(kind, nb, nm, rng):
    if kind == "random":      # any two movable bodies, or one and a fixed one (index nb)
        a = rng.integers(0, nb, nm)
        b = rng.integers(0, nb, nm)
        b = np.where((a == b) | (rng.random(nm) < 0.2), nb, b)
        return np.where(rng.random((nm, 1)) < 0.5, np.stack([a, b], 1), np.stack([b, a], 1))
    if kind == "chain":       # one manifold a level
        i = np.arange(nm) % (nb - 1)
        return np.stack([i, i + 1], 1)
    i = 2 * (np.arange(nm) % (nb // 2))   # "wide": disjoint pairs, one level a sweep
    return np.stack([i, i + 1], 1)


def _world(islands, seed):
    """One world whose islands are (kind, movable bodies, manifolds)."""
    rng = np.random.default_rng(seed)
    nmov = sum(nb for _, nb, _ in islands)
    n = nmov + 2                                    # two fixed bodies at the end
    nm = sum(m for _, _, m in islands)
    ids, starts, counts, base = [], [], [], 0
    for kind, nb, m in islands:
        p = _pairs(kind, nb, m, rng)
        fixed = nmov + rng.integers(0, 2, p.shape)
        ids.append(np.where(p == nb, fixed, p + base))
        starts.append(sum(counts))
        counts.append(m)
        base += nb
    ids = np.concatenate(ids)
    npts = rng.integers(1, 5, nm)
    pstart = np.concatenate([[0], np.cumsum(npts)[:-1]])
    npt = int(npts.sum())
    f4 = lambda *shape: np.concatenate([rng.normal(size=shape + (3,)), np.zeros(shape + (1,))], -1)
    unit = lambda v: v / np.linalg.norm(v, axis=-1, keepdims=True)
    pos, rot = f4(n), unit(rng.normal(size=(n, 4)))
    mass = np.zeros((n, 4))
    mass[:nmov, 0] = rng.uniform(0.5, 3.0, nmov)
    mass[:nmov, 1] = 1.0 / mass[:nmov, 0]
    inertia = np.zeros((n, 4))
    inertia[:nmov, :3] = rng.uniform(0.5, 8.0, (nmov, 3))
    vel, spin = 0.3 * f4(n), 0.3 * f4(n)
    vel[nmov:] = spin[nmov:] = 0.0
    spin[n - 1, 1] = 0.5                            # a fixed body that turns (kinematic)
    lock = np.ones((n, 4))
    lock[:, 3] = 0.0
    nd = np.concatenate([unit(rng.normal(size=(npt, 3))), rng.uniform(-0.005, 0.05, (npt, 1))], 1)
    fv = np.concatenate([unit(rng.normal(size=(nm, 3))), np.zeros((nm, 1))], 1)
    iiw = np.zeros((n, 3, 4))
    return D.DynWorld({
        "position": pos, "orientation": rot, "com_world": pos, "com_local": np.zeros((n, 4)), "linear_velocity": vel,
        "angular_velocity": spin, "force": f4(n), "torque": f4(n), "inv_inertia_local": inertia, "mass": mass,
        "linear_lock": lock, "angular_lock": lock, "gravity": np.ones(n), "inv_inertia_world": iiw.reshape(-1, 4),
        "body": np.arange(n), "local_position": np.zeros((n, 4)),
        "local_orientation": np.tile([0.0, 0.0, 0.0, 1.0], (n, 1)), "world_position": pos, "world_orientation": rot,
        "material": np.tile([0.3, 0.2, 0.0, 0.0], (n, 1)),
        "ids": np.concatenate([ids, ids], 1), "point_start": pstart, "nb_points": npts, "friction_vector1": fv,
        "friction_vector2": np.roll(fv, 1, 0), "friction_impulse": 0.02 * f4(nm), "normal_depth": nd,
        "local1": 0.5 * f4(npt), "local2": 0.5 * f4(npt), "penetration_impulse": rng.uniform(0.0, 0.05, npt),
        "is_resting": rng.integers(0, 2, npt), "manifold_start": np.array(starts), "manifold_count": np.array(counts),
    }, nmov, nmov)


CASES = {
    "around the thread-per-island limit": [("random", 6, m) for m in (1, 4, 7, 8, 9, 10, 12, 13)],
    "one chunk and two": [("wide", 16, 8), ("wide", 18, 9), ("chain", 12, 9)],
    "warp stage": [("random", 40, 64), ("random", 60, 65), ("random", 200, 256), ("wide", 300, 200)],
    "warp stage full": [("random", 302, 250), ("random", 310, 256)],
    "levels wider than the ring": [("wide", 600, 280), ("wide", 66, 300)],
    "long chain": [("chain", 270, 600)],
    "one CTA": [("random", 150, 257), ("random", 400, 700), ("random", 90, 513)],
    "streamed": [("random", 1500, 2600)],
    "more islands than CTAs": [("random", 60, 257 + i % 3) for i in range(149)] + [("random", 330, 400), ("random", 80, 520)],
}


@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("name", CASES)
def test_islands_match_the_restatement(ctx, port, name, split):
    w = _world(CASES[name], len(name))
    params = D.make_params(split=split)
    dev = D.DynWorld(w.a, w.nb_enabled, w.nc_enabled, device="cuda")
    ref = dynio.run_oracle(C.CDLL(reflib.PORT_LIB), params, w.copy())
    ctx.dynamics_step(params, dev)
    ctx.synchronize()
    assert ctx.device_errors(clear=True) & 4 == 0
    h = dev.host()
    for k in D.OUTPUTS:
        a, b = np.asarray(h[k]), np.asarray(ref[k])
        if k == "inv_inertia_world":
            a, b = a[:3 * w.nb_enabled], b[:3 * w.nb_enabled]
        if a.dtype == np.float32:
            assert np.all(np.isfinite(b)), k
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), k
