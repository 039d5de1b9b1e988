"""The sphere scan's cheap condition (scene.cuh RayScan) never rejects a sphere that the exact
binary32 test (sphere_intersect) hits: random, grazing, tangent, inside, behind and far rays,
restated in numpy float32 (FMAs through float64, which rounds them once more at most)."""
import numpy as np
import pytest

F = np.float32
PAD = F(4.0e-6)


def _exact(o, d, c, rad):
    oc = o - c
    b = (oc[:, 0] * d[:, 0] + oc[:, 1] * d[:, 1]) + oc[:, 2] * d[:, 2]
    perp = oc - b[:, None] * d
    disc = rad * rad - ((perp[:, 0] * perp[:, 0] + perp[:, 1] * perp[:, 1]) + perp[:, 2] * perp[:, 2])
    cc = ((oc[:, 0] * oc[:, 0] + oc[:, 1] * oc[:, 1]) + oc[:, 2] * oc[:, 2]) - rad * rad
    with np.errstate(all="ignore"):
        sq = np.sqrt(np.maximum(disc, F(0)))
        q = np.where(b >= 0, -b - sq, -b + sq)
        tb = cc / q
        t = np.where(cc < 0, np.maximum(q, tb), np.minimum(q, tb))
    return (disc >= 0) & (q != 0) & (t > 0)


def _fma(a, b, c):
    return (a.astype(np.float64) * np.asarray(b, np.float64) + np.asarray(c, np.float64)).astype(F)


def _candidate(o, d, c, rad):
    w = rad * rad * (F(1) + PAD)
    dd = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
    k = F(2) - dd
    x, y, z = (o - c).T
    b = _fma(z, d[:, 2], _fma(y, d[:, 1], x * d[:, 0]))
    oc2 = _fma(z, z, _fma(y, y, x * x))
    bb = b * b
    miss = _fma(-bb, k, oc2 * (F(1) - PAD)) > w
    behind = (b > 0) & (bb > F(1.01) * w)
    return ~(miss | behind) | (np.abs(dd - F(1)) >= F(1e-3))


@pytest.mark.parametrize("scale", [1e-2, 1.0, 30.0, 900.0])
@pytest.mark.parametrize("kind", ["random", "grazing", "surface", "inside", "axis", "stretched"])
def test_no_exact_hit_is_rejected(scale, kind):
    rng = np.random.RandomState(int(scale * 100) + 7 * len(kind))
    n = 400000
    c = rng.uniform(-1, 1, (n, 3)) * scale
    rad = 10.0 ** rng.uniform(-4, 0.3, n) * scale
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    dist = 10.0 ** rng.uniform(-3, 1, n) * scale
    if kind == "random":
        o = c + u * (rad + dist)[:, None]
        d = (c + rng.normal(size=(n, 3)) * rad[:, None]) - o
    elif kind in ("grazing", "stretched"):
        side = np.cross(u, d)
        side /= np.linalg.norm(side, axis=1, keepdims=True)
        o = c + u * (rad + dist)[:, None]
        d = c + side * (rad * (1.0 + rng.normal(size=n) * 1e-6))[:, None] - o
    elif kind == "surface":   # origins on the sphere, as spawned rays
        o = c + u * (rad * (1.0 + rng.normal(size=n) * 1e-6))[:, None]
    elif kind == "inside":
        o = c + u * (rad * rng.uniform(0, 1, n))[:, None]
    else:
        o = c + np.eye(3)[rng.randint(3, size=n)] * (rad + dist)[:, None]
        d = c - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    if kind == "stretched":   # callers' rays that are not quite, or not at all, unit
        d *= (1.0 + rng.choice([1e-5, 5e-4, -9e-4, 2e-3, 0.5], n))[:, None]
    o, d, c, rad = (v.astype(F) for v in (o, d, c, rad))
    hit, cand = _exact(o, d, c, rad), _candidate(o, d, c, rad)
    assert hit.sum() > n // 20
    assert not (hit & ~cand).any()
