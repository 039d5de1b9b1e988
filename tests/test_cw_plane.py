"""The wide node test's folded plane distances (bvh.cuh cw_node) lie on the outer side of the
exact ones, restated in numpy: byte b as 1 + b 2^-15, one FMA with the offset folded in,
widened by 2^-7 of a cell, against p + b 2^e in float64, for boxes from 1e-6 to 1e3 wide seen
from far, near and inside."""
import numpy as np
import pytest

F = np.float32


def _fma(a, b, c):
    return (np.asarray(a, np.float64) * np.asarray(b, np.float64) + np.asarray(c, np.float64)).astype(F)


@pytest.mark.parametrize("exponent", [-28, -16, -8, 0, 2])
@pytest.mark.parametrize("origin", ["far", "near", "inside"])
@pytest.mark.parametrize("slant", [1.0, 1e-3, 1e-12])
def test_planes_are_conservative(exponent, origin, slant):
    rng = np.random.RandomState(exponent + 40)
    n = 200000
    cell = F(2.0 ** exponent)
    p = (rng.uniform(-1, 1, n) * 255 * cell * 4).astype(F)
    b = rng.randint(0, 256, n)
    reach = {"far": 1e4, "near": 3.0, "inside": 0.5}[origin]
    ro = (p + (0.5 + rng.uniform(-1, 1, n) * reach) * 255 * cell).astype(F)
    d = (rng.choice([-1.0, 1.0], n) * slant * 10.0 ** rng.uniform(-1, 0, n)).astype(F)
    inv = F(1) / d
    dq = cell * inv
    sc = dq * F(32768)
    c = (p - ro) * inv - sc
    pad = np.abs(dq) * F(0.0078125)
    v = (F(1) + b.astype(F) * F(2.0 ** -15)).astype(F)
    near, far = _fma(v, sc, c - pad), _fma(v, sc, c + pad)
    # the slab distance of the quantized plane, with the rounded (p - ro) and 1 / d it is given
    exact = (p - ro).astype(F).astype(np.float64) * inv.astype(np.float64) + b * (float(cell) * inv.astype(np.float64))
    # an FMA slab test rounds its offset and its result once each: what both forms may differ by
    slack = 2.0 ** -23 * (np.abs((p - ro).astype(np.float64) * inv) + np.abs(exact))
    assert (near.astype(np.float64) <= exact + slack).all()
    assert (far.astype(np.float64) >= exact - slack).all()
    assert (far - near <= 4.0 * pad + 4.0 * slack.astype(F)).all()   # and not needlessly wide
