"""The flat two-level walks over the sizes where they can go wrong: one placement, a TLAS of one
leaf, several levels, prototypes of one and of 20 triangles, scaled and overlapping
placements (ties, instances inside one another).  Hits equal the oracle's ordered scan, for
both BLAS forms and both TLAS forms, and so do the frames' samples between the forms."""
import numpy as np
import pytest

from pathtracerglsl_b200 import abi, scenes
from pathtracerglsl_b200.compiler import Compiler
from test_gpu_mesh import _rays, _trace

pytestmark = pytest.mark.gpu


def _scene(tris, n, accel, inst_accel, seed=0):
    rng = np.random.RandomState(seed + 31 * n)
    if tris == 1:
        v, f = np.array([[0.0, 0.0, 0.0], [1.0, 0.1, 0.0], [0.2, 0.9, 0.3]]), np.array([[0, 1, 2]])
    else:
        v, f = scenes.icosphere(0 if tris == 20 else 2)
    place = []
    for k in range(n):
        axis = rng.normal(size=3)
        place.append({"position": [float(x) for x in rng.uniform(-1.5, 1.5, 3)], "scale": float(10.0 ** rng.uniform(-1.5, 0.2)),
                      "rotation": {"axis": list(axis / np.linalg.norm(axis)), "angle": float(rng.uniform(0, 6.28))}})
    if n > 2:
        place[n // 2] = dict(place[0])   # the same pose twice: every hit on it is a tie
    sc = {"id": "flat", "objects": [
        {"type": "plane", "parameters": {"normal": [0, 1, 0], "offset": 1.0}, "material": "m"},
        {"kind": "instanced", "prototype": {"kind": "mesh", "positions": v.astype(np.float32).reshape(-1),
                                            "indices": f.astype(np.uint32).reshape(-1), "material": "m"},
         "placements": place}],
        "materials": {"m": {"model": "lambert"}}, "lights": [{"kind": "point", "position": [2.0, 4.0, 3.0], "emission": 20.0}]}
    st = {"id": "s", "measurement": {"camera": {"position": [0, 1, 5], "target": [0, 0, 0]}, "maxBounces": 3},
          "estimator": {"directLighting": "nee", "russianRoulette": None, "meshTraversal": accel, "instanceAccel": inst_accel}}
    return Compiler().compile(sc, st)


@pytest.mark.parametrize("tris,n", [(1, 1), (1, 5), (20, 1), (20, 2), (20, 3), (20, 33), (320, 200)])
def test_flat_walks(engine, oracle_lib, tris, n):
    rays = _rays(6000, tris + n, spread=1.5, dist=6.0)
    images, hits = [], None
    for accel, code in (("bvh", abi.ACCEL_BVH), ("cwbvh", abi.ACCEL_CWBVH)):
        for inst_accel in ("tlas", "cwbvh"):
            r, pk = _scene(tris, n, accel, inst_accel)
            engine.register_scene(pk)
            engine.load_renderer(r)
            engine.select_renderer(r.id)
            got = _trace(engine, code, rays)
            if hits is None:
                hits = oracle_lib.trace_closest(pk, r, rays)
                assert (hits[2] >= 0).any()
            for a, b in zip(got[:1] + got[2:], hits[:1] + hits[2:]):
                np.testing.assert_array_equal(a, b)
            inst = hits[2] >= 0
            np.testing.assert_array_equal(got[1][inst], hits[1][inst])
            engine.pin_reset_salt(2)
            engine.reset()
            images.append(engine.render_samples(33, 21, 2))
            assert engine.counters()["error_flags"] == 0
    for im in images[1:]:
        np.testing.assert_array_equal(im, images[0])
