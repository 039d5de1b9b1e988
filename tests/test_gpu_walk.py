"""The one-kernel walk (k_walk) against the wavefront kernels, and the region scans' forms.

A counting render (PROFILE_WORK) runs the wavefront kernels whatever the scene, so the same
frame through both gives the same film bit for bit and the same query counts: one path, a
lane short of and past a warp, ragged images, waves that end inside a sample pass, every
program form.  The sphere scan works in chunks of 32: scenes around the chunk's edges give
the hits of the region BVH (the exact per-sphere test).
"""
import numpy as np
import pytest

from pathtracerglsl_b200 import abi, scenes
from pathtracerglsl_b200.compiler import Compiler

pytestmark = pytest.mark.gpu

SCENES = {
    "cornell": lambda: scenes.cornell(),
    "cornell-nee": lambda: scenes.cornell(direct="nee"),
    "cornell-none": lambda: scenes.cornell(direct="none", max_depth=4),
    "rough": lambda: scenes.cornell_rough(),
    "furnace": lambda: scenes.furnace(),
    "medium": lambda: scenes.adjoint_box_scene(),
    "fog-expression": lambda: scenes.het_fog(kind="blobs", max_depth=5),
    "absorbing": lambda: scenes.het_fog(kind="absorb", max_depth=5),
    "spectral-media": lambda: scenes.media_scene(max_depth=12)[:2],
    "rgb-media": lambda: scenes.media_scene(max_depth=12, spectral=False)[:2],
}


def _both(engine, sc, st, w, h, spp, special=False):
    r, pk = Compiler().compile(sc, st)
    engine.register_scene(pk)
    engine.load_renderer(r)
    engine.select_renderer(r.id)
    engine.pin_reset_salt(11)
    if special:
        engine.specialize()
    out = []
    for counting in (False, True):
        engine.reset()
        if counting:
            engine.profile_render(w, h, spp, abi.PROFILE_WORK)
        else:
            engine.render_frame(w, h, spp)
        c = engine.counters()
        out.append((engine.read_export("radiance").copy(), engine.read_export("variance").copy(),
                    (c["paths"], c["closest_queries"], c["shadow_queries"], c["error_flags"])))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]
    assert out[0][2][0] == w * h * spp


@pytest.mark.parametrize("size", [(1, 1, 1), (31, 1, 1), (33, 5, 3), (64, 20, 2)], ids=str)
@pytest.mark.parametrize("scene", sorted(SCENES))
def test_walk_equals_wavefront(engine, scene, size):
    _both(engine, *SCENES[scene](), *size)


@pytest.mark.parametrize("scene", ["cornell", "medium", "spectral-media"])
def test_specialised_walk_equals_wavefront(engine, scene):
    _both(engine, *SCENES[scene](), 33, 17, 2, special=True)


def test_walk_waves_end_inside_a_sample_pass(engine, monkeypatch):
    monkeypatch.setenv("PTR_CAPACITY", "1100")
    _both(engine, *scenes.cornell(), 40, 31, 3)     # more pixels than a wave holds
    _both(engine, *scenes.cornell(), 20, 19, 5)     # two sample passes per wave, then one


def test_walk_accumulates_frames(engine):
    """Frames that accumulate equal one frame of the summed samples; a frame that does not
    starts its film from zero."""
    r, pk = Compiler().compile(*scenes.cornell())
    engine.register_scene(pk)
    engine.load_renderer(r)
    engine.select_renderer(r.id)
    engine.pin_reset_salt(4)
    engine.reset()
    for spp in (1, 2, 1):
        engine.render_frame(45, 23, spp)
    parts = engine.read_export("radiance").copy(), engine.read_export("variance").copy()
    engine.reset()
    engine.render_frame(45, 23, 4)
    np.testing.assert_array_equal(engine.read_export("radiance"), parts[0])
    np.testing.assert_array_equal(engine.read_export("variance"), parts[1])


@pytest.mark.parametrize("n", [1, 31, 32, 33, 65, 130])
def test_sphere_scan_equals_region_bvh(engine, monkeypatch, n):
    rng = np.random.RandomState(n)
    sc, st = scenes.cornell(max_depth=4)
    objects = list(sc["objects"][:5])
    for _ in range(n):   # overlapping spheres too: exact ties and nested insides
        c = rng.uniform([-0.9, 0.1, -0.9], [0.9, 1.8, 0.9])
        objects.append({"type": "sphere", "parameters": {"center": [float(x) for x in c], "radius": float(rng.uniform(0.02, 0.3))},
                        "material": ("matte", "glass")[int(rng.randint(2))]})
    r, pk = Compiler().compile(dict(sc, objects=objects), st)
    out = []
    for minimum in ("1000000", "2"):
        monkeypatch.setenv("PTR_REGION_BVH_MIN", minimum)
        engine.register_scene(pk)
        engine.load_renderer(r)
        engine.select_renderer(r.id)
        engine.pin_reset_salt(6)
        engine.reset()
        out.append(engine.render_samples(37, 29, 2))
    np.testing.assert_array_equal(out[1], out[0])
