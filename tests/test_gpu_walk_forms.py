"""The one-kernel walk against the wavefront kernels in the forms test_gpu_walk leaves out: waves
that fill 512-thread blocks on every SM, light trees and instanced spheres without a mesh,
first-hit pictures, per-scene kernels through heterogeneous media, batches and the adjoint.

A counting render runs the wavefront whatever the scene; for a batch and the adjoint a triangle
that no ray reaches (inside the matte sphere) does the same.  Films agree bit for bit, gradients up
to the order of their float64 sums."""
import numpy as np
import pytest

from pathtracerglsl_b200 import abi, scenes
from pathtracerglsl_b200.compiler import Compiler
from test_gpu_walk import _both

pytestmark = pytest.mark.gpu


def _lamps(**kw):
    sc, st = scenes.many_lights(n=32, **kw)
    return dict(sc, objects=[o for o in sc["objects"] if o.get("kind") != "mesh"]), st


def _aovs(sc, st):
    return sc, dict(st, measurement=dict(st["measurement"], aovs=["albedo", "normal"]))


FORMS = {
    "cornell": lambda: scenes.cornell(),
    "rough": lambda: scenes.cornell_rough(),
    "medium": lambda: scenes.adjoint_box_scene(),
    "rgb-media": lambda: scenes.media_scene(max_depth=12, spectral=False)[:2],
    "spectral-media": lambda: scenes.media_scene(max_depth=12)[:2],
    "ground-fog": lambda: scenes.het_fog(max_depth=5),
    "blobs-mis": lambda: scenes.het_fog(direct="mis", kind="blobs", max_depth=5),
    "absorbing": lambda: scenes.het_fog(kind="absorb", max_depth=5),
    "lamps": lambda: _lamps(),
    "lamps-nee": lambda: _lamps(direct="nee"),
    "lamps-power": lambda: _lamps(selection="power"),
    "lamps-fog": lambda: _lamps(fog=True),
}


@pytest.mark.parametrize("special", [False, True], ids=["library", "per-scene"])
@pytest.mark.parametrize("form", sorted(FORMS))
def test_full_blocks(engine, form, special):
    _both(engine, *FORMS[form](), 331, 251, 1, special=special)   # 83,081 paths


@pytest.mark.parametrize("special", [False, True], ids=["library", "per-scene"])
@pytest.mark.parametrize("form", ["lamps", "lamps-fog", "ground-fog", "blobs-mis", "absorbing"])
@pytest.mark.parametrize("size", [(1, 1, 1), (33, 17, 3)], ids=str)
def test_small_waves(engine, form, size, special):
    _both(engine, *FORMS[form](), *size, special=special)


@pytest.mark.parametrize("capacity", [None, "1100"])
@pytest.mark.parametrize("form", ["cornell", "medium", "lamps-fog", "ground-fog"])
def test_first_hit_pictures(engine, monkeypatch, form, capacity):
    if capacity:
        monkeypatch.setenv("PTR_CAPACITY", capacity)
    r, pk = Compiler().compile(*_aovs(*FORMS[form]()))
    engine.register_scene(pk)
    engine.load_renderer(r)
    engine.select_renderer(r.id)
    engine.pin_reset_salt(11)
    out = []
    for counting in (False, True):
        engine.reset()
        if counting:
            engine.profile_render(41, 37, 3, abi.PROFILE_WORK)
        else:
            engine.render_frame(41, 37, 3)
        out.append([engine.read_export(n).copy() for n in ("radiance", "variance", "albedo", "normal")])
    for a, b in zip(*out, strict=True):
        np.testing.assert_array_equal(a, b)
    assert all(p.any() for p in out[0])


def _hidden_triangle(sc):
    """The scene with a triangle inside its matte sphere, which no ray enters."""
    ball = next(o["parameters"] for o in sc["objects"] if o.get("material") == "matte" and o.get("type") == "sphere")
    c, r = np.array(ball["center"]), 0.3 * ball["radius"]
    tri = {"kind": "mesh", "material": "matte", "closed": False, "indices": [[0, 1, 2]],
           "positions": [list(map(float, c + r * np.array(d))) for d in ([1, 0, 0], [0, 1, 0], [0, 0, 1])]}
    return dict(sc, objects=list(sc["objects"]) + [tri])


@pytest.mark.parametrize("capacity", [None, "3000"])
def test_batches(engine, monkeypatch, capacity):
    if capacity:   # waves end inside jobs
        monkeypatch.setenv("PTR_CAPACITY", capacity)
    jobs = [scenes.cornell(), scenes.cornell_rough(), _lamps(selection="power"), scenes.adjoint_box_scene(),
            scenes.het_fog(direct="mis", max_depth=5), scenes.cornell(max_depth=3)]
    frames = [(64, 40, 4, 0, 3), (33, 31, 2, 0, 4), (17, 50, 3, 0, 5), (48, 20, 2, 0, 6), (30, 30, 2, 0, 7), (1, 1, 5, 0, 8)]
    films = []
    for hidden in (False, True):
        items = [Compiler().compile(_hidden_triangle(sc) if hidden and k == 0 else sc, st) for k, (sc, st) in enumerate(jobs)]
        b = engine.batch(items)
        try:
            b.render(frames)
            ran = b.profile(frames)
            assert (ran["closest"][1] > 0) == hidden   # the route
            films.append([b.read_export(j, n).copy() for j in range(len(b)) for n in ("radiance", "variance")])
        finally:
            b.close()
    for x, y in zip(*films, strict=True):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("special", [False, True], ids=["library", "per-scene"])
@pytest.mark.parametrize("capacity", [None, "3000"])
@pytest.mark.parametrize("form", ["cornell", "cornell-nee", "cornell-none", "medium"])
def test_adjoint(engine, monkeypatch, form, capacity, special):
    if capacity:
        monkeypatch.setenv("PTR_CAPACITY", capacity)
    direct = {"cornell-nee": "nee", "cornell-none": "none"}.get(form, "mis")
    sc, st = scenes.cornell(direct=direct)
    if form == "medium":   # a grey medium in a sphere of its own beside the matte one
        sc = dict(sc, objects=list(sc["objects"]) + [
            {"type": "sphere", "parameters": {"center": [0.1, 1.1, 0.1], "radius": 0.4}, "material": "fog"}],
            materials=dict(sc["materials"], fog={"model": "none", "medium": {"sigma_a": [0.2] * 3, "sigma_s": [1.5] * 3, "phase_g": 0.4}}))
    w, h, spp = 61, 43, 3
    dl = np.random.RandomState(2).uniform(-1.0, 1.0, (h, w, 3)).astype(np.float32)
    grads = []
    for hidden in (False, True):
        r, pk = Compiler().compile(_hidden_triangle(sc) if hidden else sc, st)
        engine.register_scene(pk)
        engine.load_renderer(r)
        engine.select_renderer(r.id)
        if special:
            engine.specialize()
        grads.append(engine.backward(dl, w, h, spp, salt=8))
    scale = np.abs(grads[0]).max()
    assert scale > 0
    np.testing.assert_allclose(grads[0], grads[1], rtol=1e-9, atol=1e-12 * scale)
