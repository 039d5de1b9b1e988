"""A null interface ('none') in a scene without media is a smooth dielectric of IOR 1: rays
that meet it from inside glass refract out of the glass's IOR.

CPU: every model that reads the IORs of the surface's two sides says so (kUsesIor: the walk
classifies the incident side for those only), and the oracle renders the interface as the
dielectric.  GPU: a bubble of 'none' inside a glass sphere gives the samples of a bubble of IOR 1
and those of the oracle, on the library's and the per-scene kernels, the one-kernel walk, the
wavefront, a batch and the adjoint.
"""
import glob
import os
import re

import numpy as np
import pytest

from pathtracerglsl_b200 import scenes
from pathtracerglsl_b200.compiler import Compiler
from test_gpu_parity import compare

MAT_DIR = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pathtracerglsl_b200", "csrc", "device", "materials")
MODELS = {"none": {"model": "none"}, "unit": {"model": "dielectric", "ior": 1.0}}


def bubble(kind, mesh=False, direct="mis", spectral=False):
    """The Cornell box with a glass sphere around a bubble of the model under test (mesh: with an
    emissive panel of triangles, which the wavefront renders)."""
    sc, st = scenes.cornell_mesh_light(direct=direct) if mesh else scenes.cornell(direct=direct)
    objects = [o for o in sc["objects"] if o.get("type") != "sphere"] + [
        {"type": "sphere", "parameters": {"center": [0.3, 0.55, 0.3], "radius": 0.5}, "material": "glass"},
        {"type": "sphere", "parameters": {"center": [0.3, 0.55, 0.3], "radius": 0.42}, "material": "bubble"}]
    if spectral:
        st = dict(st, measurement=dict(st["measurement"], color="spectral"))
    return dict(sc, objects=objects, materials=dict(sc["materials"], bubble=MODELS[kind])), st


def test_models_that_read_the_iors_say_so():
    checked = 0
    for path in sorted(glob.glob(os.path.join(MAT_DIR, "*.cuh"))):
        for name, body in re.findall(r"struct (\w+) : MaterialModel \{(.*?)\n\};", open(path).read(), re.S):
            reads = re.search(r"\bs\.n_(from|to)\b", body) is not None
            declares = "static constexpr bool kUsesIor = true;" in body
            assert reads == declares, f"{os.path.basename(path)}: {name}"
            checked += reads
    assert checked == 3   # the smooth and the rough dielectric, the null interface


def test_oracle_renders_the_interface_as_a_dielectric(oracle_lib):
    out = []
    for kind in sorted(MODELS):
        r, pk = Compiler().compile(*bubble(kind))
        out.append(oracle_lib.render(pk, r, 24, 24, 4, salt=11, keep_samples=True)["samples"])
    np.testing.assert_array_equal(out[0], out[1])


def _samples(engine, kind, special, **form):
    r, pk = Compiler().compile(*bubble(kind, **form))
    engine.register_scene(pk)
    engine.load_renderer(r)
    engine.select_renderer(r.id)
    engine.pin_reset_salt(11)
    if special:
        engine.specialize()
    return engine.render_samples(48, 40, 4)


@pytest.mark.gpu
@pytest.mark.parametrize("special", [False, True], ids=["library", "per-scene"])
@pytest.mark.parametrize("form", [{}, {"direct": "nee"}, {"direct": "none"}, {"mesh": True}, {"spectral": True}], ids=str)
def test_bubble_equals_a_dielectric_of_ior_1(engine, form, special):
    np.testing.assert_array_equal(_samples(engine, "none", special, **form), _samples(engine, "unit", special, **form))


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", [False, True])
def test_bubble_matches_oracle(engine, oracle_lib, mesh):
    sc, st = bubble("none", mesh=mesh)
    compare(engine, oracle_lib, sc, st, 48, 48, 8, {})


@pytest.mark.gpu
def test_bubble_in_a_batch_and_the_adjoint(engine):
    films, grads = [], []
    for kind in sorted(MODELS):
        items = [Compiler().compile(*bubble(kind)), Compiler().compile(*scenes.cornell())]
        b = engine.batch(items)
        try:
            b.render([(33, 29, 4, 0, 5), (20, 20, 2, 0, 6)])
            films.append(b.read_export(0).copy())
        finally:
            b.close()
        r, pk = items[0]
        engine.register_scene(pk)
        engine.load_renderer(r)
        engine.select_renderer(r.id)
        names = list(pk.material_names)
        g = engine.backward(np.ones((29, 33, 3), np.float32), 33, 29, 4, salt=5)
        # the gradients of the walls and the glass; the bubble's own slots differ by model
        grads.append(g[[i for i, n in enumerate(names) if n != "bubble"]])
    np.testing.assert_array_equal(films[0], films[1])
    # float64 sums in the order the blocks finish
    np.testing.assert_allclose(grads[0], grads[1], rtol=1e-9, atol=1e-12 * np.abs(grads[1]).max())
    assert np.abs(grads[0]).max() > 0
