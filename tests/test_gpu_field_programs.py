"""Typed coefficient-field programs on the GPU: every operation with scalar and vector operands,
constants first, last and between, folded, swapped and pushed, rendered as the scattering
field of the room's fog against the oracle, which runs the untyped program.  Both sides draw
the same numbers; the fields' transcendentals come from two libms, so a rare lottery may fall
differently (98 % of samples, as for the heterogeneous workloads).  A field may leave its
domain somewhere along a ray (a logarithm below zero): NaN then meets NaN."""
import numpy as np
import pytest

from pathtracerglsl_b200 import scenes
from pathtracerglsl_b200.compiler import Compiler
from test_gpu_parity import CASE_CAMERAS
from test_het_media import EXPRS

pytestmark = pytest.mark.gpu

SOURCES = [src.replace("u_a_gain", "2.5").replace("u_b", "0.75") for src, _ in EXPRS] + [
    "2.0 - p.x", "1.0 / (0.5 + abs(p.y))", "pow(2.0, p.x)", "pow(abs(p), vec3(1.5, 2.0, 0.5))", "mix(0.2, p.y, 0.5)",
    "mix(p.x, 0.2, p.z)", "clamp(0.3, p.x, 2.0)", "smoothstep(0.0, 2.0, p.y)", "smoothstep(p.x, 2.0, p)",
    "vec3(0.5, p.y, 0.2) * 0.7", "mod(3.0, 0.5 + abs(p.x))", "mod(p, 0.4) + 0.1", "step(0.5, p.y) + 0.1", "step(p.y, 0.5) + 0.1",
    "dot(vec3(0.2, 0.3, 0.4), p) + 1.0", "dot(p, p) * 0.5",
    "max(0.2, p.y * vec3(0.5, 0.6, 0.7))", "min(p, 0.5) - 1.0", "(1.0 + 2.0) * 0.25 - -0.1", "length(p) * 0.3 + floor(p.y * 3.0) * 0.1",
    "0.7", "vec3(0.3, 0.6, 0.9)", "(p.x + (2.0 - (p.y * (0.5 + p.z * 0.25)))) / (1.0 + p.y * p.y)",
]


@pytest.mark.parametrize("src", SOURCES)
def test_field_expression_matches_oracle(engine, oracle_lib, src):
    sc, st = scenes.het_fog(max_depth=4)
    fog = dict(sc["materials"]["fog"]["medium"], majorant=2.0,
               sigma_s={"kind": "glsl", "source": f"clamp(abs({src}), 0.02, 1.8)"})
    sc = dict(sc, materials=dict(sc["materials"], fog=dict(sc["materials"]["fog"], medium=fog)))
    r, pk = Compiler().compile(sc, st)
    engine.register_scene(pk)
    engine.load_renderer(r)
    engine.select_renderer(r.id)
    engine.params = dict(CASE_CAMERAS["cornell"])
    engine.pin_reset_salt(11)
    got = engine.render_samples(20, 20, 4)
    want = oracle_lib.render(pk, r, 20, 20, 4, salt=11, params=engine.params, keep_samples=True)["samples"]
    with np.errstate(invalid="ignore"):
        close = (np.abs(got - want) <= 1e-4 * np.maximum(1.0, np.abs(want))) | (np.isnan(got) & np.isnan(want))
    assert close.all(axis=-1).mean() >= 0.98
