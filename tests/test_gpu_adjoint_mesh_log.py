"""The adjoint's walk log on instanced meshes: the forward walk's refilling traversal records its
closest hits and the replay reads them instead of walking the trees again.  Gradients equal
those of a run that logs nothing, or only the first iterations, or several waves; and with
no shadow queries the run that logs is faster, by the replay's traversal."""
import time

import numpy as np
import pytest

from pathtracerglsl_b200 import scenes
from pathtracerglsl_b200.compiler import Compiler

pytestmark = pytest.mark.gpu

FORMS = [(a, i) for a in ("bvh", "cwbvh") for i in ("bvh", "cwbvh")]


def _load(engine, accel, instance_accel, level, instances, depth, direct):
    sc, st, _ = scenes.mesh_scene(level=level, instances=instances, max_depth=depth, env_size=(128, 64), direct=direct, accel=accel)
    r, pk = Compiler().compile(sc, dict(st, estimator=dict(st["estimator"], instanceAccel=instance_accel)))
    engine.register_scene(pk)
    engine.load_renderer(r)
    engine.select_renderer(r.id)


@pytest.mark.parametrize("special", [False, True], ids=["library", "per-scene"])
@pytest.mark.parametrize("accel,instance_accel", FORMS)
def test_gradients_do_not_depend_on_the_log(engine, monkeypatch, accel, instance_accel, special):
    w, h, spp = 45, 31, 3
    _load(engine, accel, instance_accel, 3, 5, 5, "mis")
    if special:
        engine.specialize()
    dl = np.random.RandomState(3).uniform(-1.0, 1.0, (h, w, 3)).astype(np.float32)
    grads = []
    # the whole log, none, two iterations of the pool's 4185 paths, and two sample passes per wave
    for log, capacity in ((None, None), ("0", None), (str(2 * 64 * w * h * spp), None), (None, str(2 * w * h))):
        with monkeypatch.context() as m:
            if log:
                m.setenv("PTR_HIT_LOG_BYTES", log)
            if capacity:
                m.setenv("PTR_CAPACITY", capacity)
            grads.append(engine.backward(dl, w, h, spp, salt=8))
    scale = np.abs(grads[0]).max()
    assert scale > 0
    for g in grads[1:]:
        np.testing.assert_allclose(g, grads[0], rtol=1e-9, atol=1e-12 * scale)


@pytest.mark.parametrize("accel,instance_accel", FORMS)
def test_replay_reads_the_log(engine, monkeypatch, accel, instance_accel):
    w, h, spp = 512, 384, 4
    _load(engine, accel, instance_accel, 6, 16, 6, "none")
    dl = np.ones((h, w, 3), np.float32)

    def best():
        times = []
        for _ in range(8):
            t = time.perf_counter()
            engine.backward(dl, w, h, spp, salt=8)   # waits for its result
            times.append(time.perf_counter() - t)
        return min(times[2:])
    logged = best()
    monkeypatch.setenv("PTR_HIT_LOG_BYTES", "0")
    walked = best()
    assert logged < 0.9 * walked, (logged, walked)
