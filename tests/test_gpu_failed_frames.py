"""A frame that fails for lack of device memory leaves a defined film behind: a picture of it is
black, and the next frame starts from zero even if it accumulates (the C ABI's accumulate flag;
CudaEngine itself asks for a fresh frame then).

The failures are single allocations beyond the device's memory, which the runtime refuses: a
path pool of 2^30 paths (some 250 GB) and films of 10^10 and 4.9 * 10^9 pixels (sums of 240 GB, and
of 118 GB each, of which the second does not fit beside the first)."""
import ctypes as C

import numpy as np
import pytest

from pathtracerglsl_b200 import abi, scenes
from pathtracerglsl_b200.compiler import Compiler
from pathtracerglsl_b200.engine import EngineError

pytestmark = pytest.mark.gpu

W, H = 48, 32
SCENES = {
    "walk": lambda: scenes.cornell(),
    "walk-aov": lambda: _aovs(*scenes.cornell()),
    "wavefront": lambda: scenes.cornell_mesh_light(),
    "wavefront-aov": lambda: _aovs(*scenes.cornell_mesh_light()),
}


def _aovs(sc, st):
    return sc, dict(st, measurement=dict(st["measurement"], aovs=["albedo", "normal"]))


def _load(engine, name):
    r, pk = Compiler().compile(*SCENES[name]())
    engine.register_scene(pk)
    engine.load_renderer(r)
    engine.select_renderer(r.id)
    engine.pin_reset_salt(9)


def _frame(engine, w, h, spp, first=0, accumulate=False):
    """One ptr_render as a C caller makes it: the caller's own accumulate flag."""
    engine.width, engine.height = w, h
    engine.sample_count = first
    fr = engine._frame(w, h, spp, accumulate)
    engine._check(engine.lib.ptr_render(engine.programs[engine.current], engine.scene, C.byref(fr)))


def _pictures(engine):
    engine.width, engine.height = W, H
    names = ["radiance", "variance"] + (["albedo", "normal"] if engine.renderers[engine.current].program.aovs else [])
    return [engine.read_export(n).copy() for n in names]


def _fails(engine, *args, **kw):
    with pytest.raises(EngineError) as e:
        _frame(engine, *args, **kw)
    assert e.value.code == abi.PTR_E_NOMEM


def _same(a, b):
    for x, y in zip(a, b, strict=True):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("scene", ["wavefront", "wavefront-aov"])
def test_frame_after_a_failed_pool(engine, monkeypatch, scene):
    _load(engine, scene)
    _frame(engine, W, H, 2, first=5)
    want = _pictures(engine)
    spp = (1 << 30) // (W * H)
    _load(engine, scene)
    monkeypatch.setenv("PTR_CAPACITY", str(1 << 30))
    _fails(engine, W, H, spp)                             # the first frame of its film
    monkeypatch.delenv("PTR_CAPACITY")
    for picture in _pictures(engine):
        assert not picture.any()
    _frame(engine, W, H, 2, first=5, accumulate=True)
    _same(_pictures(engine), want)
    monkeypatch.setenv("PTR_CAPACITY", str(1 << 30))
    _fails(engine, W, H, spp)                             # a restart of a film that holds a picture
    monkeypatch.delenv("PTR_CAPACITY")
    _frame(engine, W, H, 2, first=5, accumulate=True)
    _same(_pictures(engine), want)
    monkeypatch.setenv("PTR_CAPACITY", str(1 << 30))
    _fails(engine, W, H, spp, first=7, accumulate=True)   # an addition: the picture stays
    monkeypatch.delenv("PTR_CAPACITY")
    _same(_pictures(engine), want)


@pytest.mark.parametrize("scene", sorted(SCENES))
def test_frame_after_a_film_that_does_not_fit(engine, scene):
    _load(engine, scene)
    _frame(engine, W, H, 2, first=5)
    want = _pictures(engine)
    for side in (70000, 100000):
        _frame(engine, W, H, 3)
        _fails(engine, side, side, 1)
        with pytest.raises(EngineError, match="nothing rendered"):
            _pictures(engine)
        _frame(engine, W, H, 2, first=5, accumulate=True)
        _same(_pictures(engine), want)


def test_jobs_after_a_failed_batch(engine):
    """The second job's film does not fit: the first job's film, already restarted, is fresh."""
    items = [Compiler().compile(*scenes.cornell(max_depth=d)) for d in (4, 5)]
    b = engine.batch(items)
    try:
        b.render([(W, H, 2, 0, 9), (W, H, 1, 0, 9)])
        want = [b.read_export(0, n).copy() for n in ("radiance", "variance")]
        with pytest.raises(EngineError) as e:
            b.render([(W, H, 3, 0, 9), (100000, 100000, 1, 0, 9)])
        assert e.value.code == abi.PTR_E_NOMEM
        assert not b.read_export(0).any()
        with pytest.raises(EngineError):
            b.render([(W, H, 3, 0, 9), (100000, 100000, 1, 0, 9)])
        arr = b._jobs([(W, H, 2, 0, 9), (W, H, 1, 0, 9)])
        for job in arr:
            job.frame.accumulate = 1
        engine._check(engine.lib.ptr_render_batch(engine.ctx, arr, len(arr)))
        _same([b.read_export(0, n) for n in ("radiance", "variance")], want)
    finally:
        b.close()
