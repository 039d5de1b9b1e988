"""A scene is uploaded while a frame of another renders: the upload returns with the frame still in
flight (a stream of uploads carries the copies), the frame's picture is what it is alone, and the
uploaded scene renders as one uploaded to an idle context.  Uploads that run kernels (trees built
on the device, rails) may have to wait for room beside the frame's; their pictures agree too.
Contexts on several threads share that stream: each thread's scenes render as they do alone."""
import ctypes as C
import threading

import numpy as np
import pytest

from pathtracerglsl_b200 import _native, abi, rails, scenes
from pathtracerglsl_b200.compiler import Compiler
from pathtracerglsl_b200.engine import CudaEngine, EngineError

pytestmark = pytest.mark.gpu


def _small():
    return scenes.cornell_rough()


def _mesh():
    sc, st, _ = scenes.mesh_scene(level=4, instances=5, env_size=(256, 128), max_depth=4)
    return sc, st


@pytest.mark.parametrize("scene,build", [(_small, "host"), (_mesh, "host"), (_mesh, "device"), (_mesh, "rails")],
                         ids=["tables", "host-trees", "device-trees", "rails"])
def test_upload_beside_a_frame(scene, build):
    eng = CudaEngine(0)
    try:
        r, pk = Compiler().compile(*scenes.cornell(max_depth=16, rr_start=None))
        other, packed = Compiler().compile(*scene())
        packed_rails = rails.pack(packed, _native.load()) if build == "rails" else None
        channels = packed_rails.struct() if packed_rails else None
        eng.set_accel_build("device" if build == "device" else "host")

        def upload():
            desc, h = packed.desc(), C.c_void_p()
            if channels is not None:
                eng._check(eng.lib.ptr_upload_scene_rails(eng.ctx, C.byref(desc), C.byref(channels), C.byref(h)))
            else:
                eng._check(eng.lib.ptr_upload_scene(eng.ctx, C.byref(desc), C.byref(h)))
            return h

        def picture(h):
            p, fr = C.c_void_p(), abi.Frame()
            eng._check(eng.lib.ptr_compile(eng.ctx, C.byref(other.program), C.byref(p)))
            fr.width, fr.height, fr.spp, fr.reset_salt = 40, 30, 2, 5
            fr.camera = other.camera({}, 40, 30)
            out = np.zeros((30, 40, 3), np.float32)
            eng._check(eng.lib.ptr_render(p, h, C.byref(fr)))
            eng._check(eng.lib.ptr_read_export(p, b"radiance", out.ctypes.data_as(C.POINTER(C.c_float)), out.size))
            eng._check(eng.lib.ptr_free_program(p))
            eng._check(eng.lib.ptr_free_scene(h))
            return out

        def long_frame():   # some hundreds of milliseconds
            eng.reset()
            eng.render_frame(1024, 1024, 512)
        eng.register_scene(pk)
        eng.load_renderer(r)
        eng.pin_reset_salt(3)
        long_frame()
        want = eng.read_export("radiance").copy()
        idle = picture(upload())
        long_frame()
        h = upload()
        if build == "host":
            with pytest.raises(EngineError) as e:   # the frame is still in flight
                eng.sync(0)
            assert e.value.code == abi.PTR_E_TIMEOUT
        np.testing.assert_array_equal(eng.read_export("radiance"), want)
        np.testing.assert_array_equal(picture(h), idle)
    finally:
        eng.close()


def test_contexts_on_several_threads():
    jobs = [_small(), _mesh(), scenes.cornell(max_depth=3), scenes.cornell_mesh_light(), _mesh(), scenes.het_fog(max_depth=3)]
    compiled = [Compiler().compile(*j) for j in jobs]
    want, got, errors = [None] * len(jobs), [[] for _ in jobs], []

    def render(k, eng):
        r, pk = compiled[k]
        eng.set_accel_build("device" if k % 2 else "host")
        eng.register_scene(pk)
        eng.load_renderer(r)
        eng.select_renderer(r.id)
        eng.pin_reset_salt(7)
        eng.reset()
        eng.render_frame(37, 29, 2)
        return eng.read_export("radiance").copy()

    def work(k):
        try:
            for _ in range(4):
                eng = CudaEngine(0)
                got[k] += [render(k, eng) for _ in range(3)]
                eng.close()
        except Exception as e:   # noqa: BLE001
            errors.append(e)
    for k in range(len(jobs)):
        eng = CudaEngine(0)
        want[k] = render(k, eng)
        eng.close()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for w, pictures in zip(want, got, strict=True):
        assert len(pictures) == 12
        for p in pictures:
            np.testing.assert_array_equal(p, w)
