"""Where a batch's 8-bit frames go (fr_batch_download): frames whose copy is split over
several threads, and a process that can have no pinned memory."""

import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, TESTS, gpu_available

pytestmark = pytest.mark.gpu

EYE = (0.0, 6.0, 9.0)


def _need_gpu():
    if not gpu_available():
        pytest.skip("no CUDA GPU")


def _scene_and_view(width, height):
    """A small deferred scene and a camera of its own size: (scene, config, matrices)."""
    import forkerrenderer_gb300 as fr
    from scenes import render_config, scene_path

    scene = fr.Scene(scene_path("def_ao_128"))
    cfg = render_config("def_ao_128", ssao_samples=4)
    m = scene.view_matrices(EYE, (0, 0, 0), cfg["shadow_size"])
    m.width, m.height = width, height
    vp = np.array([[width / 2, 0, 0, width / 2], [0, height / 2, 0, height / 2], [0, 0, 0.5, 0.5], [0, 0, 0, 1]], np.float32)
    m.viewport[:] = list(vp.reshape(-1))
    return scene, cfg, m


def _batch(scene, cfg, m):
    import forkerrenderer_gb300 as fr
    from forkerrenderer_gb300.batch import Batch, point_light, view

    r = fr.Renderer(**cfg)
    r.Preconfigure(scene)
    info = scene.info
    b = Batch(r, [view(m, EYE)], [point_light(info.light_pos, info.light_color, cfg["shadow_size"])])
    b.render()
    return b


def _download_into(b, buf, n):
    from forkerrenderer_gb300 import _native as N

    return N.lib().fr_batch_download(b._h, 0, N.FR_BUF_FRAME_U8, buf.ctypes.data_as(C.c_void_p), n)


@pytest.mark.parametrize("width,height", [(1023, 701), (1281, 901), (1501, 1001)])
def test_threaded_copies_match_the_single_frame(width, height):
    """Frames of 2, 3 and 4 MiB and some odd bytes, into pageable memory at an odd address:
    the bytes that fr_render_frame gives for the same camera and light, and none beside them."""
    _need_gpu()
    import forkerrenderer_gb300 as fr

    scene, cfg, m = _scene_and_view(width, height)
    r = fr.Renderer(**cfg)
    r.Preconfigure(scene)
    r.set_matrices(m, EYE)
    r.Render()
    want = r.frame8().reshape(-1)
    assert want.size == 3 * width * height and want.any()
    b = _batch(scene, cfg, m)
    buf = np.full(want.size + 16, 77, np.uint8)
    assert _download_into(b, buf[7:], want.size) >= 0
    assert np.array_equal(buf[7:7 + want.size], want)
    assert (buf[:7] == 77).all() and (buf[7 + want.size:] == 77).all()
    b.close()
    r.close()


FAKE = r"""
#include <dlfcn.h>
#include <stddef.h>
int fail_pinned = 0, asked = 0;
int cudaHostAlloc(void** p, size_t n, unsigned flags)
{
    ++asked;
    if (fail_pinned) return 2; /* cudaErrorMemoryAllocation */
    int (*real)(void**, size_t, unsigned) =
        (int (*)(void**, size_t, unsigned))dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaHostAlloc");
    return real ? real(p, n, flags) : 2;
}
"""

CHILD = r"""
import ctypes as C, sys
sys.path[:0] = [%r, %r]
import numpy as np
import test_batch_downloads_gpu as T
from forkerrenderer_gb300 import _native as N

fake = C.CDLL(%r)
fail, asked = C.c_int.in_dll(fake, "fail_pinned"), C.c_int.in_dll(fake, "asked")
scene, cfg, m = T._scene_and_view(161, 97)
first = T._batch(scene, cfg, m)
want = first.download(0, N.FR_BUF_FRAME_U8)
assert want.any() and asked.value > 0  # pinned memory was asked for, of the fake
import forkerrenderer_gb300 as fr
from forkerrenderer_gb300.batch import Batch, point_light, view
r = fr.Renderer(**cfg)
r.Preconfigure(scene)
info = scene.info
fail.value, asked.value = 1, 0
b = Batch(r, [view(m, T.EYE)], [point_light(info.light_pos, info.light_color, cfg["shadow_size"])])
b.render()
assert np.array_equal(b.download(0, N.FR_BUF_DEPTH), first.download(0, N.FR_BUF_DEPTH))
assert asked.value == 0  # none for a batch whose frames are not read as bytes
assert np.array_equal(b.download(0, N.FR_BUF_FRAME_U8), want)
assert asked.value > 0
fail.value = 0
assert np.array_equal(b.download(0, N.FR_BUF_FRAME_U8), want)
print("ok")
"""


def test_batch_without_pinned_memory(tmp_path):
    """With every pinned allocation failing (a stand-in for cudaHostAlloc in front of the
    runtime's) a batch is created, renders, and gives the same frame."""
    _need_gpu()
    src, so = tmp_path / "fake.c", str(tmp_path / "fake.so")
    src.write_text(FAKE)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", so, str(src), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD % (ROOT, TESTS, so)], capture_output=True, text=True,
                       env=dict(os.environ, LD_PRELOAD=so), timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr
