"""Destinations that are pinned in part only: the device writes host memory itself only
where one pinned range holds all of the destination; any other is copied to by the host."""

import ctypes as C
import mmap

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu

PAGE = 65536  # a multiple of every host page size in use


@pytest.fixture(scope="module")
def memory():
    """32 pages, of which 4..7 and, apart from them, 8..9 and 12..13 are registered:
    (bytes as an array, address of each page)."""
    if not gpu_available():
        pytest.skip("no CUDA GPU")
    import torch

    torch.zeros(1, device="cuda")
    rt = torch.cuda.cudart()
    m = mmap.mmap(-1, 33 * PAGE)
    whole = np.frombuffer(m, np.uint8)
    at = -whole.ctypes.data % PAGE
    buf = whole[at:at + 32 * PAGE]
    base = buf.ctypes.data
    regs = [(4, 4), (8, 2), (12, 2)]
    for first, pages in regs:
        assert int(rt.cudaHostRegister(base + first * PAGE, pages * PAGE, 2)) == 0
    yield buf
    for first, _ in regs:
        assert int(rt.cudaHostUnregister(base + first * PAGE)) == 0


def test_only_a_whole_pinned_range_is_written_by_the_device(memory):
    from forkerrenderer_gb300 import _native as N

    f = N.lib().frctx_pinned_destination
    f.restype, f.argtypes = C.c_void_p, [C.c_int32, C.c_void_p, C.c_size_t]
    base = memory.ctypes.data
    p = lambda page, off=0: base + page * PAGE + off
    for at, n in [(p(4), 4 * PAGE), (p(4, 77), 1), (p(7, PAGE - 1), 1), (p(8), 2 * PAGE), (p(13), PAGE)]:
        assert f(0, at, n) == at, (at - base, n)
    for at, n in [(p(0), 1), (p(3), 2 * PAGE), (p(3, PAGE - 1), 2),  # pageable, at least at first
                  (p(4), 4 * PAGE + 1), (p(7, PAGE - 1), 2),         # into the next registration
                  (p(8), 2 * PAGE + 1), (p(9, PAGE - 1), 2),         # past the end
                  (p(8), 6 * PAGE), (p(9), 4 * PAGE),                # pinned at both ends, a hole between
                  (p(14), 1), (p(4), 0), (0, 16)]:
        assert f(0, at, n) is None, (at - base, n)
    assert f(1, p(4), PAGE) is None  # another device's
    assert f(0, p(4), (1 << 64) - 1) is None


@pytest.mark.parametrize("what", ["frame", "batch"])
def test_downloads_into_partly_pinned_memory(memory, what, tmp_path):
    """The same bytes whether the destination is pinned, pageable or both, and nothing
    written beside it."""
    import forkerrenderer_gb300 as fr
    from forkerrenderer_gb300 import _native as N
    from forkerrenderer_gb300.batch import Batch, point_light, view
    from scenes import render_config, stress_scene

    scene = fr.Scene(stress_scene(str(tmp_path), width=201, height=149))
    cfg = render_config("def_stress", shadow_size=64)
    r = fr.Renderer(**cfg)
    r.Preconfigure(scene)
    b = None
    if what == "frame":
        r.Render()
        get = lambda buf: r.download(N.FR_BUF_FRAME_U8, buf)
        want = r.frame8().reshape(-1)
    else:
        info = scene.info
        b = Batch(r, [view(scene.frame_matrices(64), info.eye)], [point_light(info.light_pos, info.light_color, 64)])
        b.render()
        want = b.download(0, N.FR_BUF_FRAME_U8).reshape(-1)

        def get(buf):
            assert N.lib().fr_batch_download(b._h, 0, N.FR_BUF_FRAME_U8, buf.ctypes.data_as(C.c_void_p), buf.size) >= 0
    n = want.size
    assert want.any() and PAGE < n < 3 * PAGE
    # within a range, across its end, across two, from pageable into one, and pageable
    for at in (4 * PAGE, 4 * PAGE + 5, 8 * PAGE - n + 1, 8 * PAGE - 3, 10 * PAGE - 16, 14 * PAGE - 1, 4 * PAGE - 7, 20 * PAGE + 1):
        memory[:] = 77
        get(memory[at:at + n])
        assert np.array_equal(memory[at:at + n], want), at
        assert (memory[at - 64:at] == 77).all() and (memory[at + n:at + n + 64] == 77).all(), at
    if b is not None:
        b.close()
    r.close()


def test_device_memory_as_destination():
    """fr_download into device memory copies there, as CUDA's copies do."""
    if not gpu_available():
        pytest.skip("no CUDA GPU")
    import torch

    import forkerrenderer_gb300 as fr
    from forkerrenderer_gb300 import _native as N
    from scenes import render_config, scene_path

    r = fr.Renderer(**render_config("def_pcss", shadow_size=64))
    r.Preconfigure(fr.Scene(scene_path("def_pcss")))
    r.Render()
    want = r.frame8()
    there = torch.zeros(want.size, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert N.lib().fr_download(r._h, N.FR_BUF_FRAME_U8, C.c_void_p(there.data_ptr()), want.size) == N.FR_OK
    assert np.array_equal(there.cpu().numpy(), want.reshape(-1))
    assert np.array_equal(r.frame8(), want)
    r.close()
