"""The maps' device memory beside what else the process does."""
import threading

import numpy as np
import pytest

from tests.helpers import MAXCAM, SCALING, circle_frames

pytestmark = pytest.mark.gpu


def _make(leaves=30000):
    from fastfusion_b200.fusion import FusionMipMapCPU
    return FusionMipMapCPU(0, 0, 0, 0.005, 0.01, 0, True, leaves_max=leaves, branches_max=1 << 21, rcp="exact")


def _fuse(m, n=4, wh=(160, 120)):
    from fastfusion_b200.fusion import CameraInfo
    K, frames = circle_frames(0, n, *wh)
    m.addMapSequence([f[0] for f in frames], [CameraInfo(K, f[2], f[3]) for f in frames], [f[1] for f in frames],
                     SCALING, MAXCAM)
    return [np.array(x) for x in (*m.bricks(), *m.leaves())]


def _same(a, b):
    return all(x.shape == y.shape and x.tobytes() == y.tobytes() for x, y in zip(a, b))


def test_closing_and_growing_while_another_thread_records(lib_built):
    """A thread records a stream (thread-local mode, as this library's own
    recordings) while another closes a map, makes one and grows its buffers: the
    recording stays whole and the maps are right."""
    import torch
    m = _make()
    want = _fuse(m)
    x = torch.zeros(1000, device="cuda")
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    got, errors = [], []

    def other():
        try:
            m.close()
            k = _make()
            _fuse(k, 2, (97, 61))
            k.close()
            k = _make()
            got.append(_fuse(k))
            k.close()
        except Exception as e:  # (reported by the main thread)
            errors.append(repr(e))

    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="thread_local")
        x.add_(1.0)
        t = threading.Thread(target=other)
        t.start()
        t.join()
        x.add_(1.0)
        g.capture_end()
    assert not errors, errors
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 6.0
    assert _same(got[0], want)


def test_image_that_does_not_fit_leaves_the_map_usable(lib_built):
    """The buffers of a larger image cannot be allocated (the device is full): the
    call fails, again too, and the map goes on with the image size it had, is
    closed, and leaves the next map unharmed."""
    import torch
    from fastfusion_b200.fusion import CameraInfo, FFError
    k = _make()
    want = _fuse(k, 8)
    k.close()
    K, frames = circle_frames(0, 8, 160, 120)
    cams = [CameraInfo(K, R, t) for _, _, R, t in frames]
    m = _make()
    for (depth, bgr, _, _), cam in list(zip(frames, cams))[:3]:
        m.addMap(depth, cam, bgr, SCALING, MAXCAM)
    large = np.full((6000, 8000), 5000, np.uint16)  # 66 B of buffers per pixel, 3.2 GB
    colour = np.zeros((6000, 8000, 3), np.uint8)
    other = _make()
    torch.cuda.synchronize()
    full = torch.empty(torch.cuda.mem_get_info()[0] - (600 << 20), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        with pytest.raises(FFError) as e:
            m.addMap(large, cams[3], colour, SCALING, MAXCAM)
        assert "out of memory" in str(e.value)
    for (depth, bgr, _, _), cam in list(zip(frames, cams))[3:5]:
        m.addMap(depth, cam, bgr, SCALING, MAXCAM)
    m.addMapSequence([f[0] for f in frames[5:]], cams[5:], [f[1] for f in frames[5:]], SCALING, MAXCAM)
    assert _same([np.array(x) for x in (*m.bricks(), *m.leaves())], want)
    m.close()
    del full
    torch.cuda.empty_cache()
    assert _same(_fuse(other, 8), want)
    other.close()


def test_kept_memory_is_given_back(lib_built):
    """What closed maps leave: at most 1 GB at once (the rest is back when the
    call returns), all of it with release_memory."""
    import torch
    from fastfusion_b200.fusion import release_memory
    torch.cuda.synchronize()
    k = _make()
    _fuse(k)
    k.updateMeshes()
    k.close()
    release_memory()
    before = torch.cuda.mem_get_info()[0]
    k = _make(leaves=400000)  # 2.9 GB
    _fuse(k)
    k.updateMeshes()
    k.close()
    assert before - torch.cuda.mem_get_info()[0] < (1 << 30) + (256 << 20)
    release_memory()
    assert before - torch.cuda.mem_get_info()[0] < 64 << 20


def test_mesh_gets_what_closed_maps_left(lib_built):
    """The device is full but for what closed maps left: a mesh update that needs
    buffers gets them."""
    import torch
    from fastfusion_b200.fusion import release_memory
    a, b = _make(60000), _make(60000)
    for m in (a, b):
        _fuse(m, 8, (640, 480))
    b.updateMeshes()
    want = b.getMeshInterleavedMarchingCubes()
    b.close()
    release_memory()
    k = _make(120000)  # 0.9 GB
    k.close()
    torch.cuda.synchronize()
    full = torch.empty(torch.cuda.mem_get_info()[0] - (4 << 20), dtype=torch.uint8, device="cuda")
    a.updateMeshes()
    del full
    torch.cuda.empty_cache()
    got = a.getMeshInterleavedMarchingCubes()
    assert len(got.faces) > 0
    assert got.vertices.tobytes() == want.vertices.tobytes() and np.array_equal(got.faces, want.faces)
    a.close()
