"""Sequences of more frames than one update pass takes: the second chunk's marks
are made while the first chunk's pass may still run, and none is lost (small
images: the chunk's allocation is shorter than the pass)."""
import numpy as np
import pytest

from tests.helpers import MAXCAM, SCALING, circle_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [17, 20, 33, 40])
def test_long_sequence_equals_frame_by_frame(lib_built, n):
    from fastfusion_b200.fusion import CameraInfo, FusionMipMapCPU
    K, frames = circle_frames(0, n, 160, 120)

    def make():
        return FusionMipMapCPU(0, 0, 0, 0.005, 0.01, 0, True, leaves_max=100000, branches_max=1 << 21, rcp="exact")

    one = make()
    for depth, bgr, R, t in frames:
        one.addMap(depth, CameraInfo(K, R, t), bgr, SCALING, MAXCAM)
    want = one.bricks()
    for _ in range(8):
        s = make()
        s.addMapSequence([f[0] for f in frames], [CameraInfo(K, f[2], f[3]) for f in frames], [f[1] for f in frames],
                         SCALING, MAXCAM)
        got = s.bricks()
        for a, b in zip(got, want):
            assert np.array_equal(a.view(np.uint16), b.view(np.uint16))
        s.close()
    one.close()
