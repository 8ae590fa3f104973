"""The exposure resolve writes four pixels a thread as one vector where the
target's address allows: frame widths around the vector and row-piece sizes,
blit targets at every alignment and with padded rows. The target must equal
the copying blit, and nothing outside the frame's rows may change."""
import numpy as np
import pytest

import scenes
import swr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 4), (2, 3), (3, 2), (5, 7), (63, 5), (130, 9), (1021, 4), (1023, 3), (1026, 4)])
def test_resolve_into_any_alignment(w, h):
    s = swr.Scene(scenes.small_scene(seed=8, count=3))
    cam = swr.make_camera(*scenes.default_camera_params(s.info(), w, h))
    for lead in range(4):
        for pad in (0, 1, 4):
            stride = w + pad
            mem = np.full(stride * h + 16, 0xABCDEF01, np.uint32)
            r = swr.Renderer(w, h)
            r.set_blit_target(mem.ctypes.data + 4 * lead, stride, keep=mem)
            r.render(s, cam, 0.05)
            r.sync()
            want = r.blit()
            r.close()
            rows = h & ~1
            expect = np.full_like(mem, 0xABCDEF01)
            for y in range(rows):
                expect[lead + y * stride:lead + y * stride + w] = want[y]
            assert np.array_equal(mem, expect), (lead, pad)
    s.close()
