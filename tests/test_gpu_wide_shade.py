"""The shading kernel's CTAs have 1,024 threads, one to an SM, from four rounds
of 1,024 pixels per SM (of 152) on, and 128 below: padded sizes on both sides,
odd widths, each reciprocal square root, and views of mixed sizes and modes in
one launch, against the oracle."""
import numpy as np
import pytest

import oracle
import scenes
import swr

pytestmark = pytest.mark.gpu
MODES = (swr.RSQRT_AARCH64, swr.RSQRT_IEEE)


@pytest.fixture(scope="module")
def scene():
    s = swr.Scene(scenes.small_scene(seed=12))
    yield s
    s.close()


def close_to_oracle(s, cam, w, h, mode, rgba, vis):
    want, wvis, _, _ = oracle.render(s, cam, w, h, rsqrt_mode=mode)
    assert np.array_equal(vis, wvis)
    d = np.abs(rgba[:h & ~1].view(np.uint8).astype(np.int32) - want[:h & ~1].view(np.uint8).astype(np.int32))
    assert d.max() <= 1


def camera(s, w, h):
    pos, at, fov, w, h, far = scenes.default_camera_params(s.info(), w, h)
    return swr.make_camera(pos, at, fov, w, h, far)


@pytest.mark.parametrize("size", [(960, 640), (1023, 611), (1920, 333)])
@pytest.mark.parametrize("mode", MODES)
def test_frames_on_both_sides(scene, size, mode):
    w, h = size
    cam = camera(scene, w, h)
    r = swr.Renderer(w, h, rsqrt_mode=mode, sched_tile=32)
    r.render(scene, cam)
    close_to_oracle(scene, cam, w, h, mode, r.blit(), r.visbuffer())
    r.close()


def test_views_of_mixed_sizes_and_modes(scene):
    sizes = [(64, 64), (1023, 611), (65, 3), (130, 257), (700, 401)]
    items = [(scene, camera(scene, w, h), w, h, 2.0, MODES[i % 2]) for i, (w, h) in enumerate(sizes)]
    b = swr.Batch(sched_tile=32)
    b.render(swr.Batch.views(items))
    for i, (s, cam, w, h, _, mode) in enumerate(items):
        close_to_oracle(s, cam, w, h, mode, *b.output(i, w, h))
    b.close()
