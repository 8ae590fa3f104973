"""Frames and batches that a caller captures into a graph of its own: the
renderer goes on rendering afterwards, with and without blits, past the ring
of staging buffers and past the growth of every device buffer, and each launch
of the caller's graph still gives the frame that was captured."""
import numpy as np
import pytest

import scenes
import swr

pytestmark = pytest.mark.gpu
W, H = 210, 130


@pytest.fixture(scope="module")
def small():
    s = swr.Scene(scenes.small_scene(seed=4))
    yield s
    s.close()


@pytest.fixture(scope="module")
def large():
    """More nodes, triangles and bin entries than the small scene's buffers hold."""
    s = swr.Scene(scenes.spheres_scene(seed=4, count=300, subdiv=3, tex_size=16, cube_size=16, voxel=16))
    yield s
    s.close()


def camera(s, i):
    pos, at, fov, w, h, far = scenes.default_camera_params(s.info(), W, H)
    return swr.make_camera((pos[0] + 0.1 * i, pos[1], pos[2] - 0.05 * i), at, fov, w, h, far)


def fresh(s, cam):
    r = swr.Renderer(W, H)
    r.render(s, cam)
    out = r.blit(), r.visbuffer()
    r.close()
    return out


def captured(torch, stream, call, mode="relaxed"):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream, capture_error_mode=mode):
        call()
    return g


def replayed(torch, r, graph):
    graph.replay()
    torch.cuda.synchronize()
    return r.blit(), r.visbuffer()


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("blit", [True, False])
@pytest.mark.parametrize("warm", [1, 3, 8])
def test_renderer_goes_on(small, warm, blit):
    torch = pytest.importorskip("torch")
    r, s = swr.Renderer(W, H), torch.cuda.Stream()
    for i in range(warm):
        r.render(small, camera(small, i), stream=s.cuda_stream)
        r.blit(stream=s.cuda_stream)
    cam = camera(small, 3)
    graph = captured(torch, s, lambda: r.render(small, cam, stream=s.cuda_stream))
    want = fresh(small, cam)
    for _ in range(2):
        assert same(replayed(torch, r, graph), want)
        for i in range(9):
            r.render(small, camera(small, 20 + i), stream=s.cuda_stream)
            if blit:
                assert same((r.blit(stream=s.cuda_stream), r.visbuffer()), fresh(small, camera(small, 20 + i))), i
        assert same((r.blit(), r.visbuffer()), fresh(small, camera(small, 28)))
    assert same(replayed(torch, r, graph), want)
    r.close()


def test_graph_outlives_growth(small, large):
    """Every buffer grows between two launches of the graph; a graph of the larger scene beside it."""
    torch = pytest.importorskip("torch")
    r, s = swr.Renderer(W, H), torch.cuda.Stream()
    r.render(small, camera(small, 0), stream=s.cuda_stream)
    r.sync()
    ca, cb = camera(small, 3), camera(large, 2)
    a = captured(torch, s, lambda: r.render(small, ca, stream=s.cuda_stream))
    before = r.stats().bin_capacity
    for i in range(6):
        r.render(large, camera(large, i), stream=s.cuda_stream)
        assert same((r.blit(), r.visbuffer()), fresh(large, camera(large, i))), i
    assert r.stats().bin_capacity > before
    b = captured(torch, s, lambda: r.render(large, cb, stream=s.cuda_stream))
    for _ in range(3):
        assert same(replayed(torch, r, a), fresh(small, ca))
        assert same(replayed(torch, r, b), fresh(large, cb))
    r.close()


def test_many_captures(small):
    """Staging buffers of dropped graphs are used again; those of kept graphs are not."""
    torch = pytest.importorskip("torch")
    r, s = swr.Renderer(W, H), torch.cuda.Stream()
    r.render(small, camera(small, 0), stream=s.cuda_stream)
    r.sync()
    kept = []
    for i in range(12):
        cam = camera(small, i)
        g = captured(torch, s, lambda: r.render(small, cam, stream=s.cuda_stream))
        assert same(replayed(torch, r, g), fresh(small, cam)), i
        if i % 4 == 1:
            kept.append((g, cam))
        g.reset() if i % 4 != 1 else None
        r.render(small, camera(small, 30 + i), stream=s.cuda_stream)
        r.sync()
    for g, cam in kept:
        assert same(replayed(torch, r, g), fresh(small, cam))
    r.close()


def test_captured_exposure_steps(small):
    """Each launch of a captured frame with dt > 0 is one exposure step of that dt, whatever steps follow the capture."""
    torch = pytest.importorskip("torch")
    cam = camera(small, 1)
    r, p, s = swr.Renderer(W, H), swr.Renderer(W, H), torch.cuda.Stream()
    for x in (r, p):
        x.render(small, cam, 0.0, s.cuda_stream)
        x.sync()
    graph = captured(torch, s, lambda: r.render(small, cam, 0.1, s.cuda_stream))
    for i in range(6):
        if i % 3 == 2:
            for x in (r, p):
                x.render(small, camera(small, i), 0.02, s.cuda_stream)
                x.sync()
        else:
            graph.replay()
            torch.cuda.synchronize()
            p.render(small, cam, 0.1)
            assert same((r.blit(), r.visbuffer()), (p.blit(), p.visbuffer())), i
        assert r.exposure() == p.exposure(), i
    for x in (r, p):
        x.close()


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_capture_modes_and_growth_while_captured(small, large, mode):
    """Captures of a new renderer, of one whose buffers have to grow, and two frames in one capture."""
    torch = pytest.importorskip("torch")
    r, s = swr.Renderer(W, H), torch.cuda.Stream()
    a = captured(torch, s, lambda: r.render(small, camera(small, 1), stream=s.cuda_stream), mode)
    b = captured(torch, s, lambda: r.render(large, camera(large, 2), stream=s.cuda_stream), mode)

    def two():
        r.render(large, camera(large, 3), stream=s.cuda_stream)
        r.render(small, camera(small, 4), stream=s.cuda_stream)

    c = captured(torch, s, two, mode)
    for _ in range(2):
        for graph, (sc, i) in ((a, (small, 1)), (b, (large, 2)), (c, (small, 4))):
            assert same(replayed(torch, r, graph), fresh(sc, camera(sc, i))), i
        for i in range(6):
            r.render(small, camera(small, 10 + i), stream=s.cuda_stream)
        assert same((r.blit(), r.visbuffer()), fresh(small, camera(small, 15)))
    r.close()


def test_captured_batch(small, large):
    torch = pytest.importorskip("torch")
    b, s = swr.Batch(), torch.cuda.Stream()

    def outputs(n):
        return torch.zeros(n, H, W, dtype=torch.int32, device="cuda"), torch.zeros(n, H, W, dtype=torch.int64, device="cuda")

    def views(items, rgba, vis):
        v = swr.Batch.views([(sc, cam, W, H, 2.0, swr.RSQRT_AARCH64) for sc, cam in items])
        for i in range(len(items)):
            v[i].rgba8, v[i].vis = rgba[i].data_ptr(), vis[i].data_ptr()
        return v

    few = [(small, camera(small, i)) for i in range(2)]
    many = [(large, camera(large, i)) for i in range(7)]
    rgba, vis = outputs(2)
    v = views(few, rgba, vis)
    b.render(v, s.cuda_stream)
    b.sync()
    graph = captured(torch, s, lambda: b.render(v, s.cuda_stream))
    rgba2, vis2 = outputs(7)
    v2 = views(many, rgba2, vis2)
    for _ in range(3):
        for _ in range(6):
            b.render(v2, s.cuda_stream)
        b.sync()
        rgba.zero_(), vis.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for got, items in (((rgba, vis), few), ((rgba2, vis2), many)):
            for i, (sc, cam) in enumerate(items):
                want_rgba, want_vis = fresh(sc, cam)
                assert np.array_equal(got[0][i].cpu().numpy().view(np.uint32)[:H & ~1], want_rgba[:H & ~1]), i
                assert np.array_equal(got[1][i].cpu().numpy().view(np.uint64), want_vis), i
    b.close()
