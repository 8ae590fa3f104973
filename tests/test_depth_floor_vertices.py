"""The depth floor with what the front end passes it: the vertices' own
clip-space z and w and the end of the whole bounding box, where 1/w spans many
decades and its rounded differences no longer give the vertices back. It must
not exceed a depth that the tile raster computes for a covered lane
(oracle_packet_depths walks each packet)."""
import numpy as np
import pytest

import oracle
import swr
from test_depth_floor import bbox, record, tiles, triangle

f32 = np.float32
RANGES = {"plain": (0.05, 500.0), "steep": (1e-3, 100.0), "near plane": (1e-7, 1e3), "far apart": (1e-20, 1e10)}


def vertices(rng, span, depth):
    """Clip-space w, and z from behind the camera's far plane to past the near one, or all on one plane."""
    w = np.exp(rng.uniform(np.log(span[0]), np.log(span[1]), 3)).astype(f32)
    if rng.random() < 0.3:
        w[rng.integers(3)] = f32(span[0])
    z = rng.uniform(*depth, 3).astype(f32) if rng.random() < 0.8 else np.full(3, rng.uniform(*depth), f32)
    return (w * z).astype(f32), w


@pytest.mark.parametrize("depth", [(-1.0, 1.2), (0.99, 1.0)])
@pytest.mark.parametrize("name", list(RANGES))
def test_floor_below_every_covered_depth(name, depth):
    rng = np.random.default_rng(len(name) * 10 + int(depth[1] * 10))
    taken = covered = differ = 0
    for i in range(1500):
        xy = triangle(rng, ("any", "any", "sliver")[i % 3])
        rec = record(rng, xy)
        if rec is None:
            continue
        p, ooa, _, _ = rec
        z, w = vertices(rng, RANGES[name], depth)
        o = (f32(1.0) / w).astype(f32)
        zw = (z * o).astype(f32)
        zow = np.array([zw[0], zw[1] - zw[0], zw[2] - zw[0]], f32)
        oow = np.array([o[0], o[1] - o[0], o[2] - o[0]], f32)
        back = oow[0] + oow[1:]
        differ += bool(np.any(np.abs(back * w[1:] - 1.0) > 1e-6))
        bb = bbox(p)
        zlo = swr.selftest_depth_floor_vertices(p, zow, oow, z, w, bb[2] * 16, bb[3] * 16)
        for rect in tiles(rng, bb):
            zmin, lanes = oracle.packet_depths(p, ooa, zow, oow, rect)
            if lanes == 0:
                continue
            covered += 1
            taken += zlo != -np.inf
            assert zlo <= zmin, (p.tolist(), float(ooa), z.tolist(), w.tolist(), rect.tolist(), zlo, zmin)
    print("%s %s: floor taken for %d of %d covered packets; %d triangles whose interpolants lost a vertex"
          % (name, depth, taken, covered, differ))
    assert covered > 300
    if name in ("plain", "steep"):
        assert taken > 0.5 * covered
    else:
        assert differ > 100
