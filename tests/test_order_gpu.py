"""Tile lists of frames at the edges of the pair sort's three forms (one block up to 5,120
pairs, 4 keys per thread up to 524,288, 12 above): the depth sort, which leaves out the
Gaussians that the camera does not see, and the tile sort, whose record count lies on the
device below a fixed capacity. Against numpy's order (tile, depth key, id) of the
renderer's own rectangles and depths, exactly."""
import numpy as np
import pytest

import gsn
import scenes
from helpers import dev, empty, gsn_sorted_lists, host, sync, torch

pytestmark = pytest.mark.gpu


def expected_lists(renderer, cam, n, key_shift):
    b = renderer.buffers()
    seen = np.flatnonzero(host(b.tile_counts, np.int32, n))
    rects = host(b.rects, np.int32, 4 * n).reshape(n, 4)[seen].astype(np.int64)
    keys = host(b.depths, np.float32, n)[seen].view(np.uint32) >> key_shift
    width, height = rects[:, 2] - rects[:, 0], rects[:, 3] - rects[:, 1]
    counts = width * height
    owner = np.repeat(np.arange(len(seen)), counts)
    k = np.arange(len(owner)) - np.repeat(np.cumsum(counts) - counts, counts)
    tiles = (rects[owner, 1] + k // width[owner]) * cam.tile_count_x + rects[owner, 0] + k % width[owner]
    order = np.lexsort((seen[owner], keys[owner], tiles))
    return len(seen), seen[owner][order], np.searchsorted(tiles[order], np.arange(cam.tiles + 1))


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("n,capacity,away", [
    (300, 5000, False), (300, 5121, False), (5120, 0, False), (5121, 0, False), (5120, 0, True), (6000, 0, True),
    (20_000, 400_000, False), (20_000, 600_000, False), (524_288, 0, False), (524_289, 0, False)])
def test_lists_at_the_edges_of_the_sorts_forms(n, capacity, away, fast):
    t = torch()
    params = scenes.random_gaussians(n, n % 1000 + capacity % 77)
    params[3:6] -= 1.0
    params[0:3, : n // 5] = params[0:3, n // 5: 2 * (n // 5)]  # equal depths: ties by id
    cam = scenes.make_camera(403, 301, fx=90.0, fy=90.0)  # in the middle of the cloud
    if away:
        params[2] = -np.abs(params[2]) - 1.0
    p = dev(params)
    image = empty((cam.height, cam.width, 3), t.float32)
    r = gsn.Renderer()
    r.set_fast_blend(fast)
    if capacity:
        assert r.set_record_capacity(capacity) == 0
    for _ in range(2):  # the second frame finds the first one's scratch and buffers
        assert r.render(p.data_ptr(), n, cam, [0, 0, 0], image.data_ptr(), 0) == 0
    sync()
    seen, ids, offsets = expected_lists(r, cam, n, 8 if fast else 0)
    assert seen == 0 if away else 0.2 * n < seen < 0.8 * n
    if capacity:
        assert len(ids) < capacity
    got_ids, got_offsets = gsn_sorted_lists(r, cam)
    assert np.array_equal(got_offsets, offsets) and np.array_equal(got_ids, ids)


@pytest.mark.parametrize("n", [250_000, 470_000])
def test_more_records_than_an_int_counts_are_refused_or_reported(n):
    """Every Gaussian covers all 10,000 tiles: 2.5 and 4.7 billion records, beyond 2^31 and
    2^32. Grow mode refuses the frame; with a fixed capacity the records that fit are
    rendered and the overflow flag is set."""
    t = torch()
    params = scenes.random_gaussians(n, 4, mean_sigma=0.1)
    params[2] += 3.0
    params[3:6] = 4.0
    cam = scenes.make_camera(1600, 1600, fx=400.0, fy=400.0)
    p = dev(params)
    image = empty((1600, 1600, 3), t.float32)
    assert gsn.Renderer().render(p.data_ptr(), n, cam, [0, 0, 0], image.data_ptr(), 0) != 0
    r = gsn.Renderer()
    assert r.set_record_capacity(300_000) == 0
    assert r.render(p.data_ptr(), n, cam, [0, 0, 0], image.data_ptr(), 0) == 0
    sync()
    b = r.buffers()
    assert host(b.tile_counts, np.int32, n).astype(np.int64).sum() == n * cam.tiles
    assert host(b.overflow, np.int32, 1)[0] == 1 and bool(t.isfinite(image).all())
    ids, offsets = gsn_sorted_lists(r, cam)
    assert offsets[-1] == 300_000 and len(np.unique(ids)) == 30
