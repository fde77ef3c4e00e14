"""The backward blend for a camera with more tiles than the renderer's last frame: tiles
that frame had not keep the bounds and offsets of an older frame, and must add nothing
and read nothing past the record buffers."""
import numpy as np
import pytest

import gsn
import scenes
from helpers import dev, empty, host, sync, torch
from test_backward_segments_gpu import faint_scene, replay

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fast", [False, True])
def test_tiles_of_an_older_frame_add_nothing(fast):
    t = torch()
    n = 600
    params = faint_scene(n, 5)
    big = scenes.make_camera(64, 64, fx=60.0, fy=60.0)
    small = scenes.make_camera(64, 48, fx=60.0, fy=60.0)
    # half of the big frame's records lie in tile 12, the first that the small one has not;
    # the small frame's end close below that tile's end
    big.cx, big.cy, small.cx, small.cy = 4.0, 48.0, 4.0, 36.0
    p = dev(params)
    image = empty((64, 64, 3), t.float32)
    target = dev(np.random.default_rng(2).integers(0, 256, (64, 64, 3), dtype=np.uint8))
    probe = gsn.Renderer()
    assert probe.render(p.data_ptr(), n, big, [0, 0, 0], image.data_ptr(), 0) == 0
    records = int(probe.buffers().record_count_host)
    r, s = gsn.Renderer(), gsn.Solver()
    r.set_fast_blend(fast)
    assert r.set_record_capacity(records) == 0  # no slack behind the records of the big frame
    assert r.render(p.data_ptr(), n, big, [0, 0, 0], image.data_ptr(), 0) == 0
    assert r.render(p.data_ptr(), n, small, [0, 0, 0], image.data_ptr(), 0) == 0
    gptr = s.image_gradients(big, image.data_ptr(), target.data_ptr())
    sync()
    b = r.buffers()
    offsets = host(b.tile_offsets, np.int64, big.tiles + 1)
    held = int(offsets[small.tiles])
    assert 0.7 * records < held <= offsets[small.tiles + 1]
    f = dict(grad=host(gptr, np.float32, image.numel()).reshape(64, 64, 3).astype(np.float64),
             image=image.cpu().numpy().astype(np.float64), means=host(b.means, np.float32, 2 * n).reshape(n, 2),
             conic=host(b.conic_opacity, np.float32, 4 * n).reshape(n, 4).astype(np.float64),
             colors=host(b.colors, np.float32, 3 * n).reshape(n, 3).astype(np.float64),
             ids=host(b.tile_gaussian_ids, np.int32, held), offsets=offsets,
             limit=host(b.contributors, np.int32, big.pixels).reshape(64, 64))
    expected = replay(f, small, n)
    sptr = s.screen_gradients(big, r, image.data_ptr(), p.data_ptr(), n)
    sync()
    screen = host(sptr, np.float32, 12 * n).reshape(n, 12)
    scale = np.abs(expected).max(0)
    # fp32 terms summed in float atomics over tiles and segments
    assert np.all(np.abs(screen[:, :11] - expected) <= 1e-4 * np.abs(expected) + 1e-5 * scale)
