"""The backward blend on frames of few tiles, where a tile's list is cut into segments
that start from the forward pass's checkpoints: screen-space gradients of lists from a
handful of records to more than sixteen strides (the warps share them evenly) against
a float64 replay of the renderer's own lists, in both arithmetic forms, on ragged
frames, and the same frame just above and below the tile count that switches it on."""
import numpy as np
import pytest

import gsn
import scenes
from helpers import dev, empty, host, sync, torch

pytestmark = pytest.mark.gpu


def frame(params, cam, target, fast):
    t = torch()
    n = params.shape[1]
    p, tgt = dev(params), dev(target)
    image = empty((cam.height, cam.width, 3), t.float32)
    r, s = gsn.Renderer(), gsn.Solver()
    r.set_fast_blend(fast)
    assert r.render(p.data_ptr(), n, cam, [0.1, 0.2, 0.3], image.data_ptr(), 0) == 0
    gptr = s.image_gradients(cam, image.data_ptr(), tgt.data_ptr())
    sync()
    grad = host(gptr, np.float32, image.numel()).reshape(cam.height, cam.width, 3).astype(np.float64)
    sptr = s.screen_gradients(cam, r, image.data_ptr(), p.data_ptr(), n)
    sync()
    b = r.buffers()
    records = int(b.record_count_host)
    return dict(screen=host(sptr, np.float32, 12 * n).reshape(n, 12), grad=grad,
                image=image.cpu().numpy().astype(np.float64), means=host(b.means, np.float32, 2 * n).reshape(n, 2),
                conic=host(b.conic_opacity, np.float32, 4 * n).reshape(n, 4).astype(np.float64),
                colors=host(b.colors, np.float32, 3 * n).reshape(n, 3).astype(np.float64),
                ids=host(b.tile_gaussian_ids, np.int32, records),
                offsets=host(b.tile_offsets, np.int64, cam.tiles + 1),
                limit=host(b.contributors, np.int32, cam.pixels).reshape(cam.height, cam.width))


def replay(f, cam, n):
    out = np.zeros((n, 11))
    for tile in range(cam.tiles):
        ys = np.arange(tile // cam.tile_count_x * 16, min(tile // cam.tile_count_x * 16 + 16, cam.height))
        xs = np.arange(tile % cam.tile_count_x * 16, min(tile % cam.tile_count_x * 16 + 16, cam.width))
        Y, X = np.meshgrid(ys, xs, indexing="ij")
        g, lim = f["grad"][Y, X], f["limit"][Y, X]
        T, P, S = np.ones(X.shape), np.zeros(X.shape), (g * f["image"][Y, X]).sum(-1)
        for k, i in enumerate(f["ids"][f["offsets"][tile]:f["offsets"][tile + 1]]):
            if k >= lim.max():
                break
            A, B, C, o = f["conic"][i]
            dx, dy = f["means"][i, 0].astype(np.float64) - X, f["means"][i, 1].astype(np.float64) - Y
            raw = o * np.exp(-0.5 * (A * dx * dx + C * dy * dy) - B * dx * dy)
            take = (k < lim) & (raw >= 1 / 255)
            if not take.any():
                continue
            alpha = np.where(take, np.minimum(raw, 0.99), 0.0)
            w, G = alpha * T, g @ f["colors"][i]
            common = np.where(raw < 0.99, (P + T * G - S) / (1 - alpha) * alpha, 0.0)
            qx, qy = A * dx + B * dy, B * dx + C * dy
            u, v = common * qx, common * qy
            out[i] += [-u.sum(), -v.sum(), 0.5 * (u * qx).sum(), (u * qy).sum(), 0.5 * (v * qy).sum(),
                       (1 - o) * common.sum(), *np.einsum("yx,yxc->c", w, g), np.abs(u).sum(), np.abs(v).sum()]
            P += w * G
            T *= 1 - alpha
    return out


def faint_scene(count, seed):
    """`count` faint Gaussians in front of a small camera: nothing saturates."""
    rng = np.random.default_rng(seed)
    p = scenes.random_gaussians(count, seed, mean_sigma=0.25)
    p[2] += 4.0
    p[3:6] = rng.normal(-2.6, 0.4, (3, count))
    p[9] = rng.normal(-4.2, 0.5, count)
    return p


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("count,width,height", [(60, 33, 20), (129, 16, 16), (700, 41, 17), (5000, 30, 30)])
def test_segments_match_a_float64_replay(count, width, height, fast):
    params = faint_scene(count, count)
    cam = scenes.make_camera(width, height, fx=60.0, fy=60.0)
    target = np.random.default_rng(1).integers(0, 256, (height, width, 3), dtype=np.uint8)
    f = frame(params, cam, target, fast)
    if count == 5000:
        assert f["limit"].max() > 17 * 128
    expected = replay(f, cam, count)
    scale = np.abs(expected).max(0)
    # fp32 terms summed in float atomics over tiles and segments
    assert np.all(np.abs(f["screen"][:, :11] - expected) <= 1e-4 * np.abs(expected) + 1e-5 * scale)
    assert not f["screen"][:, 11].any()


@pytest.mark.parametrize("fast", [False, True])
def test_the_tile_count_rule_leaves_gradients_alone(fast):
    # 64 x 64 tiles keep checkpoints, 65 x 64 do not; the model covers the same corner of both
    params = faint_scene(3000, 9)
    screens = []
    for width in (1024, 1040):
        cam = scenes.make_camera(width, 1024, fx=60.0, fy=60.0)
        cam.cx, cam.cy = 20.0, 20.0
        target = np.full((1024, width, 3), 90, np.uint8)
        f = frame(params, cam, target, fast)
        screens.append(f["screen"] * cam.pixels)  # the loss is a mean over the pixels
    scale = np.abs(screens[0]).max(0)
    assert np.all(np.abs(screens[0] - screens[1]) <= 1e-4 * np.abs(screens[0]) + 1e-5 * scale)
