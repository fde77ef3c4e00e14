"""The blend kernels' region test and the exact culling's tile intervals on the device,
approximate divides, square roots and fused products included, where they are most
delicate: needles up to the condition number at which culling is switched off, grazing or
crossing the frame, opacities around 1/255. The renderer's image and contributor counts
against a float32 evaluation of every record of a tile at every pixel of it, without any
region test. Pixels with a record whose alpha is within rounding of the threshold are left
out of the comparison of counts."""
import numpy as np
import pytest

import gsn
import scenes
from helpers import dev, empty, gsn_sorted_lists, host, sync, torch

pytestmark = pytest.mark.gpu

F, D = np.float32, np.float64
W, H, COUNT = 101, 75, 500
LOG2E, LOG2_ALPHA_MIN = F(1.4426950408889634), F(-7.9943534368588578)


def fma(a, b, c):
    """float32 fused multiply-add (the product of two float32 is exact in float64)."""
    return (D(1) * a * b + c).astype(F)


def needles(seed):
    rng = np.random.default_rng(seed)
    p = scenes.random_gaussians(COUNT, seed)
    p[0] = rng.uniform(-1.6, 1.6, COUNT)
    p[1] = rng.uniform(-1.2, 1.2, COUNT)
    p[2] = rng.uniform(3.0, 6.0, COUNT)
    p[3] = rng.uniform(-4.0, 1.6, COUNT)        # one long axis, up to hundreds of pixels
    p[4:6] = rng.uniform(-7.0, -4.5, (2, COUNT))  # two that the low-pass filter bounds from below
    opacity = np.where(rng.random(COUNT) < 0.4, rng.uniform(0.9, 2.0, COUNT) / 255, rng.uniform(0.004, 0.99, COUNT))
    p[9] = np.log(opacity / (1 - opacity))
    cam = scenes.make_camera(W, H, fx=130.0, fy=130.0)
    return p.astype(F), cam


def blend(frame, cam, tile, fast):
    """Colours, contributor counts and which pixels' counts are certain, for one tile."""
    X, Y = np.meshgrid(np.arange(16) + tile % cam.tile_count_x * 16, np.arange(16) + tile // cam.tile_count_x * 16)
    X, Y = X.astype(F), Y.astype(F)
    T, C = np.ones(X.shape, F), np.zeros(X.shape + (3,), F)
    done, certain = np.zeros(X.shape, bool), np.ones(X.shape, bool)
    consumed = np.zeros(X.shape, np.int32)
    for k, i in enumerate(frame["ids"][frame["offsets"][tile]:frame["offsets"][tile + 1]]):
        A, B, Cc, o = frame["conic"][i]
        dx, dy = frame["means"][i, 0] - X, frame["means"][i, 1] - Y
        if fast:
            kx, ky, kz, kw = F(-0.5) * LOG2E * A, -LOG2E * B, F(-0.5) * LOG2E * Cc, np.log2(o)
            Ax, Bx = fma(kx * dx, dx, kw), ky * dx
            pw2 = fma(fma(kz, dy, Bx), dy, Ax)
            take = pw2 >= LOG2_ALPHA_MIN
            alpha = np.minimum(F(0.99), np.exp2(np.minimum(pw2, F(0))))
            close = np.abs(pw2 - LOG2_ALPHA_MIN) < F(1e-6) * (np.abs(Ax) + np.abs(Bx * dy) + F(8))
            nextT = T - alpha * T
        else:
            t = fma(A * dx, dx, (Cc * dy) * dy)
            power = fma(F(-0.5), t, -((B * dx) * dy))
            raw = o * np.exp(np.minimum(power, F(0)))
            take = (power <= 0) & (raw >= F(1 / 255))
            alpha = np.minimum(F(0.99), raw)
            close = np.abs(raw * F(255) - F(1)) < F(1e-6)
            nextT = T * (F(1) - alpha)
        take = take & ~done
        # within rounding of the threshold, or of the stop
        certain &= ~(close & ~done) & ~(take & (np.abs(nextT - F(1e-4)) < F(1e-8)))
        stop = take & (nextT < F(1e-4))
        done |= stop
        take &= ~stop
        w = np.where(take, alpha * T, F(0))
        C += w[..., None] * frame["colors"][i]
        T = np.where(take, nextT, T)
        consumed = np.where(take, k + 1, consumed)
    return C, consumed, certain


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("seed", [1, 2])
def test_no_region_test_changes_a_pixel(seed, fast):
    t = torch()
    params, cam = needles(seed)
    p = dev(params)
    frames = []
    for culled in (False, True):
        r = gsn.Renderer()
        r.set_fast_blend(fast)
        r.set_exact_culling(culled)
        image = empty((H, W, 3), t.float32)
        assert r.render(p.data_ptr(), COUNT, cam, [0, 0, 0], image.data_ptr(), 0) == 0
        sync()
        b = r.buffers()
        ids, offsets = gsn_sorted_lists(r, cam)
        frames.append(dict(image=image.cpu().numpy(), ids=ids, offsets=offsets,
                           means=host(b.means, F, 2 * COUNT).reshape(-1, 2),
                           conic=host(b.conic_opacity, F, 4 * COUNT).reshape(-1, 4),
                           colors=host(b.colors, F, 3 * COUNT).reshape(-1, 3),
                           consumed=host(b.contributors, np.int32, W * H).reshape(H, W)))
    plain, culled = frames
    assert len(culled["ids"]) < 0.5 * len(plain["ids"])
    assert np.array_equal(plain["image"], culled["image"])
    q = plain["conic"][np.unique(plain["ids"])].astype(D)
    half, disc = 0.5 * (q[:, 0] + q[:, 2]), np.hypot(0.5 * (q[:, 0] - q[:, 2]), q[:, 1])
    kappa = (half + disc) / (half - disc)
    assert kappa.max() > 3e4 and np.sum(kappa > 1e3) > 50
    compared = 0
    for frame in frames:
        for tile in range(cam.tiles):
            y, x = tile // cam.tile_count_x * 16, tile % cam.tile_count_x * 16
            h, w = min(16, H - y), min(16, W - x)
            colour, consumed, certain = blend(frame, cam, tile, fast)
            window = np.s_[y:y + h, x:x + w]
            sure = certain[:h, :w]
            compared += sure.sum()
            assert np.array_equal(frame["consumed"][window][sure], consumed[:h, :w][sure])
            # one approximate exponential per record taken
            assert np.abs(frame["image"][window] - colour[:h, :w])[sure].max(initial=0) < 2e-5
    assert compared > 1.9 * W * H
