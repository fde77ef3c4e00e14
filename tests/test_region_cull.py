"""CPU check of the formula of the blend kernels' region test (raster_common.cuh cull_limit
and region_hit), restated in float32 with exact divides: a record it drops for a rectangle
of pixels has alpha below 1/255 at each of them. Conics up to the condition number at which
culling is switched off, means inside, beside and far from the rectangle, opacities down to
the threshold. The kernels' own arithmetic is checked in test_region_cull_gpu.py."""
import numpy as np
import pytest

F = np.float32


def cull_limit(mean, q):
    lo = F(255) * q[:, 3]
    det = q[:, 0] * q[:, 2] - q[:, 1] * q[:, 1]
    tr = F(0.5) * (q[:, 0] + q[:, 2])
    disc = np.sqrt(np.maximum(tr * tr - det, F(0)))
    kappa = (tr + disc) / np.maximum(tr - disc, F(1e-30))
    Q = F(2) * np.log(np.maximum(lo, F(1e-30))) * (F(1.02) + F(1e-6) * kappa) + F(0.05)
    Q = np.where((q[:, 0] > 0) & (q[:, 2] > 0) & (det > 0) & (kappa < 1e5), Q, F(np.inf))
    return np.where(lo > 1, Q, F(-1)).astype(F)


def region_hit(mean, q, limit, x0, x1, y0, y1):
    a, b, c = q[:, 0], F(2) * q[:, 1], q[:, 2]
    lx, hx, ly, hy = x0 - mean[:, 0], x1 - mean[:, 0], y0 - mean[:, 1], y1 - mean[:, 1]
    dx, dy = np.minimum(np.maximum(F(0), lx), hx), np.minimum(np.maximum(F(0), ly), hy)
    ey = np.minimum(np.maximum((F(-0.5) * b / c) * dx, ly), hy)
    ex = np.minimum(np.maximum((F(-0.5) * b / a) * dy, lx), hx)
    q1 = (c * ey + b * dx) * ey + a * dx * dx
    q2 = (a * ex + b * dy) * ex + c * dy * dy
    return ~(np.minimum(q1, q2) > limit)


@pytest.mark.parametrize("width,height", [(8, 8), (16, 8), (8, 4)])
@pytest.mark.parametrize("kappa", [1.0, 30.0, 3e3, 9e4])
def test_a_dropped_record_passes_at_no_pixel_of_the_region(width, height, kappa):
    rng = np.random.default_rng(int(kappa) + width)
    n = 20000
    x0, y0 = F(1600), F(1064)
    small = np.exp(rng.uniform(np.log(0.3), np.log(400), n))     # smaller variance, pixels^2
    large = small * kappa * rng.uniform(0.5, 1.0, n)
    th = rng.uniform(0, np.pi, n)
    co, si = np.cos(th), np.sin(th)
    A = co * co / large + si * si / small
    B = co * si * (1 / large - 1 / small)
    C = si * si / large + co * co / small
    o = np.where(rng.random(n) < 0.3, rng.uniform(0.9, 1.6, n) / 255, rng.uniform(0.004, 1, n))
    q = np.stack([A, B, C, o], 1).astype(F)
    # means along the long axis, so that ellipses graze the rectangle
    reach = np.sqrt(large) * rng.normal(0, 2.5, n)
    side = np.sqrt(small) * rng.normal(0, 2.5, n)
    mean = np.stack([x0 + rng.uniform(0, width, n) + co * reach - si * side,
                     y0 + rng.uniform(0, height, n) + si * reach + co * side], 1).astype(F)
    hit = region_hit(mean, q, cull_limit(mean, q), x0, x0 + F(width - 1), y0, y0 + F(height - 1))
    assert 0.02 < hit.mean() < 0.98
    drop = ~hit
    m, k = mean[drop], q[drop]
    for y in range(height):
        for x in range(width):
            dx, dy = m[:, 0] - (x0 + F(x)), m[:, 1] - (y0 + F(y))
            power = F(-0.5) * (k[:, 0] * dx * dx + k[:, 2] * dy * dy) - k[:, 1] * dx * dy
            with np.errstate(over="ignore"):
                alpha = k[:, 3] * np.exp(power)
            assert not ((alpha >= F(1 / 255)) & (power <= 0)).any()
