"""Panoramas with texels that are not finite, or beyond the FP32 range once a row of them
is added up: as the texel-by-texel projection (vlb_skybox_sh_noalloc) has them; and
rows whose sums cancel."""
import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu
PI = 3.1415926538  # shaders/sh_common.h:1


def texel_by_texel(torch, image, layout, w, h, lmax):
    dev, out = torch.from_numpy(image).cuda(), torch.zeros((vlb.k_of(lmax), 3), device="cuda")
    torch.cuda.synchronize()
    assert vlb.lib.vlb_skybox_sh_noalloc(dev.data_ptr(), vlb.TEXEL_RGB32F, layout, w, h, lmax, 0, out.data_ptr(),
                                         None) == vlb.OK
    return out.cpu().numpy()


def kind(a):
    return np.where(np.isnan(a), 3, np.where(np.isposinf(a), 1, np.where(np.isneginf(a), 2, 0)))


INF = np.float32(np.inf)
# (row, column, channel) -> value, fractions of the image
SPOTS = {"one": [(0.3, 0.4, 0, INF)], "negative": [(0.3, 0.4, 1, -INF)], "nan": [(0.5, 0.1, 2, np.float32(np.nan))],
         "pair": [(0.3, 0.4, 0, INF), (0.31, 0.9, 0, INF)], "opposite": [(0.3, 0.4, 0, INF), (0.7, 0.2, 0, -INF)],
         "same row": [(0.6, 0.1, 1, INF), (0.6, 0.35, 1, INF), (0.6, 0.8, 1, -INF)]}


@pytest.mark.parametrize("layout", [vlb.SKY_PANORAMA, vlb.SKY_ENVMAP])
@pytest.mark.parametrize("lmax", [2, 3])
@pytest.mark.parametrize("w,h", [(64, 33), (1500, 70), (2048, 1024)])
def test_texels_that_are_not_finite(ctx, w, h, lmax, layout):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(h)
    base = rng.uniform(0, 2, (h, w, 3)).astype(np.float32)
    for name, spots in SPOTS.items():
        image = base.copy()
        for y, x, c, v in spots:
            image[int(y * h), int(x * w), c] = v
        got, ref = ctx.skybox_sh(image, layout, w, h, lmax), texel_by_texel(torch, image, layout, w, h, lmax)
        assert np.array_equal(kind(got), kind(ref)), name
        ok = np.isfinite(ref)
        assert np.linalg.norm(got[ok] - ref[ok]) <= 1e-5 * np.linalg.norm(ref[ok]), name
    all_inf = np.full_like(base, INF)
    assert np.array_equal(kind(ctx.skybox_sh(all_inf, layout, w, h, lmax)),
                          kind(texel_by_texel(torch, all_inf, layout, w, h, lmax)))


@pytest.mark.parametrize("layout", [vlb.SKY_PANORAMA, vlb.SKY_ENVMAP])
@pytest.mark.parametrize("w,h", [(64, 33), (2048, 1024)])
def test_texels_whose_row_overflows(ctx, w, h, layout):
    torch = pytest.importorskip("torch")
    image = np.random.default_rng(w).uniform(0, 2, (h, w, 3)).astype(np.float32)
    image[h // 3] *= np.float32(1.5e38)
    got, ref = ctx.skybox_sh(image, layout, w, h, 3), texel_by_texel(torch, image, layout, w, h, 3)
    assert np.all(np.isfinite(ref)) and np.linalg.norm(got.astype(np.float64) - ref) <= 1e-5 * np.linalg.norm(
        ref.astype(np.float64))


@pytest.mark.parametrize("layout", [vlb.SKY_PANORAMA, vlb.SKY_ENVMAP])
@pytest.mark.parametrize("w,h", [(64, 33), (2048, 1024), (1500, 700), (8192, 4096)])
def test_rows_that_cancel(ctx, w, h, layout):
    """Rows of one whole number each: their sums are exact, so the first coefficient is,
    up to one rounding, an FP64 sum over the rows with the row weights in FP32."""
    rng = np.random.default_rng(w)
    c = rng.integers(-1000, 1001, h).astype(np.float64)
    c = np.where(np.arange(h) < h // 2, c, -c[::-1])
    th = PI * (np.arange(h) + 0.5) / h
    weight = np.float32((2.0 * PI / w) * (PI / h) * np.sin(th)).astype(np.float64)
    terms = 0.282095 * weight * (c * w)
    image = np.broadcast_to(np.float32(c)[:, None, None], (h, w, 3)).copy()
    got = ctx.skybox_sh(image, layout, w, h, 3)[0]
    ref = terms.sum()
    assert np.all(np.abs(got - ref) <= 2.0**-23 * abs(ref) + 2.0**-45 * np.abs(terms).sum())
