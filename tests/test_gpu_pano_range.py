"""Panoramas with texels that are not finite, or beyond the FP32 range once a row of them
is added up: as the texel-by-texel projection (vlb_skybox_sh_noalloc) has them."""
import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu


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
