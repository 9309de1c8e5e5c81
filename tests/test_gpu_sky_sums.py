"""The last step of a sky projection adds the partial sums without losing bits: an
image whose partial sums cancel gives what its parts give one by one, added in FP64."""
import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu


def cancelling(parts, ones, rng):
    """A factor for each part, after which the parts' sums of value 0 cancel (ones: their
    sums with factor 1)."""
    w = ones[:, 0, 0].astype(np.float64)
    c = rng.normal(size=len(parts))
    return (c - w * (c @ w) / (w @ w)).astype(np.float32)


def check(whole, parts):
    parts = parts.astype(np.float64)
    ref = parts.sum(0)
    # one rounding of the result to FP32, and of FP64 sums of the parts
    assert np.all(np.abs(whole - ref) <= 2.0**-23 * np.abs(ref) + 2.0**-45 * np.abs(parts).sum(0))


@pytest.mark.parametrize("lmax", [2, 3])
@pytest.mark.parametrize("n", [64, 128, 130])
def test_cubemap(ctx, n, lmax):
    rng = np.random.default_rng(n + lmax)
    part = np.arange(6 * n * n) // 1024  # texels of a partial sum
    m = part[-1] + 1
    image = rng.uniform(0.5, 2, (6 * n * n, 3)).astype(np.float32)

    def alone(c):
        maps = np.where((part == np.arange(m)[:, None])[..., None], image * c[part][:, None], np.float32(0))
        return ctx.skybox_sh(maps, vlb.SKY_CUBEMAP, n, n, lmax, count=m)

    c = cancelling(range(m), alone(np.ones(m, np.float32)), rng)
    whole = ctx.skybox_sh(image * c[part][:, None], vlb.SKY_CUBEMAP, n, n, lmax)
    check(whole, alone(c))


@pytest.mark.parametrize("layout", [vlb.SKY_CUBEMAP, vlb.SKY_PANORAMA])
def test_without_allocation(layout):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    w, h = (64, 64) if layout == vlb.SKY_CUBEMAP else (256, 128)
    T = (6 if layout == vlb.SKY_CUBEMAP else 1) * w * h
    t = np.arange(T)
    part = t // 8192 * 8 + t % 256 // 32  # a slab's texels by the warp that adds them up
    m = part[-1] + 1
    image = rng.uniform(0.5, 2, (T, 3)).astype(np.float32)
    out = torch.zeros((16, 3), device="cuda")

    def run(img):
        dev = torch.from_numpy(img).cuda()
        torch.cuda.synchronize()
        assert vlb.lib.vlb_skybox_sh_noalloc(dev.data_ptr(), vlb.TEXEL_RGB32F, layout, w, h, 3, 0, out.data_ptr(),
                                             None) == vlb.OK
        return out.cpu().numpy()

    def alone(c):
        return np.array([run(image * np.where(part == k, c[k], np.float32(0))[:, None]) for k in range(m)])

    c = cancelling(range(m), alone(np.ones(m, np.float32)), rng)
    check(run(image * c[part][:, None]), alone(c))
