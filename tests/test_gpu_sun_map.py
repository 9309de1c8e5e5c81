"""Shadow rays answered by the sun map (bakes of many rays) against
packet walks, which trace every one of them: visibility, radiance and
coefficients must be the same bits.

Suns: high, grazing, along an axis (walls seen edge on), from below; scenes:
boxes, a bumpy sheet of small triangles (every ray near its own surface), one
triangle, degenerate triangles, far from the origin; a ray limit that ends
shadow rays before their occluder; a shadow origin far off its surface.
"""
import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu


def sheet(m):
    g = np.linspace(0, 1, m + 1)
    x, z = np.meshgrid(g, g)
    p = np.stack([x, 0.1 * np.sin(9 * x) * np.cos(7 * z), z], -1).reshape(-1, 3)
    i = (np.arange(m)[:, None] * (m + 1) + np.arange(m)).reshape(-1, 1)
    t = np.concatenate([i + [0, m + 1, m + 2], i + [0, m + 2, 1]], 1).reshape(-1, 3)
    return p.astype(np.float32), t.astype(np.uint32), np.full((len(t), 3), 0.5, np.float32)


def scenes():
    pos, idx, alb = vlb.synth_box_scene(21, 300)
    yield "boxes", pos, idx, alb
    yield "far", pos + np.float32([400, -300, 250]), idx, alb
    yield "sheet", *sheet(60)
    yield "one", pos[idx[7]], np.uint32([[0, 1, 2]]), alb[:1]
    flat = np.concatenate([idx, np.stack([idx[:, 0], idx[:, 1], idx[:, 0]], 1)])
    yield "degenerate", pos, flat, np.concatenate([alb, alb])


SUNS = [((0.3, 0.9, 0.2), 1e4, 0.005), ((1.0, 0.02, 0.01), 1e4, 0.005), ((0, 1, 0), 1e4, 0.005),
        ((0.2, -3.0, 0.1), 1e4, 0.005), ((0.3, 0.9, 0.2), 0.1, 0.005), ((0.3, 0.9, 0.2), 1e4, 0.5)]


@pytest.mark.parametrize("sun,tmax,bias", SUNS)
@pytest.mark.parametrize("precision", [vlb.PREC_FP32, vlb.PREC_FUSED])
def test_mapped_shadows_keep_their_bits(ctx, sun, tmax, bias, precision):
    rng = np.random.default_rng(8)
    ds = ctx.fibonacci(1024)
    for name, pos, idx, alb in scenes():
        scene = ctx.scene(pos, idx, alb)
        b = scene.bounds(False)
        probes = (b[:3] + rng.uniform(-0.1, 1.1, (1300, 3)) * np.maximum(b[3:] - b[:3], 0.1)).astype(np.float32)
        out = []
        for prec, flags in ((vlb.PREC_FP32, vlb.BAKE_TRAVERSAL_PACKET), (precision, vlb.BAKE_TRAVERSAL_LANE)):
            p = vlb.bake_params(ds, 2, prec, sun, flags=flags)
            p.tmax, p.shadow_bias = tmax, bias
            out.append(ctx.bake(scene, probes, p, debug=True))
        for k, (x, y) in enumerate(zip(*out)):
            if k or precision == vlb.PREC_FP32:  # the fused sums have an order of their own
                assert np.array_equal(x, y), (name, k)
