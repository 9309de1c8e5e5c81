"""The reference's point-light shading with shadow rays answered by the light's
map (bakes of many rays) against the 32-probe packets of a small bake's size,
whose shadow rays all walk: visibility and radiance must be the same bits.

Lights: the reference's own, one close above the scene, one that grazes its
walls, one inside the scene (no map), one below; a wide bias.
"""
import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("light,bias", [((1, 10, 1), 0.005), ((0.4, 1.6, 0.6), 0.005), ((30, 0.5, 0.5), 0.005),
                                        ((0.5, 0.5, 0.5), 0.005), ((0.2, -3, 0.1), 0.005), ((1, 10, 1), 0.2)])
@pytest.mark.parametrize("nboxes", [0, 64, 1500])
def test_mapped_point_light_keeps_its_bits(ctx, light, bias, nboxes):
    pos, idx, alb = vlb.synth_box_scene(31, nboxes)
    scene, ds = ctx.scene(pos, idx, alb), ctx.fibonacci(1024)
    probes = np.random.default_rng(3).uniform(-0.1, 1.1, (4000, 3)).astype(np.float32)

    def bake(pr):
        p = vlb.bake_params(ds, 3, vlb.PREC_FP32, shading=vlb.SHADE_REF_PHONG, light_pos=light)
        p.shadow_bias = bias
        return ctx.bake(scene, pr, p, debug=True)

    whole = bake(probes)
    for at in range(0, 4000, 500):  # 40 probes at a time: too few rays for a map
        part = bake(probes[at:at + 40])
        for a, b in zip(whole[1:], part[1:]):
            assert np.array_equal(a[at:at + 40], b), (light, at)
