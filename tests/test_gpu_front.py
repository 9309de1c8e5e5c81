"""Lane walks that start at probe frontiers against packet walks, which start at
the root: per-ray decisions, radiance and coefficients must be the same bits.

Sizes: ray groups that straddle probes (direction counts not a multiple of
32), the smallest scene and direction count with a frontier, lists cut at
their capacity (origins inside hundreds of boxes), probes outside the scene and
far from it, axis-parallel directions, a scene far from the origin.
"""
import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu


def nested_boxes(n):
    """n concentric boxes around the unit cube's centre: a probe there is inside all of them."""
    one, idx, alb = vlb.synth_box_scene(3, 1)
    room, corner = one[:8] - 0.5, one[8:] - one[8:].mean(0)
    s = np.linspace(0.2, 4.0, n)[:, None, None]
    pos = np.concatenate([room * 5, (corner[None] / np.abs(corner).max(0) * s).reshape(-1, 3)]).astype(np.float32)
    tri = np.concatenate([idx[:10]] + [idx[10:] + 8 * k for k in range(n)]).astype(np.uint32)
    return pos, tri, np.concatenate([alb[:10]] + [alb[10:]] * n).astype(np.float32)


def scenes():
    pos, idx, alb = vlb.synth_box_scene(21, 300)
    rng = np.random.default_rng(4)
    around = rng.uniform(-0.3, 1.3, (37, 3))
    yield "boxes", pos, idx, alb, around
    yield "far", pos + np.float32([1000, -1000, 250]), idx, alb, around + [1000, -1000, 250]
    yield "smallest", *vlb.synth_box_scene(2, 5), np.concatenate([around[:5], around[:4] * 1e4])
    yield "nested", *nested_boxes(400), rng.uniform(-0.02, 0.02, (9, 3))


@pytest.mark.parametrize("S", [64, 130, 515, 1024])
@pytest.mark.parametrize("precision", [vlb.PREC_FP32, vlb.PREC_MIXED])
def test_walks_from_frontiers_keep_their_bits(ctx, S, precision):
    rng = np.random.default_rng(S)
    d = rng.normal(size=(S, 3))
    d[:6] = [[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1]]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    ds = ctx.dirset(d, np.full(S, 4 * np.pi / S))
    for name, pos, idx, alb, probes in scenes():
        scene, probes = ctx.scene(pos, idx, alb), probes.astype(np.float32)
        out = []
        for flags in (vlb.BAKE_TRAVERSAL_PACKET, vlb.BAKE_TRAVERSAL_LANE):
            p = vlb.bake_params(ds, 2, precision, (0.3, 0.9, 0.2), flags=flags)
            out.append(ctx.bake(scene, probes, p, debug=True))
        for a, b in zip(*out):
            assert np.array_equal(a, b), (name, S)
