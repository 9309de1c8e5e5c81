"""Probe frontiers of dense scenes, whose lists are longer than the 128 entries of
ordinary ones (up to 256, 512 and 1024 by the scene's layers), against packet walks:
the same bits, for walks that take the list in stages and for one that may not."""
import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu


def nested(n):
    """n concentric boxes in a room: a probe near the centre is inside all of them."""
    one, idx, alb = vlb.synth_box_scene(3, 1)
    room, corner = one[:8] - 0.5, one[8:] - one[8:].mean(0)
    s = np.linspace(1.0, 4.0, n)[:, None, None]
    pos = np.concatenate([room * 9, (corner[None] / np.abs(corner).max(0) * s).reshape(-1, 3)]).astype(np.float32)
    tri = np.concatenate([idx[:10]] + [idx[10:] + 8 * k for k in range(n)]).astype(np.uint32)
    return pos, tri, np.concatenate([alb[:10]] + [alb[10:]] * n).astype(np.float32)


@pytest.mark.parametrize("boxes", [300, 1500, 6000])
def test_long_lists_keep_their_bits(ctx, boxes):
    rng = np.random.default_rng(boxes)
    scene = ctx.scene(*nested(boxes))
    # inside all boxes, between them, outside
    probes = np.concatenate([rng.uniform(-0.1, 0.1, (9, 3)), rng.uniform(-4.2, 4.2, (37, 3)),
                             rng.uniform(-9, 9, (5, 3))]).astype(np.float32)
    ds = ctx.fibonacci(200)
    got = {}
    for flags in (vlb.BAKE_TRAVERSAL_PACKET, vlb.BAKE_TRAVERSAL_LANE):
        p = vlb.bake_params(ds, 2, vlb.PREC_FP32, (0.3, 0.9, 0.2), flags=flags)
        got[flags] = ctx.bake(scene, probes, p, debug=True)
    for a, b in zip(*got.values()):
        assert np.array_equal(a, b)
    fused = vlb.bake_params(ds, 2, vlb.PREC_FUSED, (0.3, 0.9, 0.2))
    one = ctx.bake(scene, probes, fused)
    for refill in (32, 16):
        sched = vlb.BatchSchedule(dirs_per_item=0, cost_order=1, graph=0, ctas_per_sm=8, node_steps=6, refill_idle=refill)
        jobs = [(scene, probes, None), (scene, probes[::2].copy(), None)]
        a, b = ctx.bake_batch(jobs, fused, sched)
        assert np.array_equal(a, one) and np.array_equal(b, one[::2])
