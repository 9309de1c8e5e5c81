"""Scene loads on the device: the clustered tree and its node layout at the
sizes where the build changes form (blocks of 224 clusters, the one-CTA end at
2048, more blocks than a merge block adds up itself, one and two triangles), as
bakes that equal those through the Karras tree; and what a load refuses.
"""
import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu


def soup(n, seed=5):
    rng = np.random.default_rng(seed)
    c = rng.random((n, 1, 3))
    size = 2.0 / max(4, n) ** (1 / 3)
    pos = (c + rng.uniform(-size, size, (n, 3, 3))).reshape(-1, 3).astype(np.float32)
    return pos, np.arange(3 * n, dtype=np.uint32).reshape(n, 3), rng.random((n, 3)).astype(np.float32)


@pytest.mark.parametrize("n", [1, 2, 3, 223, 224, 225, 449, 2047, 2048, 2049, 5000, 70_001, 470_000])
def test_trees_of_every_size_agree(ctx, n):
    pos, idx, alb = soup(n)
    ds = ctx.fibonacci(96)
    probes = np.random.default_rng(n).random((40, 3)).astype(np.float32)
    out = []
    for flags in (0, vlb.SCENE_TRAVERSAL_LBVH, vlb.SCENE_TRAVERSAL_WIDE):
        scene = ctx.scene(pos, idx, alb, flags=flags)
        p = vlb.bake_params(ds, 2, vlb.PREC_FP32, (0.3, 0.9, 0.2))
        out.append(ctx.bake(scene, probes, p, debug=True))
        b = scene.bounds(False)
        assert np.array_equal(b[:3], pos.min(0)) and np.array_equal(b[3:], pos.max(0))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)


def test_equal_triangles_load(ctx):
    """Every pair of clusters ties: the clustering still ends."""
    pos, idx, alb = soup(1)
    scene = ctx.scene(pos, np.tile(idx, (5000, 1)), np.tile(alb, (5000, 1)))
    p = vlb.bake_params(ctx.fibonacci(64), 2, vlb.PREC_FP32)
    one = ctx.scene(pos, idx, alb)
    probes = np.float32([[0.5, 0.5, 3.0], [2, 2, 2]])
    assert np.array_equal(ctx.bake(scene, probes, p), ctx.bake(one, probes, p))


@pytest.mark.parametrize("at", [0, 7, 3 * 3000 - 1])
def test_refused_geometry(ctx, at):
    pos, idx, alb = soup(3000)
    bad = idx.copy()
    bad.reshape(-1)[at] = len(pos)
    with pytest.raises(vlb.VlbError) as e:
        ctx.scene(pos, bad, alb)
    assert e.value.status == vlb.ERR_INVALID and f"at {at}" in e.value.message
    for v in (np.nan, np.inf):
        p2 = pos.copy()
        p2[at, 1] = v
        with pytest.raises(vlb.VlbError) as e:
            ctx.scene(p2, idx, alb)
        assert e.value.status == vlb.ERR_INVALID and f"vertex {at}" in e.value.message


def test_device_arrays_load_like_host_arrays(ctx):
    torch = pytest.importorskip("torch")
    pos, idx, alb = soup(4000)
    host = ctx.scene(pos, idx, alb).bvh_export()
    dev = ctx.scene(torch.from_numpy(pos).cuda(), torch.from_numpy(idx.view(np.int32)).cuda(),
                    torch.from_numpy(alb).cuda()).bvh_export()
    for k in host:
        assert np.array_equal(host[k], dev[k])
