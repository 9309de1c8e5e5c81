"""Light maps over triangles seen nearly edge on, where the FP32 triangle test's
error is far larger than a cell's margin: a shadow ray that the packet walk, which
tests every box and triangle on its way, finds occluded must be occluded with a map.

Slivers tilted by 5e-6 to 5e-5 against the line to the light stand over a receiver
that faces it; probes close above the receiver aim their rays at the slivers'
shadow edges.
"""
import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu

LIGHT = np.float32([4.0, 3.5, 5.0])
AIMS = 400  # shadow-edge points a sliver


def unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def slivers(light, seed):
    """(positions, indices, shadow-edge points, axis): 144 slivers over a receiver of two
    triangles facing `light` (a direction, or a point if it has a 1 behind it)."""
    rng = np.random.default_rng(seed)
    point = len(light) == 4
    to = np.asarray(light[:3], np.float64)
    axis = unit(to)
    u = unit(np.cross(axis, [0.1, 1.0, 0.3]))
    v = np.cross(axis, u)
    foot = -0.9 * axis
    pos = [foot + 1.4 * (a * u + b * v) for a, b in ((-1, -1), (1, -1), (1, 1), (-1, 1))]
    aims = []
    for g in range(144):
        at = 0.15 * ((g % 12 - 5.5) * u + (g // 12 - 5.5) * v) + rng.uniform(-0.3, 0.3) * axis
        d = unit(to - at) if point else axis
        across = unit(np.cross(d, rng.normal(size=3)))
        along = (d + 10 ** rng.uniform(-5.3, -4.3) * across) * rng.uniform(0.12, 0.25)
        tri = np.array([at, at + along, at + unit(rng.normal(size=3)) * rng.uniform(0.08, 0.17)])
        tri = tri[np.roll([0, 1, 2], rng.integers(3))][:: rng.choice([-1, 1])]
        pos += list(tri)
        i, w = rng.integers(3, size=AIMS), rng.random((AIMS, 1))
        x = tri[i] * (1 - w) + tri[(i + 1) % 3] * w
        r = unit(to - x) if point else axis  # down onto the receiver
        aims.append(x - r * (((x - foot) @ axis) / (r @ axis if point else 1.0))[..., None])
    n = (len(pos) - 4) // 3
    idx = np.concatenate([[[0, 1, 2], [0, 2, 3]], 4 + np.arange(3 * n).reshape(n, 3)])
    return np.float32(pos), idx.astype(np.uint32), np.concatenate(aims), axis


def meets_box(x, r, tris):
    """Whether each ray meets some triangle's box.  (A lane also tests the triangle that
    its last shadow ray met, without its box; what only that finds is no walk's answer.)"""
    lo, hi = tris.min(1)[None], tris.max(1)[None]
    a, b = (lo - x[:, None]) / r[:, None], (hi - x[:, None]) / r[:, None]
    return (np.minimum(a, b).max(-1) <= np.maximum(a, b).min(-1)).any(1)


@pytest.mark.parametrize("kind,seed", [("sun", 1), ("sun", 2), ("point", 1), ("point", 2), ("point", 3)])
def test_no_occluder_is_left_out(ctx, kind, seed):
    light = np.append(LIGHT, 1) if kind == "point" else LIGHT
    pos, idx, aims, axis = slivers(light, seed)
    rng = np.random.default_rng(100 + seed)
    S = 1024
    d = rng.normal(size=(S, 3))
    d -= axis * (d @ axis)[:, None]
    d = unit(rng.random((S, 1)) * unit(d) - axis)  # down, within 45 degrees
    probes = np.float32(aims + 10 ** rng.uniform(-3.5, -2, (len(aims), 1)) * axis)
    scene, ds = ctx.scene(pos, idx, np.full((len(idx), 3), 0.5, np.float32)), ctx.dirset(d, np.full(S, 4 * np.pi / S))

    def bake(part, flags):
        if kind == "sun":
            p = vlb.bake_params(ds, 2, vlb.PREC_FP32, LIGHT, flags=flags)
        else:
            p = vlb.bake_params(ds, 2, vlb.PREC_FP32, shading=vlb.SHADE_REF_PHONG, light_pos=tuple(LIGHT))
        p.tmin = 0.0
        p.shadow_bias = 0.0005
        return ctx.bake(scene, part, p, debug=True)[1:3]

    left_out = shadowed = 0
    for at in range(0, len(probes), 8000):
        part = probes[at:at + 8000]
        hit, vis = bake(part, vlb.BAKE_TRAVERSAL_LANE)
        if kind == "sun":
            hit0, vis0 = bake(part, vlb.BAKE_TRAVERSAL_PACKET)
        else:  # too few rays for a map: every shadow ray walks
            few = [bake(part[k:k + 200], 0) for k in range(0, len(part), 200)]
            hit0, vis0 = (np.concatenate(x) for x in zip(*few))
        floor = (hit == hit0) & (hit >= 0) & (hit < 2)
        assert floor.mean() > 0.9
        shadowed += np.count_nonzero(floor & (vis0 == 0))
        k, t = np.nonzero(floor & (vis0 == 0) & (vis == 1))
        x = part[k] - d[t] * (((part[k] - pos[0]) @ axis) / (d[t] @ axis))[:, None] + 0.0005 * axis
        r = unit(light[:3] - x) if kind == "point" else np.broadcast_to(axis, x.shape)
        left_out += np.count_nonzero(meets_box(x, r, pos[idx[2:]]))
    assert shadowed > 1000
    assert left_out == 0
