"""A probe's projection has the same bits alone and beside any number of others, at
every length of rows: vlb_bake_batch and the service promise the bits of vlb_bake."""
import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu


# whole rows; two splits; splits of two lengths; rows that TMA cannot take (S % 4, S % 8)
@pytest.mark.parametrize("S", [2000, 2048, 4100, 5003, 20000])
@pytest.mark.parametrize("dtype", [vlb.DTYPE_F32, vlb.DTYPE_BF16, vlb.DTYPE_BF16_SPLIT])
def test_tiles_of_any_size(ctx, S, dtype):
    torch = pytest.importorskip("torch")
    ds = ctx.fibonacci(S)
    most, lmax = 13500, 3  # 40,500 rows: more row tiles than SMs
    wide = 2 * S if dtype == vlb.DTYPE_BF16_SPLIT else S
    tile = torch.rand((most, 3, wide), device="cuda", dtype=torch.float32)
    if dtype != vlb.DTYPE_F32:
        tile = tile.to(torch.bfloat16).view(torch.int16)
    rows = {}
    for n in (most, 4000, 1700, 43, 1):
        out = torch.empty((n, vlb.k_of(lmax), 3), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        ctx.project(tile[:n], n, ds, lmax, dtype=dtype, out=out)
        ctx.synchronize()
        rows[n] = out
    for n, out in rows.items():
        assert torch.equal(out, rows[most][:n]), n


@pytest.mark.parametrize("precision", [vlb.PREC_FP32, vlb.PREC_MIXED])
def test_slices_of_a_bake(ctx, precision):
    pos, idx, alb = vlb.synth_box_scene(4, 20)
    scene, ds = ctx.scene(pos, idx, alb), ctx.fibonacci(4099)
    probes = np.random.default_rng(2).uniform(0, 1, (900, 3)).astype(np.float32)
    p = vlb.bake_params(ds, 2, precision, (0.3, 0.9, 0.2))
    whole = ctx.bake(scene, probes, p)
    jobs = [(scene, probes[a:b].copy(), None) for a, b in ((0, 1), (1, 40), (40, 900))]
    assert np.array_equal(whole, np.concatenate([ctx.bake(s, x, p) for s, x, _ in jobs]))
    assert np.array_equal(whole, np.concatenate(ctx.bake_batch(jobs, p)))
