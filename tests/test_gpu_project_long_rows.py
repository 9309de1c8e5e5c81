"""tcgen05 projections of rows long enough to be split (more than 4096 values):
against FP64 on the samples the tile holds, and the same bits for a probe alone and
beside others."""
import numpy as np
import pytest

import oracle as O
import vlb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [False, True])
# values a row: 4096 (whole), one more TMA column block, a last split of 8 values,
# several splits; rows: less than a tile, a tile and one row
@pytest.mark.parametrize("nprobes,values", [(1, 4096), (43, 4160), (2, 8200), (43, 65536), (5, 200000)])
def test_long_rows_match_fp64(ctx, nprobes, values, pairs):
    torch = pytest.importorskip("torch")
    S, lmax = (values // 2 if pairs else values), 3
    ds = ctx.fibonacci(S)
    d, w = O.dirs_fibonacci(S)
    B = O.basis_matrix(d.astype(np.float64), w, lmax)
    g = torch.Generator().manual_seed(nprobes + values)
    rad = torch.rand((nprobes, 3, S), generator=g) * 5
    hi = rad.to(torch.bfloat16)
    held, tile = hi.float(), hi
    if pairs:
        lo = (rad - hi.float()).to(torch.bfloat16)
        held, tile = hi.float() + lo.float(), torch.cat([hi, lo], dim=2).contiguous()
    kind = vlb.DTYPE_BF16_SPLIT if pairs else vlb.DTYPE_BF16
    out = torch.empty((nprobes, vlb.k_of(lmax), 3), dtype=torch.float32, device="cuda")
    dev = tile.cuda().view(torch.int16)
    ctx.project(dev, nprobes, ds, lmax, dtype=kind, out=out)
    ctx.synchronize()
    ref = O.project(held.numpy(), nprobes, S, B)
    # 256 accumulation steps of a split lose up to an ulp each of a growing sum
    # (256 x 2^-24 = 1.5e-5), the hi/lo basis and the dropped low products 2^-18 each
    assert np.linalg.norm(out.cpu().numpy() - ref) / np.linalg.norm(ref) < 2.5e-5
    one = torch.empty_like(out[-1:])
    ctx.project(dev[-1:].clone(), 1, ds, lmax, dtype=kind, out=one)
    ctx.synchronize()
    assert torch.equal(one[0], out[-1])
