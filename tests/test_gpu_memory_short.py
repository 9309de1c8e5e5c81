"""Bakes with device memory for what they must have and none for what only makes
them faster (probe frontiers): the same bits, no error."""
import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu

PROBES, S = 8192, 1024
# device memory left: the FP32 tile takes 96 MiB and the frontiers 32 MiB, so the
# tile fits only without them; the one-kernel bake needs neither
LEFT = {vlb.PREC_FP32: 112 << 20, vlb.PREC_FUSED: 24 << 20}


@pytest.mark.parametrize("precision", list(LEFT))
def test_bakes_do_without_extra_scratch(precision):
    torch = pytest.importorskip("torch")
    pos, idx, alb = vlb.synth_box_scene(3, 64)
    probes = np.random.default_rng(9).uniform(0, 1, (PROBES, 3)).astype(np.float32)
    got = []
    for short in (False, True):
        c = vlb.Context(0)
        hog = None
        try:
            scene = c.scene(pos, idx, alb)
            p = vlb.bake_params(c.fibonacci(S), lmax=2, precision=precision, sun=vlb.synth_sun(1))
            c.bake(scene, probes[:64], p)  # the kernels are loaded
            if short:
                torch.cuda.empty_cache()
                free = torch.cuda.mem_get_info()[0]
                hog = torch.empty(free - LEFT[precision], dtype=torch.uint8, device="cuda")
            got.append(c.bake(scene, probes, p))
        finally:
            del hog
            torch.cuda.empty_cache()
            c.close()
    assert np.array_equal(got[0], got[1])
