"""Calls made while the context holds probe frontiers of an earlier bake and little
device memory is free: the frontiers are given back, and the call returns what it
returns with memory to spare."""
import contextlib

import numpy as np
import pytest

import vlb

pytestmark = pytest.mark.gpu

# 65,536 probes: 268 MB of frontiers; 2056 directions make rows of 4112 BF16 values,
# two splits, whose sums take 25 MB at lmax 3
PROBES, S = 65536, 2056
# a bake that holds all a bake of those takes but split sums: its rows are whole
WARM_PROBES, WARM_S = 66200, 2040


@contextlib.contextmanager
def little_memory(torch, left):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hog
        torch.cuda.empty_cache()


def setup(c):
    pos, idx, alb = vlb.synth_box_scene(3, 64)
    probes = np.random.default_rng(9).uniform(0, 1, (WARM_PROBES, 3)).astype(np.float32)
    return c.scene(pos, idx, alb), probes[:PROBES], c.fibonacci(S), (probes, c.fibonacci(WARM_S))


def params(ds, precision):
    return vlb.bake_params(ds, lmax=3, precision=precision, sun=vlb.synth_sun(1))


def test_split_projection_of_a_bake_keeps_its_bits():
    torch = pytest.importorskip("torch")
    got = []
    for short in (False, True):
        c = vlb.Context(0)
        try:
            scene, probes, ds, warm = setup(c)
            c.bake(scene, warm[0], params(warm[1], vlb.PREC_FP32))
            c.bake(scene, probes[:64], params(ds, vlb.PREC_MIXED))
            with little_memory(torch, 12 << 20) if short else contextlib.nullcontext():
                got.append(c.bake(scene, probes, params(ds, vlb.PREC_MIXED)))
        finally:
            c.close()
    assert np.array_equal(got[0], got[1])


def test_split_projection_of_a_batch_keeps_its_bits():
    """With memory for the sums or not, and in the calls after it (the second of a shape is captured)."""
    torch = pytest.importorskip("torch")
    got = []
    for short in (False, True):
        c = vlb.Context(0)
        try:
            scene, probes, ds, warm = setup(c)
            mixed = params(ds, vlb.PREC_MIXED)
            c.bake_batch([(scene, warm[0], None)], params(warm[1], vlb.PREC_FP32))
            c.bake_batch([(scene, probes[:64], None)], mixed)
            with little_memory(torch, 12 << 20) if short else contextlib.nullcontext():
                got.append(c.bake_batch([(scene, probes, None)], mixed)[0])
            for _ in range(3):
                got.append(c.bake_batch([(scene, probes, None)], mixed)[0])
        finally:
            c.close()
    for other in got[1:]:
        assert np.array_equal(got[0], other)


def test_batch_that_ran_out_of_memory_runs_later():
    """The call after a batch that failed for want of its split sums is a first call: nothing
    of it is captured, and the ones after it are."""
    torch = pytest.importorskip("torch")
    c = vlb.Context(0)
    try:
        # few triangles and many jobs: no frontiers and no light maps that could be given back
        scene = c.scene(*vlb.synth_box_scene(3, 2))
        warm = np.random.default_rng(9).uniform(0, 1, (WARM_PROBES, 3)).astype(np.float32)
        probes = warm[:PROBES]
        jobs = [(scene, part, None) for part in np.array_split(probes, 600)]
        ds = c.fibonacci(S)
        mixed = params(ds, vlb.PREC_MIXED)
        c.bake_batch([(scene, part, None) for part in np.array_split(warm, 600)],
                     params(c.fibonacci(WARM_S), vlb.PREC_FP32))
        c.bake_batch([(scene, probes[:64], None)], mixed)
        with little_memory(torch, 12 << 20):
            with pytest.raises(vlb.VlbError) as e:
                c.bake_batch(jobs, mixed)
            assert e.value.status == vlb.ERR_OOM
        got = [np.concatenate(c.bake_batch(jobs, mixed)) for _ in range(3)]
        assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
        assert np.array_equal(got[0], c.bake(scene, probes, mixed))
    finally:
        c.close()


@pytest.mark.parametrize("what", ["scene", "directions", "sky", "cubemap tables"])
def test_objects_are_made(what):
    torch = pytest.importorskip("torch")
    c = vlb.Context(0)
    try:
        scene, probes, ds, _ = setup(c)
        few = c.fibonacci(64)
        big = vlb.synth_box_scene(5, 6000)
        cube = vlb.synth_cubemap(4, 512)
        texels = torch.from_numpy(vlb.synth_cubemap(6, 256)).cuda()
        out = torch.zeros((16, 3), device="cuda")
        c.bake(scene, probes, params(few, vlb.PREC_FP32))
        c.skybox_sh(vlb.synth_cubemap(6, 64), vlb.SKY_CUBEMAP, 64, 64, 3)  # the kernels are loaded
        with little_memory(torch, 6 << 20):
            if what == "scene":
                assert c.scene(*big).device_bytes > 8 << 20
            elif what == "directions":
                c.fibonacci(1 << 19)
            elif what == "sky":
                c.sky(cube, 512)
            else:
                c.skybox_sh(texels, vlb.SKY_CUBEMAP, 256, 256, 3, out=out)
                c.synchronize()
                assert torch.isfinite(out).all() and out[0, 0] != 0
    finally:
        c.close()


def test_service_keeps_frontiers_within_its_budget():
    """Frontiers of a large batch do not stay beside kept hits that use the budget up."""
    torch = pytest.importorskip("torch")
    c = vlb.Context(0)
    try:
        pos, idx, alb = vlb.synth_box_scene(3, 64)
        scene, ds = c.scene(pos, idx, alb), c.fibonacci(64)
        n, m, budget = 1 << 18, 1 << 15, 1 << 30
        probes = np.random.default_rng(9).uniform(0, 1, (n, 3)).astype(np.float32)
        p = vlb.bake_params(ds, 2, vlb.PREC_FP32, vlb.synth_sun(1))
        want = c.bake(scene, probes, p)
        c.bake_batch([(scene, probes[:64], None)], p)  # the kernels are loaded
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        svc = vlb.Service(c, budget_bytes=budget, lmax=2, precision=vlb.PREC_FP32, slice_probes=0xFFFFFFFF)
        assert np.array_equal(svc.wait(svc.submit(scene, probes, p))[0], want)  # its lists are cut to fit
        # the radiance tile, outputs and order of the large batch stay: 904 bytes a probe
        must = n * (64 * 12 + 12 + 4 + 16 + 108)
        keep = m * 64 * 8 + m * 12  # a kept set
        for k in range((budget - m * 1024) // keep):
            svc.wait(svc.submit(scene, probes[:m], p, keep_hits=True))
        assert svc.stats()["evictions"] == 0
        used = free - torch.cuda.mem_get_info()[0]
        svc.close()
        assert used < budget + must + (96 << 20)  # the rest: allocation granularity, the stream-ordered pool
    finally:
        c.close()


def test_service_gives_its_frontiers_back():
    """A batch whose radiance tile fits only without the frontiers of the batch before it."""
    torch = pytest.importorskip("torch")
    c = vlb.Context(0)
    try:
        scene, probes, _, _ = setup(c)
        first, second = (vlb.bake_params(c.fibonacci(s), 2, vlb.PREC_FP32, vlb.synth_sun(1)) for s in (64, 128))
        want = c.bake(scene, probes, second)
        svc = vlb.Service(c, lmax=2, precision=vlb.PREC_FP32, slice_probes=0xFFFFFFFF)
        svc.wait(svc.submit(scene, probes, first))
        with little_memory(torch, 24 << 20):  # the tile grows from 50 to 101 MB
            assert np.array_equal(svc.wait(svc.submit(scene, probes, second))[0], want)
        svc.close()
    finally:
        c.close()
