"""Batched strack (sb_strack_batch) against one sb_strack call per pair.

A batch groups its pairs by window size and runs every stage once per group
over all the group's points, with the images of all pairs in two atlases; per
point the arithmetic is sb_strack's, so each pair's grids and statistics must
equal its own sb_strack result bit for bit -- with pairs of different sizes,
windows, grids, initial shifts (polynomial and offset grid with holes), masks,
host and device images, and in both transform forms.
"""
import numpy as np
import pytest

from specklesource_b200 import abi, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from specklesource_b200 import build, runtime
    build.build()
    c = runtime.Context(0)
    yield c
    c.close()


def _pairs():
    rng = np.random.default_rng(9)
    cases = []
    for k, (na, nr, W) in enumerate([(512, 768, 32), (700, 512, 64), (640, 1024, 24), (512, 640, 48),
                                      (896, 700, 64), (600, 800, 32), (520, 900, 48), (768, 768, 24),
                                      (1024, 600, 64), (560, 560, 32)]):
        s1, s2 = synth.small_pair(device="cuda", na=na, nr=nr, seed=60 + k)
        step = max(8, W // 2)
        m = W + 8
        kw = dict(rStart=m, aStart=m, deltaR=step, deltaA=step + 4 * (k % 3), wR=W, wA=W, wRa=W, wAa=W)
        kw["nR"] = (nr - 2 * m) // kw["deltaR"] + 1
        kw["nA"] = (na - 2 * m) // kw["deltaA"] + 1
        if k == 3:  # offset-grid initial shift with holes
            g = {"nr": 12, "na": 10, "r0": 0.0, "a0": 0.0, "deltaR": 64.0, "deltaA": 64.0,
                 "dr": np.full((10, 12), 2.0, np.float32), "da": np.full((10, 12), 0.5, np.float32)}
            g["dr"][2:4, 3:6] = -2e9
            kw.update(polyShift=0, initOffsets=g)
        if k == 5:  # mask
            mk = (rng.random((20, 30)) > 0.25).astype(np.uint8)
            kw["mask"] = {"r0": 0, "a0": 0, "nr": 30, "na": 20, "nrl": 32, "nal": 32, "mask": mk}
        if k == 7:
            kw.update(rShiftPoly=(1.0, 0.001, 0.0), aShiftPoly=(-0.5, 0.0, 0.0005))
        p = abi.TrackParams(**kw)
        # alternate host and device images
        a, b = (s1, s2) if k % 2 else (synth.to_numpy(s1), synth.to_numpy(s2))
        cases.append((p, a, b))
    return cases


@pytest.mark.parametrize("form", [abi.SB_FORM_FP32, abi.SB_FORM_SPLIT_BF16])
def test_batch_equals_single_calls(ctx, form):
    cases = _pairs()
    ctx.set_form(form)
    try:
        single = [ctx.strack(p, a, b) for p, a, b in cases]
        batch = ctx.strack_batch([c[0] for c in cases], [c[1] for c in cases], [c[2] for c in cases])
    finally:
        ctx.set_form(abi.SB_FORM_FP32)
    for k, (s, t) in enumerate(zip(single, batch)):
        for key in ("offR", "offA", "corr", "azd", "type"):
            assert np.array_equal(s[key], t[key], equal_nan=True), (k, key)
        assert s["stats"] == t["stats"], k
        assert (t["type"] > 0).mean() > 0.5, k
    assert ctx.launch_count() < 10 * 14  # stages run per window group, not per pair


def test_batch_rejects_mixed_flags(ctx):
    from specklesource_b200.runtime import SpeckleError
    cases = _pairs()[:2]
    cases[1][0].hanningFlag = 0
    with pytest.raises(SpeckleError, match="same for every pair"):
        ctx.strack_batch([c[0] for c in cases], [c[1] for c in cases], [c[2] for c in cases])


def test_batch_more_buckets_than_partition_keys(ctx):
    """35 (complex, amplitude) window buckets, above the 32 keys of one
    ordered partition: the batch plans every pair on the host and must still
    equal each pair's own call."""
    cases = []
    k = 0
    for W in (16, 24, 32, 48, 64):
        for WA in (16, 24, 32, 48, 64, 96, 128):
            s1, s2 = synth.small_pair(device="cuda", na=400, nr=400, seed=200 + k)
            p = abi.TrackParams(rStart=80, aStart=80, deltaR=24, deltaA=24, nR=11, nA=11, wR=W, wA=W, wRa=WA,
                                wAa=WA, maxTries=1)
            cases.append((p, s1, s2))
            k += 1
    single = [ctx.strack(p, a, b) for p, a, b in cases]
    batch = ctx.strack_batch([c[0] for c in cases], [c[1] for c in cases], [c[2] for c in cases])
    for k, (s, t) in enumerate(zip(single, batch)):
        for key in ("offR", "offA", "corr", "azd", "type"):
            sv = s[key].cpu().numpy() if hasattr(s[key], "cpu") else s[key]
            tv = t[key].cpu().numpy() if hasattr(t[key], "cpu") else t[key]
            assert np.array_equal(sv, tv, equal_nan=True), (k, key)
        assert s["stats"] == t["stats"], k


@pytest.mark.parametrize("nR,nA,keep", [(1, 1, 1.0), (1, 1, 0.0), (7, 5, 0.2), (64, 37, 1.0), (64, 37, 0.0),
                                        (64, 37, 0.02), (400, 390, 0.7)])
def test_list_length_on_the_device(ctx, nR, nA, keep):
    """One sb_strack call launches its complex stage for the whole grid and
    reads the list's length on the device; the batch counts on the host.  Grids
    of one tile and of more than four warps of tiles, lists that are empty,
    shorter than the launch, and full."""
    na, nr = 448, 512
    s1, s2 = synth.small_pair(device="cuda", na=na, nr=nr, seed=77)
    mk = (np.random.default_rng(3).random((na // 8, nr // 8)) < keep).astype(np.uint8)
    p = abi.TrackParams(rStart=24, aStart=24, nR=nR, nA=nA, wR=16, wA=16, wRa=16, wAa=16, rShiftPoly=(1.0, 0.0, 0.0),
                        mask={"r0": 0, "a0": 0, "nr": nr // 8, "na": na // 8, "nrl": 8, "nal": 8, "mask": mk})
    s = ctx.strack(p, s1, s2)
    t, = ctx.strack_batch([p], [s1], [s2])
    for key in ("offR", "offA", "corr", "azd", "type"):
        assert np.array_equal(s[key], t[key], equal_nan=True), key
    assert s["stats"] == t["stats"]


@pytest.mark.parametrize("int16", [False, True])
def test_device_images_of_any_row_length(ctx, int16):
    """Device images into the atlases: rows of a multiple of 16, 8 and 4 bytes,
    an image that starts between two words of that size, one-row remainders."""
    import torch
    cases = []
    for k, (na, nr, shift) in enumerate([(120, 128, 0), (121, 131, 0), (127, 133, 1), (97, 161, 3)]):
        s = []
        for im in synth.small_pair(device="cuda", na=na, nr=nr, seed=80 + k):
            if int16:
                im = torch.view_as_real(im)
                im = torch.clamp((im * (1000.0 / im.abs().max())).round(), -32767, 32767).to(torch.int16)
            flat = torch.empty(im.numel() + 2 * shift, dtype=im.dtype, device="cuda")
            off = 2 * shift if int16 else shift
            v = flat[off:off + im.numel()].view(im.shape)
            v.copy_(im)
            s.append(v)
        p = abi.TrackParams(rStart=24, aStart=24, deltaR=16, deltaA=16, nR=5, nA=4, wR=16, wA=16, wRa=16, wAa=16)
        cases.append((p, s[0], s[1]))
    single = [ctx.strack(*c) for c in cases]
    batch = ctx.strack_batch([c[0] for c in cases], [c[1] for c in cases], [c[2] for c in cases])
    for k, (s, t) in enumerate(zip(single, batch)):
        for key in ("offR", "offA", "corr", "azd", "type"):
            assert np.array_equal(s[key], t[key], equal_nan=True), (k, key)
        assert s["stats"] == t["stats"]
