"""cullst on the GPU (through the C ABI) against the oracle: keep masks and
culled offsets bit-exact, smoothed offsets and sigmas within float tolerance."""
import numpy as np
import pytest

from oracle import oracle
from specklesource_b200 import abi
from specklesource_b200.synth import offsets_field

pytestmark = pytest.mark.gpu

LARGE = np.float32(-2e9)


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


def _same(a, b):
    return np.array_equal(a, b, equal_nan=True)


def _check(g, o, keys_exact=("offR", "offA", "type")):
    for k in keys_exact:
        assert _same(g[k], o[k]), f"{k} differs at {np.argwhere(~((g[k] == o[k]) | (np.isnan(g[k]) & np.isnan(o[k]))))[:5]}"
    for k in ("offRS", "offAS"):
        vg, vo = g[k] > -1.9e9, o[k] > -1.9e9
        assert np.array_equal(vg, vo), f"{k} keep mask differs"
        assert np.allclose(g[k][vo], o[k][vo], rtol=1e-6, atol=1e-6)
    for k in ("sigmaR", "sigmaA"):
        vg, vo = g[k] > -1.9e9, o[k] > -1.9e9
        assert np.array_equal(vg, vo), f"{k} validity differs"
        assert np.allclose(g[k][vo], o[k][vo], rtol=2e-3, atol=1e-5)


@pytest.mark.parametrize("kw", [
    dict(),                                                          # cullst defaults
    dict(bR=5, bA=5, nGood=12, sR=3, sA=3, islandThresh=10),          # 5x5 median, 3x3 smoothing, islands
    dict(bR=7, bA=3, nGood=5, maxA=0.5, maxR=0.5, sR=4, sA=1, corrThresh=0.2, islandThresh=4, connectivity=4),
    dict(bR=13, bA=13, nGood=40, islandThresh=6),  # box above 128 values: the row-wavefront median kernel
])
def test_cull_pipeline_matches_oracle(ctx, kw):
    nA, nR = 150, 230
    offR, offA, corr, mt = offsets_field(nA, nR, 7)
    p = abi.CullParams(nR=nR, nA=nA, **kw)
    g = ctx.cull(p, offR, offA, corr, mt)
    o = oracle.cull(p, offR, offA, corr, mt)
    _check(g, o)
    assert g["nCulled"] == o["nCulled"]
    if p.islandThresh > 0:
        assert (g["nIslands"], g["nIslandPoints"]) == (o["nIslands"], o["nIslandPoints"])


def test_cull_single_passes(ctx):
    nA, nR = 80, 120
    offR, offA, corr, mt = offsets_field(nA, nR, 8)
    p = abi.CullParams(nR=nR, nA=nA)
    g = ctx.cull(p, offR, offA, corr, mt, passes=("st",))
    o = oracle.cull(p, offR, offA, corr, mt, passes=("st",))
    assert _same(g["offR"], o["offR"]) and _same(g["offA"], o["offA"])
    g = ctx.cull(p, offR, offA, corr, mt, passes=("st", "stats", "smooth", "islands"))
    o = oracle.cull(p, offR, offA, corr, mt, passes=("st", "stats", "smooth", "islands"))
    _check(g, o)


def test_cull_mask_single_mt_and_sim(ctx):
    nA, nR = 90, 140
    offR, offA, corr, mt = offsets_field(nA, nR, 9)
    rng = np.random.default_rng(3)
    mask = rng.integers(0, 8, (nA, nR)).astype(np.uint8)
    simR = (0.5 * rng.standard_normal((nA, nR))).astype(np.float32)
    simA = (0.5 * rng.standard_normal((nA, nR))).astype(np.float32)
    p = abi.CullParams(nR=nR, nA=nA, singleMT=2, useSim=1, islandThresh=6)
    g = ctx.cull(p, offR, offA, corr, mt, mask=mask, simR=simR, simA=simA)
    o = oracle.cull(p, offR, offA, corr, mt, mask=mask, simR=simR, simA=simA)
    _check(g, o)


@pytest.mark.parametrize("nA,nR,kw", [
    (1, 1, dict(bR=1, bA=1, nGood=0)),
    (7, 5, dict(bR=9, bA=9, nGood=4)),                         # box larger than the grid
    (33, 65, dict(bR=3, bA=9, nGood=2, maxR=0.05, maxA=2.0)),   # one row and column past a block
    (64, 31, dict(bR=11, bA=11, nGood=0, maxR=0.0, maxA=0.0)),  # 121 values; everything off the median goes
    (70, 90, dict(bR=2, bA=4, nGood=1, nCullPasses=1)),
    (200, 300, dict(bR=5, bA=5, nGood=10, maxR=0.06, maxA=0.06, nCullPasses=5)),  # long chains of culls
])
def test_cull_fixpoint_edges(ctx, nA, nR, kw):
    """Decisions by counting against medians: grids and boxes at the block
    edges, limits of zero, values that differ by the limit, infinities."""
    rng = np.random.default_rng(nA * nR)
    offR = np.round(rng.normal(0, 0.1, (nA, nR)) * 20).astype(np.float32) / np.float32(20)
    offA = rng.normal(0, 0.1, (nA, nR)).astype(np.float32)
    for v in (np.nan, np.inf, -2e9):
        offR[rng.random((nA, nR)) < 0.02] = v
    offA[rng.random((nA, nR)) < 0.01] = np.inf
    corr = np.ones((nA, nR), np.float32)
    mt = np.ones((nA, nR), np.uint8)
    p = abi.CullParams(nR=nR, nA=nA, **kw)
    g = ctx.cull(p, offR, offA, corr, mt, passes=("st",))
    o = oracle.cull(p, offR, offA, corr, mt, passes=("st",))
    assert _same(g["offR"], o["offR"]) and _same(g["offA"], o["offA"]) and g["nCulled"] == o["nCulled"]


@pytest.mark.parametrize("kw,sigma,holes", [
    (dict(bR=9, bA=9, nGood=60, maxR=0.5, maxA=0.5), 0.01, 0.0),   # culls eat their way in from the edges
    (dict(bR=5, bA=5, nGood=18, maxR=0.5, maxA=0.5), 0.01, 0.1),
    (dict(bR=5, bA=5, nGood=12, maxR=0.05, maxA=0.05), 0.1, 0.0),
])
def test_cull_long_revisit_lists(ctx, kw, sigma, holes):
    """Revisit lists too long for one cluster: steps over the whole chip (two
    launches each), the cluster for the short lists after them."""
    nA, nR = 410, 530
    rng = np.random.default_rng(2)
    offR, offA = (rng.normal(0, sigma, (nA, nR)).astype(np.float32) for _ in range(2))
    offR[rng.random((nA, nR)) < holes] = -2e9
    corr = np.ones((nA, nR), np.float32)
    mt = np.ones((nA, nR), np.uint8)
    for passes in (1, 3):
        p = abi.CullParams(nR=nR, nA=nA, nCullPasses=passes, sR=1, sA=1, **kw)
        g = ctx.cull(p, offR, offA, corr, mt)
        assert ctx.launch_count() > 40
        o = oracle.cull(p, offR, offA, corr, mt)
        _check(g, o)
        assert g["nCulled"] == o["nCulled"]


def test_cull_many_passes():
    """Passes enqueued in groups: any number of them on one workspace."""
    from specklesource_b200 import runtime
    offR, offA, corr, mt = offsets_field(40, 60, 3)
    held = []
    for passes in (1, 16, 17, 1000):
        with runtime.Context(0) as c:
            p = abi.CullParams(nR=60, nA=40, bR=5, bA=5, nGood=9, maxR=0.2, maxA=0.2, nCullPasses=passes)
            g, o = c.cull(p, offR, offA, corr, mt), oracle.cull(p, offR, offA, corr, mt)
            _check(g, o)
            assert g["nCulled"] == o["nCulled"]
            held.append(c.device_bytes())
    assert held[3] == held[2] == held[1]


def test_cull_large_grid_keep_mask(ctx):
    """Keep masks on a 700 x 993 grid (rows of the large strack workload's grid)."""
    nA, nR = 700, 993
    offR, offA, corr, mt = offsets_field(nA, nR, 10)
    p = abi.CullParams(nR=nR, nA=nA, bR=5, bA=5, nGood=12, sR=3, sA=3, islandThresh=10, nCullPasses=3)
    g = ctx.cull(p, offR, offA, corr, mt)
    t = ctx.timing()
    o = oracle.cull(p, offR, offA, corr, mt)
    _check(g, o)
    print("cull 700x993:", t)
    assert o["nIslands"] > 0


def test_cull_tall_grid(ctx):
    """More than 524,280 rows, where tiles of 8 rows number more than 65,535."""
    nA, nR = 524281 + 300, 2
    rng = np.random.default_rng(5)
    offR = rng.normal(0, 0.3, (nA, nR)).astype(np.float32)
    offA = rng.normal(0, 0.3, (nA, nR)).astype(np.float32)
    offR[rng.random((nA, nR)) < 0.05] = -2e9
    corr = np.ones((nA, nR), np.float32)
    mt = np.ones((nA, nR), np.uint8)
    p = abi.CullParams(nR=nR, nA=nA, bR=3, bA=5, nGood=3, sR=1, sA=3, maxR=0.5, maxA=0.5)
    g, o = ctx.cull(p, offR, offA, corr, mt), oracle.cull(p, offR, offA, corr, mt)
    assert o["nCulled"] > 0 and (o["offR"] > -1.9e9).sum() > nA / 2
    _check(g, o)
    assert g["nCulled"] == o["nCulled"]


# ---------------------------------------------------------------- cullls

SLOW, NODATA_BIT = 0x10, 0x40  # stand-ins for lstrack.h's SLOWVEL / NODATATOUSE


def _ls_inputs(nA, nR, seed):
    X, Y, _, mt = offsets_field(nA, nR, seed)
    rng = np.random.default_rng(seed + 100)
    yy, xx = np.mgrid[0:nA, 0:nR]
    t = np.where((xx - nR / 3) ** 2 + (yy - nA / 2) ** 2 < (nA / 3) ** 2, SLOW, 0)  # a slow-moving disc
    t = t | np.where(rng.random((nA, nR)) < 0.05, NODATA_BIT, 0) | (mt & 3)
    return X, Y, t.astype(np.uint8)


def _check_ls(g, o):
    for k in ("X", "Y"):
        assert _same(g[k], o[k]), f"{k} differs at {np.argwhere(~((g[k] == o[k]) | (np.isnan(g[k]) & np.isnan(o[k]))))[:5]}"
    for k in ("XS", "YS"):
        vg, vo = g[k] > -1.9e9, o[k] > -1.9e9
        assert np.array_equal(vg, vo), f"{k} keep mask differs"
        assert np.allclose(g[k][vo], o[k][vo], rtol=1e-6, atol=1e-6)
    for k in ("sigmaX", "sigmaY"):
        vg, vo = g[k] > -1.9e9, o[k] > -1.9e9
        assert np.array_equal(vg, vo), f"{k} validity differs"
        assert np.allclose(g[k][vo], o[k][vo], rtol=2e-3, atol=1e-5)
    for k in ("nAttempt", "nMatch", "nCulled", "nIslands", "nIslandPoints"):
        assert g[k] == o[k], k


@pytest.mark.parametrize("kw", [
    dict(islandThresh=6),                                                   # cullls defaults, islands
    dict(boxSize=5, nGood=8, sX=1, sY=5, noDataLimit=-3.0, connectivity=4, islandThresh=3),
    dict(boxSize=13, nGood=40, deltaT=24.0, dx=30.0, dy=30.0),              # box above 128 values: the wavefront kernel
])
def test_cullls_matches_oracle(ctx, kw):
    nA, nR = 150, 230
    X, Y, t = _ls_inputs(nA, nR, 11)
    base = dict(nx=nR, ny=nA, deltaT=365.0, dx=15.0, dy=15.0, nOver=10.0, slowVelMask=SLOW, noDataMask=NODATA_BIT)
    base.update(kw)
    p = abi.CullLSParams(**base)
    g = ctx.cullls(p, X, Y, t)
    o = oracle.cullls(p, X, Y, t)
    _check_ls(g, o)
    assert o["nCulled"] > 0 and o["nMatch"] > o["nCulled"]


def test_cullls_large_grid(ctx):
    nA, nR = 700, 993
    X, Y, t = _ls_inputs(nA, nR, 12)
    p = abi.CullLSParams(nx=nR, ny=nA, deltaT=48.0, dx=15.0, dy=15.0, nOver=10.0, slowVelMask=SLOW,
                         noDataMask=NODATA_BIT, islandThresh=10)
    g = ctx.cullls(p, X, Y, t)
    o = oracle.cullls(p, X, Y, t)
    _check_ls(g, o)
    assert o["nIslands"] > 0


def _chains(first, second, nR=1500):
    """Rows whose points go one after the other, each because its left
    neighbour went: with nGood=2 and a 3 x 3 box a row alone loses its end
    point, then the next.  first: from the first pass on.  second: the end of
    the row stays until the outlier below it has gone in the first pass.  The
    rows at the bottom keep points for the later passes."""
    rng = np.random.default_rng(11)
    offR = rng.normal(0, 0.01, (9, nR)).astype(np.float32)
    offA = rng.normal(0, 0.01, (9, nR)).astype(np.float32)
    offR[6:][rng.random((3, nR)) < 0.2] += np.float32(3)
    for row in range(6):
        if not (row == 0 and first or row in (2, 3) and second):
            offR[row] = offA[row] = -2e9
    offR[3, 1:] = offA[3, 1:] = -2e9
    if second:
        offR[3, 0] = 100
    return offR, offA


@pytest.mark.parametrize("first,second", [(True, False), (False, True), (True, True)])
def test_cull_passes_that_do_not_converge(ctx, first, second):
    """Chains longer than the fixpoint's steps: the row-wavefront kernel does
    such a pass and the rest follow, for cullst and for cullls's limits."""
    offR, offA = _chains(first, second)
    nA, nR = offR.shape
    corr = np.ones((nA, nR), np.float32)
    mt = np.ones((nA, nR), np.uint8)
    for passes in (1, 2, 3, 5):
        p = abi.CullParams(nR=nR, nA=nA, bR=3, bA=3, nGood=2, maxR=0.5, maxA=0.5, sR=2, sA=2, nCullPasses=passes)
        g, o = ctx.cull(p, offR, offA, corr, mt), oracle.cull(p, offR, offA, corr, mt)
        _check(g, o)
        assert g["nCulled"] == o["nCulled"]
        if passes == 5:
            assert not first or (o["offR"][0] < -1e9).all()
            assert not second or (o["offR"][2] < -1e9).all()
        assert (o["offR"][6:] > -1e9).any()
        t = np.full((nA, nR), SLOW, np.uint8)
        t[:, ::3] = 1
        q = abi.CullLSParams(nx=nR, ny=nA, boxSize=3, nGood=2, maxX=0.5, maxY=0.5, nCullPasses=passes, deltaT=16.0,
                             dx=15.0, dy=15.0, nOver=10.0, slowVelMask=SLOW, noDataMask=NODATA_BIT)
        _check_ls(ctx.cullls(q, offR, offA, t), oracle.cullls(q, offR, offA, t))
    # the wavefront kernel was reached: without naps its waits run out
    assert ctx.lib.sb_set_wait_limit(ctx.h, 0) == abi.SB_OK
    try:
        with pytest.raises(Exception, match="timed out"):
            ctx.cull(p, offR, offA, corr, mt)
    finally:
        assert ctx.lib.sb_set_wait_limit(ctx.h, 1 << 26) == abi.SB_OK


def test_wavefront_wait_times_out_and_context_stays_usable(ctx):
    """The row-wavefront median kernel (13 x 13 box) waits for the previous
    grid row with a bounded wait.  With a limit of 0 naps the first unmet
    check gives up: the call fails with SB_ERR_TIMEOUT (nothing hangs), and the
    same context then culls the grid bit-exactly with the default limit."""
    from specklesource_b200.runtime import SpeckleError
    nA, nR = 150, 230
    offR, offA, corr, mt = offsets_field(nA, nR, 7)
    p = abi.CullParams(nR=nR, nA=nA, bR=13, bA=13, nGood=40, islandThresh=6)
    assert ctx.lib.sb_set_wait_limit(ctx.h, -1) == abi.SB_ERR_ARG
    assert ctx.lib.sb_set_wait_limit(ctx.h, 0) == abi.SB_OK
    try:
        with pytest.raises(SpeckleError, match="timed out") as ei:
            ctx.cull(p, offR, offA, corr, mt)
        assert ei.value.code == abi.SB_ERR_TIMEOUT
    finally:
        assert ctx.lib.sb_set_wait_limit(ctx.h, 1 << 26) == abi.SB_OK
    g = ctx.cull(p, offR, offA, corr, mt)
    o = oracle.cull(p, offR, offA, corr, mt)
    _check(g, o)
    assert g["nCulled"] == o["nCulled"]
