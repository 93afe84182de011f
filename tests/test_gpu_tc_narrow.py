"""Batches of few cluster rows: the narrower column groups of both contractions
and the split label draw at the edges of their widths, and the one-launch
Arrange of a batch, against the chains' own forms."""
import numpy as np
import pytest

from tests.test_gpu_plain_tc import _calls
from tests.test_gpu_tc_counts import _counts
from vcfpop_gb300 import _lib as B
from vcfpop_gb300 import structure as S

pytestmark = pytest.mark.gpu
FIELDS = ("Z", "NI", "FREQ", "LL", "LNL")


def _dataset(N, L):
    c = _calls(N, L, N + L)
    Nw = (N + 15) // 16
    pad = np.full((L, Nw * 16), 3, np.uint32)
    pad[:, :N] = c
    packed = np.bitwise_or.reduce(pad.reshape(L, Nw, 16) << (2 * np.arange(16, dtype=np.uint32)), axis=2).astype(np.uint32)
    ds = S.Dataset(np.full(N, 2), np.full(L, 2), np.zeros(N), 1, packed2=packed)
    return ds, c[ds.order()]


def _chains(ctx, ks, **kw):
    return [S.Chain(ctx, S.params(K, 700 + j, **{**dict(admix=0, nadmburnin=0, nburnin=2, nreps=4), **kw}))
            for j, K in enumerate(ks)]


# rows on both sides of every width (64, 96, 128, 192 and two groups), a lone
# chain, individual tiles of one and of many, K above the 16-cluster draw, and
# loci enough for 256-row count tiles
@pytest.mark.parametrize("N,L,ks", [(33, 70, (1,)), (300, 333, (1, 2, 3, 4, 5) * 4), (257, 200, (32, 32)),
                                    (257, 200, (32, 32, 1)), (700, 150, (16,) * 6), (130, 150, (16,) * 6 + (1,)),
                                    (2003, 90, (16,) * 8), (300, 150, (16,) * 8 + (1,)), (300, 150, (10,) * 20),
                                    (300, 150, (10,) * 40), (33, 39_000, (2, 3)), (40, 39_000, (16,) * 12)])
def test_narrow_groups(N, L, ks):
    """Exact counts of the labels, the same sweeps bit for bit from 144-row
    groups where those fit (the FP32 sums keep their order), and the chains'
    own form's first sweep."""
    ds, c = _dataset(N, L)
    ctx = S.Context(ds)
    a = _chains(ctx, ks, form=B.VP_FORM_TC)
    S.run_chains(a, 2)
    one = [{f: ch.get(f) for f in FIELDS} for ch in a]
    splits = S.tc_config(a)["splits"]
    for ch, K in zip(a, ks):
        assert np.array_equal(ch.get("NI").reshape(K, ds.L, 2), _counts(c, ch.get("Z"), K))
    S.finish(a)
    rows = sum(ks)
    if (rows + 191) // 192 * 192 % 144 == 0:          # the 144-row groups fit: an independent width
        b = _chains(ctx, ks, form=B.VP_FORM_TC)
        S.tc_configure(b, cols=144, piece=144, splits=splits)
        S.run_chains(b, 2)
        for x, ch in zip(one, b):
            for f in FIELDS:
                assert np.array_equal(x[f], ch.get(f)), f
        for ch in b:
            ch.close()
    # the chains' own form: the first sweep's frequencies are the same draws,
    # its likelihoods differ by the two forms' rounding (1e-5 relative)
    p = _chains(ctx, ks, form=B.VP_FORM_PLAIN)
    t = _chains(ctx, ks, form=B.VP_FORM_TC)
    S.run_chains(t, 1)
    for ch in p:
        S.run_chains([ch], 1)
    for x, y in zip(t, p):
        assert np.array_equal(x.get("FREQ"), y.get("FREQ"))
        if x.p.K > 1:        # one cluster draws no label
            assert np.abs(x.get("LL") - y.get("LL")).max() <= 1e-5 * np.abs(y.get("LL")).max()
        assert (x.get("Z") != y.get("Z")).mean() < 5e-3
    assert B.lib().vp_tc_status(ctx.h) == 0
    ctx.close()


@pytest.mark.parametrize("ks", [(1, 2, 3), (5,) * 3])
def test_arrange_of_a_batch(ks):
    """Results of a batch finished together equal those of the same chains
    arranged one at a time."""
    ds, _ = _dataset(90, 111)
    ctx = S.Context(ds)
    a, b = _chains(ctx, ks, form=B.VP_FORM_TC), _chains(ctx, ks, form=B.VP_FORM_TC)
    S.finish(a)
    S.run_chains(b, 6)
    for ch in b:
        S.finish([ch])
    for x, y in zip(a, b):
        u, v = x.result(True), y.result(True)
        assert u.keys() == v.keys()
        for f in u:
            assert np.array_equal(u[f], v[f]), f
    ctx.close()
