"""Per-copy label draws on 2-bit data against the byte layout's kernel.

The same calls as 2-bit codes and as allele bytes run through different label
kernels, with the same Philox streams and the same FP32 operations per copy, so
labels, counts and everything drawn from them are equal bit for bit."""
import numpy as np
import pytest

from vcfpop_gb300 import structure as S
from vcfpop_gb300 import synth

pytestmark = pytest.mark.gpu


def _run(d, packed, K, sweeps, **kw):
    ds = S.Dataset.from_synth(d, packed=packed)
    ctx = S.Context(ds)
    c = S.Chain(ctx, S.params(K, 77 + K, nburnin=2, nreps=max(1, sweeps - 2), nthinning=2, writelnl=1, **kw))
    c.run(sweeps)
    out = {f: c.get(f) for f in ("NI", "MI", "Q", "FREQ", "ALPHA")}
    out["lnl"] = c.result()["lnl"]
    c.close()
    ctx.close()
    return out


def _same(a, b):
    for f in ("NI", "MI", "Q", "FREQ", "ALPHA"):
        assert np.array_equal(a[f], b[f]), f
    # the copies' ln(sum q p) are added in another grouping (FP32 Kahan sums per
    # lane and range, FP64 across): within a few FP32 ulps of a lane's sum
    assert np.allclose(a["lnl"], b["lnl"], rtol=1e-7, atol=0)


# sizes around the warp, the CTA and the 16-locus slice
@pytest.mark.parametrize("N,L", [(16, 17), (31, 16), (33, 40), (128, 15), (129, 130), (257, 33), (1025, 64), (1300, 47)])
@pytest.mark.parametrize("K", [1, 4, 5])
def test_sizes(N, L, K):
    d = synth.fmodel(N + L, N, L, 3, 0.1, 0.1, admix_alpha=0.5)
    _same(_run(d, True, K, 4, admix=1), _run(d, False, K, 4, admix=1))


# every compiled cluster count, and the padded one at both ends
@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 16, 17])
def test_clusters(K):
    d = synth.fmodel(K, 150, 210, 4, 0.1, 0.05, admix_alpha=0.5)
    _same(_run(d, True, K, 4, admix=1), _run(d, False, K, 4, admix=1))


def test_admixture_burn_in():
    d = synth.fmodel(9, 90, 100, 3, 0.1, 0.05)
    kw = dict(admix=0, nadmburnin=3)
    _same(_run(d, True, 3, 3, **kw), _run(d, False, 3, 3, **kw))
