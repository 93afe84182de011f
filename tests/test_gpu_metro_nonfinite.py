"""Metropolis log ratios of 2-bit data with frequencies that are not finite or
far out of range: as the byte layout's kernel, which takes every copy's logarithm
of the ratio by itself."""
import numpy as np
import pytest

from vcfpop_gb300 import structure as S
from vcfpop_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, np.nan, 0.0, 1e38, 1e-38])
@pytest.mark.parametrize("K", [1, 3, 13])
def test_ratio(K, value):
    d = synth.fmodel(K, 40, 50, 2, 0.1, 0.1, admix_alpha=0.5)
    out = []
    for packed in (True, False):
        ds = S.Dataset.from_synth(d, packed=packed)
        ctx = S.Context(ds)
        ch = S.Chain(ctx, S.params(K, 5, admix=1, nburnin=50, nreps=50))
        rng = np.random.default_rng(K)
        f = rng.dirichlet([1, 1], (K, ds.L)).astype(np.float32)
        f[:, 7, 0] = value                   # one allele of one locus, in every cluster
        ch.set("M", [10])                    # a Metropolis sweep
        ch.set("FREQ", f)
        ch.step("UPDATEQ")
        out.append(ch.get("METRO"))
        L = ds.L
        ch.close()
        ctx.close()
    a, b = out
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.array_equal(a[np.isinf(a)], b[np.isinf(b)])
    ok = np.isfinite(a)
    # FP32 sums of the byte layout over 64 copies round at up to 64 x 5 x 2^-24 a copy
    assert np.allclose(a[ok], b[ok], rtol=0, atol=2 * 64 * 5 * 2.0 ** -24 * L)
