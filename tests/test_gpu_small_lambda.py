"""A small lambda leaves gamma draws of empty clusters below the normal numbers,
and their quotient infinite: the sweeps on the tensor cores then draw the labels
that the FP32 stream draws (nthinning = 1 keeps every sweep on it)."""
import numpy as np
import pytest

from vcfpop_gb300 import structure as S

from .test_gpu_plain_tc import _calls, _chain

pytestmark = pytest.mark.gpu


# few individuals a cluster, so that some clusters have no copy at some loci
@pytest.mark.parametrize("N,L,K", [(30, 300, 20), (24, 700, 12), (40, 140, 32), (12, 2000, 6)])
@pytest.mark.parametrize("lam", [1e-2, 1e-3])
def test_labels(N, L, K, lam):
    c, ctx, ch = _chain(_calls(N, L, N + K), K)
    ch.close()
    runs = []
    for thin in (1, 10):
        ch = S.Chain(ctx, S.params(K, 9, admix=0, nadmburnin=0, nburnin=3, nreps=6, nthinning=thin, **{"lambda": lam}))
        out = []
        for _ in range(7):
            ch.run(1)
            out.append([ch.get(f) for f in ("Z", "NI", "FREQ")])
        runs.append(out)
        ch.close()
    assert any(np.isinf(f).any() for _, _, f in runs[0])
    for a, b in zip(*runs):
        for x, y in zip(a, b):
            assert np.array_equal(x, y, equal_nan=x.dtype.kind == "f")
    ctx.close()


@pytest.mark.parametrize("K", [4, 6])
def test_frequencies_set(K):
    c, ctx, ch = _chain(_calls(600, 8200, K), K)
    f = np.random.default_rng(K).dirichlet([1, 1], (K, 8200)).astype(np.float32)
    f[1, 77, 1] = np.inf
    ch.set("FREQ", f)
    ch.set("M", [1])
    ch.step("LOGLIK")                        # the FP32 stream
    want = ch.get("LL")
    assert not np.isfinite(want).all()
    ch.step("UPDATEQ")
    got = ch.get("LL")
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want))
    f[1, 77, 1] = 0.5
    ch.set("FREQ", f)
    ch.step("UPDATEQ")
    assert np.isfinite(ch.get("LL")).all()
    ch.close()
    ctx.close()
