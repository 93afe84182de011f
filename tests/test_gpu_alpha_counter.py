"""The alpha step of the counter streams against the serial step: without a
location prior it draws from the reference's stream, so the oracle's step must
agree; with one, the formulas restated in float64 on the same Philox draws."""
import numpy as np
import pytest
from scipy.special import gammaln

from vcfpop_gb300 import _lib as B
from vcfpop_gb300 import structure as S
from vcfpop_gb300 import synth

from . import orc
from .test_gpu_admix_packed import _philox

pytestmark = pytest.mark.gpu


# odd and even K (a pair of proposals shares its two draws), both sides of the
# 32 clusters of the tabulated step; a wide walk, so that proposals out of
# bounds, acceptances with and without a uniform and rejections all occur
@pytest.mark.parametrize("K", [1, 2, 3, 8, 11, 32, 33, 64])
@pytest.mark.parametrize("diffalpha", [0, 1])
@pytest.mark.parametrize("uniformalpha", [0, 1])
def test_alpha(K, diffalpha, uniformalpha):
    N = 14
    d = synth.fmodel(K, N, 40, 2, 0.1, 0.05, admix_alpha=0.5)
    kw = dict(admix=1, diffalpha=diffalpha, uniformalpha=uniformalpha, stdalpha=0.6, maxalpha=2.5, nburnin=100, nreps=100)
    od = orc.Data(d)
    oc = orc.Chain(od, orc.params(K, 4321 + K, **kw))
    oc.init()
    ctx = S.Context(S.Dataset.from_synth(d))
    ch = S.Chain(ctx, S.params(K, 4321 + K, **kw))
    rng = np.random.default_rng(10 * K + diffalpha)
    stayed = moved = 0
    for m in range(24):
        Q = rng.dirichlet(np.full(K, 0.7), N).astype(np.float32)
        a = rng.uniform(0.1, 2.4, K) if diffalpha else np.full(K, rng.uniform(0.1, 2.4))
        for x in (oc, ch):
            x.set("Q", Q)
            x.set("ALPHA", a)
        oc.m = m
        ch.set("M", [m])
        oc.step("update_alpha")
        ch.step("ALPHA")
        got, want = ch.get("ALPHA"), oc.get("ALPHA")
        assert np.allclose(got, want, rtol=1e-12, atol=0), m
        stayed += int((want == a).sum())
        moved += int((want != a).sum())
    assert stayed and moved
    ch.close()
    ctx.close()


def _words(seed, m, b, c):
    return _philox([np.full(2, 9 | (m << 4)), np.full(2, b), np.full(2, c), np.arange(2)], seed).T.reshape(-1)


def _normal_uniform(seed, m, b, c):
    w = [int(x) for x in _words(seed, m, b, c)]
    u = [((((w[2 * j] << 32) | w[2 * j + 1]) >> 11) + 1.0) * 2.0 ** -53 for j in range(3)]
    return np.sqrt(-2 * np.log(u[0])) * np.cos(np.pi * ((2 * u[1]) % 2)), u[2]


@pytest.mark.parametrize("K,sizes", [(1, (9, 5)), (2, (1, 7, 12)), (8, (30, 3, 11, 25)), (33, (6, 18))])
def test_alpha_with_location_prior(K, sizes):
    N, n_loc = sum(sizes), len(sizes)
    pop = np.repeat(np.arange(n_loc), sizes)
    d = synth.fmodel(K, N, 40, 2, 0.1, 0.05, admix_alpha=0.5, loc_ids=pop, loc_alpha=1.0)
    ctx = S.Context(S.Dataset.from_synth(d, n_pop=n_loc))
    seed, std, mx = 987 + K, 0.5, 2.5
    ch = S.Chain(ctx, S.params(K, seed, admix=1, locpriori=1, stdalpha=std, maxalpha=mx, nburnin=100, nreps=100))
    pop = np.asarray(d["pop"])
    rng = np.random.default_rng(K)
    stayed = moved = 0
    for m in range(12):
        Q = rng.dirichlet(np.full(K, 0.7), N).astype(np.float32)
        alpha, loc = rng.uniform(0.1, 2.4, K), rng.uniform(0.1, 2.4, (n_loc, K))
        r, total = rng.uniform(0.3, 3), rng.uniform(0.5, 1.5, n_loc) * loc.sum(1)
        ch.set("M", [m])
        ch.set("Q", Q)
        ch.set("ALPHA", alpha)
        ch.set("LOCP", np.concatenate([[r], np.full(K, 1 / K), np.full(n_loc * K, 1 / K), loc.reshape(-1), total]))
        ch.step("ALPHA")
        a0, l0 = alpha.copy(), loc.copy()
        for k in range(K):
            n, u = _normal_uniform(seed, m, 0xFFFFFFFF, 2 + k)
            am = alpha[k] + std * n
            if 0 < am < mx:
                g = am - alpha[k]
                lr = n_loc * (g * r * np.log(r) + gammaln(r * alpha[k]) - gammaln(r * am)) + r * g * np.log(loc[:, k]).sum()
                if lr >= -1e-10 or u < np.exp(lr):
                    alpha[k] = am
        if m % 10 == 0:
            total = loc.sum(1)
        for s in range(n_loc):
            lnq = np.log(Q[pop == s].astype(np.float64)).sum(0)
            for k in range(K):
                n, u = _normal_uniform(seed, m, s, 2 + k)
                ao, am = loc[s, k], loc[s, k] + std * n
                if 0 < am < mx:
                    g = am - ao
                    lr = ((r * alpha[k] - 1) * np.log(am / ao) - g * r + g * lnq[k] +
                          sizes[s] * (gammaln(total[s] + g) - gammaln(total[s]) + gammaln(ao) - gammaln(am)))
                    if lr >= -1e-10 or u < np.exp(lr):
                        loc[s, k] = am
                        total[s] += g
        assert np.allclose(ch.get("ALPHA"), alpha, rtol=1e-9, atol=0), m
        v = ch.get("LOCP")[1 + K + n_loc * K:]
        assert np.allclose(v[:n_loc * K].reshape(n_loc, K), loc, rtol=1e-9, atol=0), m
        assert np.allclose(v[n_loc * K:], total, rtol=1e-9, atol=0), m
        stayed += int((alpha == a0).sum() + (loc == l0).sum())
        moved += int((alpha != a0).sum() + (loc != l0).sum())
    assert stayed and moved
    ch.close()
    ctx.close()
