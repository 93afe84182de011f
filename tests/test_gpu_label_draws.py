"""The per-copy label draws of the counter streams, restated in numpy: one Philox
stream per (individual, slice of 16 loci), vmax draws a locus, prefix sums by FP32
fused multiply-adds, the first cluster whose cumulative weight exceeds the
uniform times the total."""
import numpy as np
import pytest

from vcfpop_gb300 import structure as S
from vcfpop_gb300 import synth

from .test_gpu_admix_packed import _philox

pytestmark = pytest.mark.gpu

F = np.float32
MIN = 1e-10


def _fma(a, b, c):
    # the product of two FP32 values is exact in FP64; the sum rounds there and
    # then to FP32 (a second rounding that differs from one rounding only on a
    # near tie of FP32, about 1 in 2^29)
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def _draws(G, freq, off, Q, seed, m, vmax):
    """Labels [L, N, V] of the copies of G (-1: no copy)."""
    L, N, V = G.shape
    K = Q.shape[1]
    z = np.full(G.shape, -1)
    for a in range(V):
        l, i = np.nonzero(G[:, :, a] >= 0)
        pos = (l % 16) * vmax + a
        w = _philox([np.full(l.size, 10 | (m << 4)), l // 16, i, pos // 4], seed)[pos % 4, np.arange(l.size)]
        u = ((w >> np.uint64(8)).astype(F) + F(1)) * F(2.0 ** -24)
        j = off[l] + G[l, i, a]
        pre, sx = [], np.zeros(l.size, F)
        for k in range(K):
            sx = _fma(Q[i, k], freq[k, j], sx)
            pre.append(sx)
        t = u * (sx + F(MIN * K))
        lab = np.full(l.size, K - 1)
        for k in range(K - 2, -1, -1):
            lab = np.where(t < _fma(np.full(l.size, k + 1, F), np.full(l.size, MIN, F), pre[k]), k, lab)
        z[l, i, a] = lab
    return z


def _check(d, K, packed, m):
    ds = S.Dataset.from_synth(d, packed=packed)
    ctx = S.Context(ds)
    seed = 7_000_000_000_123 + K
    ch = S.Chain(ctx, S.params(K, seed, admix=1, nburnin=50, nreps=50))
    G, k = d["G"][ds.order()], d["k"][ds.order()]
    N, L = ds.N, ds.L
    off = np.concatenate([[0], np.cumsum(k)])
    rng = np.random.default_rng(K)
    Q = rng.dirichlet(np.full(K, 0.4), N).astype(F)
    freq = np.concatenate([rng.dirichlet(np.full(kk, 0.6), K) for kk in k], 1).astype(F)
    ch.set("M", [m])
    ch.set("Q", Q)
    ch.set("FREQ", freq)
    ch.step("UPDATEZ")
    z = _draws(G, freq, off, Q, seed, m, G.shape[2])
    ni, mi = np.zeros((K, ds.KT), int), np.zeros((N, K), int)
    l, i, a = np.nonzero(G >= 0)
    np.add.at(ni, (z[l, i, a], off[l] + G[l, i, a]), 1)
    np.add.at(mi, (i, z[l, i, a]), 1)
    # two copies may fall on the other side of a near tie
    assert np.abs(ch.get("NI").reshape(K, -1) - ni).sum() <= 4
    assert np.abs(ch.get("MI").reshape(N, K) - mi).sum() <= 4
    ch.close()
    ctx.close()


# 2-bit data, exact and padded cluster counts, both sides of 16; edges of the
# warp, the CTA and the slice
@pytest.mark.parametrize("K", [1, 2, 5, 8, 12, 13, 16, 17])
@pytest.mark.parametrize("N,L", [(33, 47), (290, 64)])
def test_two_bit(N, L, K):
    _check(synth.fmodel(K, N, L, 3, 0.1, 0.1, admix_alpha=0.5), K, True, 3)


# the byte layout over its call widths, uniform and mixed ploidy (calls of
# 1 to 10 copies, individuals taken in ascending ploidy)
@pytest.mark.parametrize("K", [1, 3, 8, 9, 13, 16, 17])
@pytest.mark.parametrize("ploidy,alleles", [((1,), 3), ((2,), 2), ((3, 1), 4), ((2, 4, 6), 8), ((5, 8), 4), ((7,), 3),
                                            ((2, 10), 6), ((9, 3), 2)])
def test_byte_layout(ploidy, alleles, K):
    rng = np.random.default_rng(K + len(ploidy))
    N, L = 270, 37
    pl = np.resize(np.array(ploidy, np.int32), N)
    d = synth.fmodel(K, N, L, 3, 0.1, 0.1, admix_alpha=0.5, ploidy=pl, n_alleles=rng.integers(2, alleles + 1, L))
    _check(d, K, False, 4)
