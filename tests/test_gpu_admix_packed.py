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
    out = {f: c.get(f) for f in ("NI", "MI", "Q", "FREQ", "ALPHA", "METRO")}
    out["L"] = ds.L
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
    # Metropolis log ratios: the byte layout's FP32 sums over 64 copies round
    # at up to 64 x 5 x 2^-24 a copy
    assert np.allclose(a["METRO"], b["METRO"], rtol=0, atol=2 * 64 * 5 * 2.0 ** -24 * a["L"])


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


def _philox(c, key):
    """Philox-4x32-10 of uint32 counters c [4, n] (Salmon et al., SC'11)."""
    c = [x.astype(np.uint64) for x in c]
    k = [int(key) & 0xFFFFFFFF, int(key) >> 32]
    m = np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k[0]), p1 & m, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k[1]), p0 & m]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    return np.stack(c)


# the initial labels of every copy: one stream per (locus, individual), its
# draws modulo K, over CTA and slice edges, both layouts and mixed ploidy
@pytest.mark.parametrize("N,L,K,poly", [(15, 17, 1, 0), (257, 33, 5, 0), (256, 16, 3, 1), (300, 70, 16, 0), (90, 41, 7, 1)])
def test_initial_labels(N, L, K, poly):
    rng = np.random.default_rng(N)
    kw = dict(ploidy=rng.choice([1, 2, 4, 6], N), n_alleles=rng.integers(2, 6, L)) if poly else {}
    d = synth.fmodel(N, N, L, 3, 0.1, 0.1, admix_alpha=0.5, **kw)
    ds = S.Dataset.from_synth(d)
    ctx = S.Context(ds)
    seed = 1234567890123 + K
    c = S.Chain(ctx, S.params(K, seed, admix=1))
    order = ds.order()
    G, k = d["G"][order], d["k"][order]
    off = np.concatenate([[0], np.cumsum(k)])
    ll, ii = (x.reshape(-1) for x in np.meshgrid(np.arange(len(order)), np.arange(N), indexing="ij"))
    draws = [_philox([np.full(ll.size, 8, np.uint32), ll, ii, np.full(ll.size, b, np.uint32)], seed) for b in range(2)]
    draws = np.concatenate(draws).reshape(8, len(order), N).astype(np.int64) % K
    Mi, Ni = np.zeros((N, K), int), np.zeros((K, ds.KT), int)
    for a in range(G.shape[2]):
        l, i = np.nonzero(G[:, :, a] >= 0)
        z = draws[a, l, i]
        np.add.at(Mi, (i, z), 1)
        np.add.at(Ni, (z, off[l] + G[l, i, a]), 1)
    assert np.array_equal(c.get("MI").reshape(N, K), Mi)
    assert np.array_equal(c.get("NI").reshape(K, -1), Ni)
    c.close()
    ctx.close()


# the byte layout's kernel over its call widths (1 to 16 bytes), ploidies and
# cluster counts: every copy counted once, in its individual and its allele
@pytest.mark.parametrize("ploidy,alleles", [((1,), 3), ((2,), 5), ((3, 4), 2), ((2, 4, 6), 8), ((8,), 4), ((2, 10), 6)])
@pytest.mark.parametrize("K", [1, 5, 13, 17])
def test_byte_layout_counts(ploidy, alleles, K):
    rng = np.random.default_rng(K + len(ploidy))
    N, L = 290, 37
    pl = np.resize(np.array(ploidy, np.int32), N)
    d = synth.fmodel(K, N, L, 3, 0.1, 0.1, admix_alpha=0.5, ploidy=pl, n_alleles=rng.integers(2, alleles + 1, L))
    ds = S.Dataset.from_synth(d, packed=False)
    ctx = S.Context(ds)
    c = S.Chain(ctx, S.params(K, 5, admix=1))
    c.run(3)
    G, k = d["G"][ds.order()], d["k"][ds.order()]
    ni = c.get("NI").reshape(K, -1).sum(0)
    off = np.concatenate([[0], np.cumsum(k)])
    for l in range(ds.L):
        assert np.array_equal(ni[off[l]:off[l + 1]], [(G[l] == a).sum() for a in range(k[l])])
    assert np.array_equal(c.get("MI").reshape(N, K).sum(1), (G >= 0).sum((0, 2)))
    c.close()
    ctx.close()
