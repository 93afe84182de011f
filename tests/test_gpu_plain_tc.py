"""The plain form's tensor-core likelihood and counts against float64 and exact
counts, at the edges of their tiles, stages and compiled widths."""
import numpy as np
import pytest

from vcfpop_gb300 import structure as S

pytestmark = pytest.mark.gpu


def _calls(N, L, seed):
    rng = np.random.default_rng(seed)
    p = rng.beta(0.5, 0.5, (L, 1)).clip(0.02, 0.98)
    c = (rng.random((L, N)) < p).astype(np.int8) + (rng.random((L, N)) < p)
    c[rng.random((L, N)) < 0.05] = 3
    c[:, 0], c[:, 1] = 1, 0                  # every locus polymorphic, and kept
    return c


def _chain(c, K):
    L, N = c.shape
    Nw = (N + 15) // 16
    pad = np.full((L, Nw * 16), 3, np.uint32)
    pad[:, :N] = c
    packed = np.bitwise_or.reduce(pad.reshape(L, Nw, 16) << (2 * np.arange(16, dtype=np.uint32)), axis=2).astype(np.uint32)
    ds = S.Dataset(np.full(N, 2), np.full(L, 2), np.zeros(N), 1, packed2=packed)
    assert ds.L == L
    ctx = S.Context(ds)
    ch = S.Chain(ctx, S.params(K, 11 + K, admix=0, nadmburnin=0, nburnin=2, nreps=4))
    return c[ds.order()], ctx, ch


def _check_ll(c, ch, K, f, rel=2.0 ** -23):
    L, N = c.shape
    lp = np.where(f > 0, np.log(np.where(f > 0, f.astype(np.float64), 1)), -709.0895657128241).reshape(K, L, 2)
    c0 = np.where(c == 3, 0, 2 - c).astype(np.float64)
    c1 = np.where(c == 3, 0, c).astype(np.float64)
    want = c0.T @ lp[:, :, 0].T + c1.T @ lp[:, :, 1].T
    got = ch.get("LL").reshape(N, K)
    # an FP32 logarithm is within 2^-23 of its value (terms of one sign) and its
    # whole number of 2^-24 within 2^-25 a copy
    assert np.all(np.abs(got - want) <= rel * np.abs(want) + 2.0 ** -25 * 2 * L)


# individuals around the CTA's 256 and a warp's 32, loci around the 32-locus
# stage, every compiled width
@pytest.mark.parametrize("N,L,K", [(512, 4096, 1), (513, 4097, 4), (545, 4127, 6), (600, 8200, 10), (1000, 4160, 11),
                                   (768, 4129, 16), (1025, 4100, 17), (520, 4128, 32), (530, 20_001, 3), (513, 8193, 1),
                                   (1025, 4127, 4), (33, 129, 5), (20, 161, 32), (257, 400, 12)])
def test_likelihood(N, L, K):
    c, ctx, ch = _chain(_calls(N, L, N + K), K)
    ch.set("M", [1])                         # a sweep that Record does not read
    ch.step("UPDATEP")
    ch.step("UPDATEQ")
    _check_ll(c, ch, K, ch.get("FREQ"))
    # extreme frequencies: zeros, ones and the smallest normal number
    rng = np.random.default_rng(K)
    f = rng.choice(np.array([0, 1, 1.2e-38, 0.5, 1e-10], np.float32), K * 2 * L)
    ch.set("FREQ", f)
    ch.step("UPDATEQ")
    _check_ll(c, ch, K, f)
    # the FP32 stream on the table rebuilt for it: up to 32 adds a slice, each
    # rounding at most 2^-24 of the slice's sum (terms of one sign)
    ch.step("LOGLIK")
    _check_ll(c, ch, K, f, 2.0 ** -23 + 32 * 2.0 ** -24)
    ch.close()
    ctx.close()


@pytest.mark.parametrize("N,L,K", [(512, 8192, 1), (513, 8193, 2), (640, 8200, 16), (641, 8319, 17), (777, 9000, 32), (1023, 8321, 7), (515, 130, 3),
                                   (2049, 2050, 9), (127, 17_000, 4), (3841, 1100, 5)])
def test_counts(N, L, K):
    c, ctx, ch = _chain(_calls(N, L, N + K), K)
    rng = np.random.default_rng(N)
    z = rng.integers(0, K, N)
    for labels in (ch.get("Z"), z):           # the initial counts, then counts of labels set
        if labels is z:
            ch.set("Z", z)
            ch.step("UPDATEZ")
        got = ch.get("NI").reshape(K, L, 2)
        for k in range(K):
            s = c[:, labels == k]
            assert np.array_equal(got[k, :, 1], np.where(s == 3, 0, s).sum(1))
            assert np.array_equal(got[k, :, 0], np.where(s == 3, 0, 2 - s).sum(1))
    ch.close()
    ctx.close()


def test_sweeps_agree_with_the_byte_layout():
    """Whole sweeps on the tensor-core path against the byte layout's FP32
    likelihood stream: the same labels and counts."""
    c = _calls(600, 9000, 5)
    G = np.stack([np.where(c == 3, -1, c > 1), np.where(c == 3, -1, c > 0)], -1).astype(np.int8)
    out = []
    for packed in (True, False):
        if packed:
            _, ctx, ch = _chain(c, 4)
        else:
            ds = S.Dataset(np.full(600, 2), np.full(9000, 2), np.zeros(600), 1, G=G)
            ctx = S.Context(ds)
            ch = S.Chain(ctx, S.params(4, 15, admix=0, nadmburnin=0, nburnin=2, nreps=4))
        ch.run(6)
        out.append([ch.get(f) for f in ("Z", "NI", "FREQ")])
        ch.close()
        ctx.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
