"""The tensor-core likelihood where one allele is rare: most terms of an
individual's sum are logarithms near zero."""
import numpy as np
import pytest

from .test_gpu_plain_tc import _calls, _chain

pytestmark = pytest.mark.gpu


# Every locus of a cluster has the same frequencies, so that roundings of the
# common logarithm add up instead of cancelling. The bound: the logarithm within
# 2^-23 of its value, and half a unit of 2^-29 a copy.
@pytest.mark.parametrize("N,L,K", [(300, 4096, 6), (257, 8200, 10)])
@pytest.mark.parametrize("rare", [1e-6, 1e-5, 1.3e-4, 1.1e-3, 0.01, 0.3])
def test_likelihood(N, L, K, rare):
    c = _calls(N, L, N)
    c[:, 2:] = np.where(c[:, 2:] == 3, 3, (np.random.default_rng(L).random((L, N - 2)) < 2 * rare).astype(np.int8))
    c, ctx, ch = _chain(c, K)
    ch.set("M", [1])                         # a sweep that Record does not read
    p1 = (rare * (1 + np.arange(K) / 7)).astype(np.float32)
    f = np.repeat(np.stack([np.float32(1) - p1, p1], -1)[:, None, :], L, 1)
    ch.set("FREQ", f)
    ch.step("UPDATEQ")
    lp = np.log(f.astype(np.float64))
    c0 = np.where(c == 3, 0, 2 - c).astype(np.float64)
    c1 = np.where(c == 3, 0, c).astype(np.float64)
    want = c0.T @ lp[:, :, 0].T + c1.T @ lp[:, :, 1].T
    got = ch.get("LL").reshape(N, K)
    assert np.all(np.abs(got - want) <= 2.0 ** -23 * np.abs(want) + 2.0 ** -30 * 2 * L)
    ch.close()
    ctx.close()
