"""The batched K-sweep's count contraction against exact counts of the labels:
the packed form (a missing call as a power of two) at the ends of its range,
and the form with a row per allele where the sums would not be exact."""
import numpy as np
import pytest

from tests.test_gpu_plain_tc import _calls
from vcfpop_gb300 import _lib as B
from vcfpop_gb300 import structure as S

pytestmark = pytest.mark.gpu


def _counts(c, labels, K):
    out = np.empty((K, c.shape[0], 2), np.int64)
    for k in range(K):
        s = c[:, labels == k]
        out[k, :, 1] = np.where(s == 3, 0, s).sum(1)
        out[k, :, 0] = np.where(s == 3, 0, 2 - s).sum(1)
    return out


# `missing` of one locus's calls are missing: N = 8,191 uses 2^14 (up to 1,022
# missing), 8,200 uses 2^15 (up to 511), 16,400 is past e5m2's range
@pytest.mark.parametrize("N,L,missing,ks", [(40, 70, 40, (1, 2, 3)), (513, 200, 500, (2, 17)), (2003, 333, 1900, (3, 5)),
                                            (8191, 130, 1022, (1, 4)), (8200, 131, 510, (2, 2)), (8200, 131, 512, (2, 3)),
                                            (16_400, 64, 100, (2,))])
def test_counts(N, L, missing, ks):
    c = _calls(N, L, N + missing)
    if missing < N:
        c[:, 2:] = np.where(np.random.default_rng(1).random((L, N - 2)) < 0.01, 3, np.minimum(c[:, 2:], 2))
    c[7, 2:2 + missing] = 3
    Nw = (N + 15) // 16
    pad = np.full((L, Nw * 16), 3, np.uint32)
    pad[:, :N] = c
    packed = np.bitwise_or.reduce(pad.reshape(L, Nw, 16) << (2 * np.arange(16, dtype=np.uint32)), axis=2).astype(np.uint32)
    ds = S.Dataset(np.full(N, 2), np.full(L, 2), np.zeros(N), 1, packed2=packed)
    ctx = S.Context(ds)
    chains = [S.Chain(ctx, S.params(K, 900 + K, form=B.VP_FORM_TC, admix=0, nadmburnin=0, nburnin=2, nreps=4))
              for K in ks]
    c = c[ds.order()]
    for sweeps in (0, 1, 2):
        if sweeps:
            S.run_chains(chains, sweeps)
        for ch, K in zip(chains, ks):
            assert np.array_equal(ch.get("NI").reshape(K, ds.L, 2), _counts(c, ch.get("Z"), K)), (K, sweeps)
    assert B.lib().vp_tc_status(ctx.h) == 0
    ctx.close()
