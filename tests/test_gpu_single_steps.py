"""Single steps taken in the middle of a run: UPDATEQ reads the frequencies that
the chain holds, whatever sweep wrote them last."""
import numpy as np
import pytest

from vcfpop_gb300 import _lib as B
from vcfpop_gb300 import structure as S

from .test_gpu_plain_tc import _calls, _chain

pytestmark = pytest.mark.gpu

# an FP32 logarithm is within 2^-23 of its value; the FP32 stream adds up to 32
# terms of one sign a slice, each rounding at most 2^-24 of the slice's sum
REL = 2.0 ** -23 + 32 * 2.0 ** -24


def _check(c, ch, K):
    L, N = c.shape
    lp = np.log(ch.get("FREQ").astype(np.float64)).reshape(K, L, 2)
    c0 = np.where(c == 3, 0, 2 - c).astype(np.float64)
    c1 = np.where(c == 3, 0, c).astype(np.float64)
    want = c0.T @ lp[:, :, 0].T + c1.T @ lp[:, :, 1].T
    got = ch.get("LL").reshape(N, K)
    assert np.all(np.abs(got - want) <= REL * np.abs(want) + 2.0 ** -25 * 2 * L)


# nburnin = 2, nthinning = 10: sweep 2 is recorded, 0, 1 and 3 to 5 are not
@pytest.mark.parametrize("N,L,K", [(200, 400, 6), (333, 129, 12), (520, 8200, 3)])
@pytest.mark.parametrize("sweeps", [1, 2, 3, 4])
def test_update_q_after_a_run(N, L, K, sweeps):
    c, ctx, ch = _chain(_calls(N, L, N + K), K)
    ch.run(sweeps)
    ch.step("UPDATEQ")
    _check(c, ch, K)
    ch.close()
    ctx.close()


def test_update_q_after_next():
    c, ctx, ch = _chain(_calls(200, 400, 1), 6)
    ch.step("UPDATEQ")                       # the initial frequencies
    _check(c, ch, 6)
    for _ in range(4):                       # over the recorded sweep and back
        ch.step("UPDATEP")
        ch.step("NEXT")
        ch.step("UPDATEQ")
        _check(c, ch, 6)
    ch.close()
    ctx.close()


@pytest.mark.parametrize("K", [3, 6])        # one table, both tables
def test_update_q_after_a_batch(K):
    c, ctx, ch = _chain(_calls(200, 400, 2), K)
    tc = S.Chain(ctx, S.params(K, 5, form=B.VP_FORM_TC, admix=0, nadmburnin=0, nburnin=2, nreps=4))
    for _ in range(3):
        tc.run(1)
        tc.step("UPDATEQ")
        _check(c, tc, K)
    tc.close()
    ch.close()
    ctx.close()
