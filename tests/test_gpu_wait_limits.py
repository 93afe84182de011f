"""Waits of the plain form's tensor-core kernels that run out: without a fault,
the launch ends with an error on its chain, and the device, the context and its
other chains stay usable."""
import pytest

from vcfpop_gb300 import _lib as B
from vcfpop_gb300 import structure as S

from .test_gpu_plain_tc import _calls, _chain

pytestmark = pytest.mark.gpu


def _stall(ch, on):
    B.check(B.lib().vp_debug_chain_stall(ch.h, on))


def _params(K, seed):
    return S.params(K, seed, admix=0, nadmburnin=0, nburnin=2, nreps=4)


# every compiled width of the likelihood and of the counts; 4,100 individuals are
# three groups of the counts' accumulators
@pytest.mark.parametrize("N,L,K", [(530, 8300, 3), (600, 8200, 6), (600, 8200, 10), (1000, 4200, 16), (4100, 1100, 20)])
def test_a_run_ends_and_the_next_chain_is_right(N, L, K):
    c, ctx, ch = _chain(_calls(N, L, K), K)
    want = S.Chain(ctx, _params(K, 5))
    want.run(6)
    _stall(ch, 1)
    ch.run(3)                                # label draws and counts give up
    with pytest.raises(B.VpError, match="timed out"):
        ch.result()
    ch.close()
    got = S.Chain(ctx, _params(K, 5))
    got.run(6)
    for f in ("Z", "NI", "FREQ", "LL"):
        assert (got.get(f) == want.get(f)).all()
    for x in (got, want):
        x.close()
    ctx.close()


def _raises(f, *a):
    with pytest.raises(B.VpError, match="timed out"):
        f(*a)


# the counts of 600 individuals run on the tensor cores, with 6 clusters the
# likelihood too
@pytest.mark.parametrize("L,K", [(6000, 4), (8200, 6)])
def test_every_way_to_the_state_reports(L, K):
    c, ctx, ch = _chain(_calls(600, L, K), K)
    other = S.Chain(ctx, _params(K, 5))
    _stall(ch, 1)
    ch.run(2)
    for f in ("FREQ", "Q", "Z", "NI", "MI", "LL", "ALPHA", "M", "FF", "LOCP"):
        _raises(ch.get, f)
    _raises(ch.result)
    _raises(ch.step, "UPDATEP")
    _raises(S.finish, [ch])
    _raises(ch.result, True)
    _raises(ch.divergence)
    S.finish([other])                        # the context's other chain is well
    other.divergence()
    assert other.result()["nr"] == 1
    ch.close()
    other.close()
    ctx.close()


def test_steps_report():
    c, ctx, ch = _chain(_calls(600, 8200, 1), 6)
    ch.step("UPDATEP")
    _stall(ch, 1)
    _raises(ch.step, "UPDATEQ")
    ch.close()
    ch = S.Chain(ctx, _params(6, 5))
    _stall(ch, 1)
    _raises(ch.step, "UPDATEZ")
    ch.close()
    ctx.close()


def test_a_cohort_reports():
    c, ctx, ch = _chain(_calls(600, 8200, 2), 6)
    other = S.Chain(ctx, _params(6, 5))
    _stall(ch, 1)
    co = S.Cohort()
    co.set([ch, other])
    co.run(3)
    _raises(co.sync)
    _raises(ch.get, "Z")
    assert other.get("M")[0] == 3
    co.close()
    for x in (ch, other):
        x.close()
    ctx.close()
