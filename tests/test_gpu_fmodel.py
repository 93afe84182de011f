"""The F model's steps over many blocks and lane groups: UpdateF against the
oracle on reference streams, UpdateA's counter-stream form against its formulas
in float64 on the same Philox draws."""
import numpy as np
import pytest
from scipy.special import gammaln

from tests.test_gpu_admix_packed import _philox
from tests.test_gpu_parity import _pair, _sync_state
from vcfpop_gb300 import structure as S
from vcfpop_gb300 import synth

pytestmark = pytest.mark.gpu


# one block, several, and more alleles than threads of the largest grid
@pytest.mark.parametrize("L,K,single", [(40, 1, 0), (700, 3, 0), (3000, 5, 1), (90_000, 2, 0)])
def test_update_f(L, K, single):
    d = synth.fmodel(L, 60, L, 3, 0.1, 0.05)
    od, oc, ds, ctx, gc = _pair(d, K=K, f=1, admix=0, nadmburnin=0, singlef=single)
    for m in range(3):
        oc.m = m
        gc.set("M", np.array([m], np.int32))
        _sync_state(oc, gc, ("NI",))
        oc.step("update_p")
        _sync_state(oc, gc, ("FREQ",))
        gc.set("FF", np.concatenate([oc.get("f"), oc.get("F")]))
        gc.set("FREQA", oc.get("FREQA")[: ds.KT])
        oc.step("update_f")
        gc.step("UPDATEF")
        assert np.allclose(gc.get("FF"), np.concatenate([oc.get("f"), oc.get("F")]), rtol=1e-9)
    ctx.close()


class _Stream:
    def __init__(self, seed, a, b):
        self.seed, self.a, self.b, self.blk, self.buf = seed, a, b, 0, []

    def next(self):
        if not self.buf:
            one = lambda v: np.array([v], np.uint32)  # noqa: E731
            self.buf = [int(x[0]) for x in _philox([one(self.a), one(self.b), one(0), one(self.blk)], self.seed)]
            self.blk += 1
        return self.buf.pop(0)

    def f(self):
        return ((self.next() >> 8) + 1) / 2.0 ** 24

    def d(self):
        h = self.next()
        return ((((h << 32) | self.next()) >> 11) + 1) / 2.0 ** 53

    def gamma(self, alpha):
        a = alpha + 1 if alpha < 1 else alpha
        d = a - 1 / 3
        c = 1 / np.sqrt(9 * d)
        while True:
            u1, u2 = self.f(), self.f()
            t = np.sqrt(-2 * np.log(u1)) * np.cos(2 * np.pi * u2)
            v = 1 + c * t
            if v <= 0:
                continue
            v, u = v ** 3, self.f()
            if u < 1 - 0.0331 * t ** 4 or np.log(u) < 0.5 * t * t + d * (1 - v + np.log(v)):
                break
        return d * v * (self.f() ** (1 / alpha) if alpha < 1 else 1)


def _log(x):
    return np.log(x) if x > 1e-300 else -6.90775527898214e2


# alleles and clusters around the eight lanes of a group
@pytest.mark.parametrize("K,alleles", [(1, (2, 2)), (4, (2, 2)), (3, (2, 8)), (9, (3, 11))])
def test_update_a_counter_streams(K, alleles):
    rng = np.random.default_rng(K)
    L, N = 150, 60
    k = rng.integers(alleles[0], alleles[1] + 1, L)
    d = synth.fmodel(K, N, L, 3, 0.1, 0.05, n_alleles=k)
    ds = S.Dataset.from_synth(d)
    ctx = S.Context(ds)
    seed = 987654321 + K
    c = S.Chain(ctx, S.params(K, seed, admix=1, f=1))
    kk = d["k"][ds.order()]
    off = np.concatenate([[0], np.cumsum(kk)])
    done = {True: 0, False: 0}
    for m in range(6):
        c.set("M", np.array([m], np.int32))
        c.step("UPDATEP")
        before, p = c.get("FREQA").astype(np.float64), c.get("FREQ").astype(np.float64).reshape(K, -1)
        f = c.get("FF")[:K]
        c.step("UPDATEA")
        after = c.get("FREQA").astype(np.float64)
        one = bool(S.run_seed(seed + m, 0) & 1)        # the hash the sweep's form is picked by
        done[one] += 1
        wrong = 0
        for l in range(len(kk)):
            s = slice(off[l], off[l + 1])
            pa, pk, n = before[s], p[:, s], int(kk[l])
            st = _Stream(seed, 7 | (m << 4), l)
            new = pa.copy()
            if one:
                pb = 1.0 + (pk * f[:, None]).sum(0)
                g = np.array([st.gamma(x) for x in pb])
                new = g / g.sum()
                r = sum((pb[a] - 1.0) * _log(pa[a] / new[a]) for a in range(n))
                r += sum(gammaln(f[j] * pa[a]) - gammaln(f[j] * new[a]) + f[j] * (new[a] - pa[a]) * _log(pk[j, a])
                         for j in range(K) for a in range(n))
            else:
                a, b = st.next() % n, st.next() % (n - 1)
                b += b >= a
                delta = st.d() * N ** -0.5
                new[a] += delta
                new[b] -= delta
                if new[a] >= 1 or new[b] <= 0:
                    assert np.array_equal(after[s], pa)
                    continue
                r = sum(gammaln(f[j] * pa[a]) + gammaln(f[j] * pa[b]) - gammaln(f[j] * new[a]) - gammaln(f[j] * new[b]) +
                        f[j] * delta * _log(pk[j, a] / pk[j, b]) for j in range(K))
            acc = r >= -1e-10 or st.d() < np.exp(r)
            wrong += not np.allclose(after[s], new if acc else pa, rtol=1e-3, atol=1e-5)
        # FP32 draws against float64 ones: a rejection or a decision may differ at its edge
        assert wrong <= 2, (m, one, wrong)
    assert done[True] and done[False]
    c.close()
    ctx.close()
