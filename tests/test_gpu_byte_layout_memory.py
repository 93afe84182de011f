"""Device memory of the byte layout: a call takes its vmax bytes, whatever vmax."""
import numpy as np
import pytest

from vcfpop_gb300 import structure as S

pytestmark = pytest.mark.gpu


def _bytes(vmax, N=300, L=2000):
    rng = np.random.default_rng(1)
    G = np.full((L, N, vmax), -1, np.int8)
    G[:, :, 0] = rng.integers(0, 3, (L, N))
    ds = S.Dataset(np.full(N, 1), np.full(L, 3), np.zeros(N), 1, G=G)
    assert ds.L == L
    srv = S.Server()
    rid = srv.submit(ds, S.params(3, 1, admix=1, nburnin=1, nreps=1))
    n = srv.wait(rid)["device_bytes"]
    srv.release(rid)
    srv.close()
    return n


@pytest.mark.parametrize("a,b", [(1, 3), (4, 5), (5, 7), (8, 9), (9, 10)])
def test_a_byte_a_copy(a, b):
    # every array is rounded to 512 bytes
    assert abs(_bytes(b) - _bytes(a) - (b - a) * 300 * 2000) <= 1024
