"""Labels that name no cluster: the counts of the tensor-core form leave their
individuals out."""
import numpy as np
import pytest

from .test_gpu_plain_tc import _calls, _chain

pytestmark = pytest.mark.gpu


# both compiled widths, 16 and 32 rows
@pytest.mark.parametrize("N,L,K", [(513, 8193, 3), (640, 8200, 16), (777, 9000, 20)])
def test_counts(N, L, K):
    c, ctx, ch = _chain(_calls(N, L, N), K)
    rng = np.random.default_rng(K)
    z = rng.integers(0, K, N)
    z[rng.choice(N, 60, replace=False)] = rng.choice([K, 15, 16, 31, 32, 33, 4096, 65534, 65535], 60)
    ch.set("Z", z)
    ch.step("UPDATEZ")
    got = ch.get("NI").reshape(K, L, 2)
    for k in range(K):
        s = c[:, z == k]
        assert np.array_equal(got[k, :, 1], np.where(s == 3, 0, s).sum(1))
        assert np.array_equal(got[k, :, 0], np.where(s == 3, 0, 2 - s).sum(1))
    ch.close()
    ctx.close()
