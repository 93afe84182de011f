"""Device memory that ingest and the locus filters keep between calls: at most
256 MiB in all, and none after vp_release_memory or where a server sizes its
default budget."""
import numpy as np
import pytest

from vcfpop_gb300 import _lib as B
from vcfpop_gb300 import structure as S

pytestmark = pytest.mark.gpu

KEPT = 256 << 20
SLACK = 64 << 20        # the pool's own grain


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _text(mib):
    line = b"1\t1\t.\tA\tC\t.\tPASS\t.\tGT" + b"\t0/1" * 25_000 + b"\n"
    return line * ((mib << 20) // len(line))


def _general(mib):
    G = np.zeros(((mib << 20) // 2000, 1000, 2), np.int8)
    G[:, ::2, 1] = 1
    return G, np.full(len(G), 2)


CALLS = {
    "pack2": lambda mib: S.vcf_pack2(_text(mib), 25_000),
    "filter": lambda mib: S.locus_filter(np.full(((mib << 20) // 4000, 1000), 0x55555554, np.uint32), 16_000,
                                         S.locus_filter_spec(bmaf=(0.1, 0.5))),
    "general_filter": lambda mib: S.locus_filter_general(*_general(mib), S.locus_filter_spec(bmaf=(0.1, 0.5))),
}


@pytest.mark.parametrize("call", CALLS)
def test_a_large_call_keeps_little(call):
    CALLS[call](1)                           # kernels loaded
    B.check(B.lib().vp_release_memory(0))
    before = _free()
    CALLS[call](640)
    assert _free() >= before - KEPT - SLACK
    CALLS[call](64)                          # kept for the next call
    B.check(B.lib().vp_release_memory(0))
    assert _free() >= before - SLACK


def test_a_server_takes_what_ingest_kept_into_its_budget():
    ds = S.Dataset(np.full(4, 2), [2, 2], np.zeros(4), 1, packed2=np.array([[0x24], [0x18]], np.uint32))
    S.Server().close()
    B.check(B.lib().vp_release_memory(0))
    before = _free()
    CALLS["pack2"](160)
    srv = S.Server()
    assert _free() >= before - SLACK
    srv.close()
    del ds
