"""Order of memory operations in the tensor-core M2L, from its source.

The gathered multipole rows reach shared memory by cp.async, which writes
through the generic proxy; tcgen05.mma reads them through the async proxy.
The mbarrier alone does not order accesses of different proxies (PTX ISA,
"Proxies" and "fence.proxy"): a proxy fence has to stand between the wait that
observes the copies and the MMAs that read them.  Hardware need not show a
missing one in any run, so the order is checked in the source text.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "minimal_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def test_proxy_fence_between_copies_and_mmas():
    kernel = _code("m2l_group.cu").split("k_m2l_tc(", 1)[1]
    issuer = kernel[kernel.index("warp == TC_MMA_WARP) {"):]
    mma = issuer.index("tc::mma_f16(")
    wait = issuer.rindex("&full[st]", 0, mma)
    assert "tc::fence_async_smem();" in issuer[wait:mma]


def test_proxy_fence_is_the_async_one():
    body = _code("tc.cuh").split("void fence_async_smem()", 1)[1].split("}", 1)[0]
    assert "fence.proxy.async.shared::cta;" in body
