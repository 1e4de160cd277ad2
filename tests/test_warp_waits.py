"""Waits of whole warps in the int8 contraction kernel (CPU only, from the source; the GPU's side is
trpdrv_selftest_bounded_wait): a warp whose lanes all poll, and whose loop holds instructions for all lanes (elect.sync,
tcgen05.ld, __syncwarp), must leave that loop as one, also when some lanes run out of time just as the phase completes."""
import os
import re

from conftest import ROOT


def _kernel():
    with open(os.path.join(ROOT, "nwchem-ccsd-trpdrv_b200", "csrc", "ozaki.cu")) as f:
        src = f.read()
    body = src[src.index("oz_gemm_kernel(const __grid_constant__ GemmParams P)"):]
    return src, body[:body.index("\n}\n")]


def test_warps_that_wait_with_all_lanes_leave_as_one():
    src, body = _kernel()
    mma = body[body.index("MMA issuer"):body.index("energy_operands<")]
    drain = body[body.index("recombination: TMEM lanes"):body.index("energy warps: the units")]
    for role in (mma, drain):
        waits = re.findall(r"if \(!(mbar_\w+)\(", role)
        assert waits and set(waits) == {"mbar_wait_warp"}, waits
    helper = src[src.index("bool mbar_wait_warp_for("):]
    assert "__all_sync(0xffffffffu, mbar_wait_for(" in helper[:helper.index("\n}\n")]
