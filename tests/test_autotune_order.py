"""What the autotuner times: small plans in the order in which they run their items (from the source, CPU)."""
import os

from conftest import ROOT


def test_candidates_are_timed_in_the_order_that_plans_run():
    with open(os.path.join(ROOT, "nwchem-ccsd-trpdrv_b200", "csrc", "host.c")) as f:
        src = f.read()
    for name in ("enqueue_fused", "tune_time"):
        body = src[src.index(f"static int {name}("):]
        body = body[:body.index("\n}\n")]
        assert "plan_pair_major(p)" in body
        for launch in body.split("LAUNCH_TRY(trpdrv_launch_fused")[1:]:
            assert "pair_major" in launch[:launch.index(";")]
