"""Emulated plans that mix even and odd nvir (B200 only): the energies of some systems run inside the contraction
launch, those of others on a second stream.  A job enqueued outside a graph after one was captured (autotune), or
captured again (a second upload), must not wait on events of the earlier capture."""
import numpy as np
import pytest

from conftest import assert_records_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nvirs", [(64, 33), (33, 64), (33, 64, 35)])
@pytest.mark.parametrize("between", ["autotune", "upload"])
def test_second_job_after_a_captured_one(T, nvirs, between):
    systems = [T.synth_system(7, v, seed=v) for v in nvirs]
    want = [T.Plan([s], mode=T.MODE_FUSED) for s in systems]
    with T.Plan(systems, mode=T.MODE_EMULATED, batch=8) as p:  # 7 x 28 triples: many batches
        p.upload()
        p.execute()
        first = [p.triple_energies(q) for q in range(len(systems))]
        getattr(p, between)()
        p.execute()
        again = [p.triple_energies(q) for q in range(len(systems))]
    for q, w in enumerate(want):
        w.upload()
        w.execute()
        assert_records_close(first[q], w.triple_energies(0))
        assert np.array_equal(again[q], first[q])
        w.close()
