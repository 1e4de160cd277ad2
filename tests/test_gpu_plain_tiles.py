"""The plain path's tiles and batches against the oracle (B200 only): 64- and 32-wide tiles with ragged edges, odd
sizes (8-byte copies), batches that end inside a system, i == k triples, and the single-triple entry point at
the sizes where its tiles change.  Bars: 1e-11 of a column's largest record, as in the parity tests."""
import numpy as np
import pytest

from conftest import assert_records_close, assert_total_close

pytestmark = pytest.mark.gpu

# batches hold 256 triples at most, so (9, .) and (12, .) end inside one
SHAPES = [(1, 1), (2, 15), (3, 16), (4, 33), (9, 48), (12, 40), (5, 63), (6, 64), (4, 65), (3, 97), (2, 130), (3, 200)]


@pytest.mark.parametrize("shape", SHAPES)
def test_plain_plan_matches_the_oracle(T, O, shape):
    nocc, nvir = shape
    s = T.synth_system(nocc, nvir, seed=300 * nocc + nvir, ncor=nvir % 3)
    want, tot, mism = O.run_system(s, "port", nthreads=4)
    assert mism == 0
    with T.Plan([s], mode=T.MODE_PLAIN) as p:
        p.upload()
        p.execute()
        e4, e5 = p.energies()
        rec = p.triple_energies(0)
        p.execute()
        assert np.array_equal(p.triple_energies(0), rec)
    assert_records_close(rec, want)
    assert_total_close(e4[0], tot[0], what="emp4")
    assert_total_close(e5[0], tot[1], what="emp5")


def test_plain_plan_of_several_systems_and_a_values(T, O):
    systems = [T.synth_system(7, 30, seed=1, a_count=2), T.synth_system(3, 70, seed=2, a_count=2)]
    with T.Plan(systems, mode=T.MODE_PLAIN) as p:
        p.upload()
        p.execute()
        recs = [p.triple_energies(q) for q in range(2)]
    for q, s in enumerate(systems):
        want = np.concatenate([O.run_system(s.a_view(a), "port", nthreads=4)[0] for a in range(2)])
        assert_records_close(recs[q], want)
