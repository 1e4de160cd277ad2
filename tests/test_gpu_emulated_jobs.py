"""The emulated form's products list and its odd-nvir energies (B200 only): triples with i == k form one group of
products, whose f serve both families; odd nvir stores f with padded columns and reads them by TMA in the
separate energy launch.  Against the oracle at 1e-11 of a column's largest record, 8 slices."""
import numpy as np
import pytest

from conftest import assert_records_close, assert_total_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 16), (2, 33), (5, 47), (4, 64), (9, 65), (12, 31)])
@pytest.mark.parametrize("batch", [8, 64])
def test_records_match_the_oracle(T, O, shape, batch):
    nocc, nvir = shape
    s = T.synth_system(nocc, nvir, seed=17 * nocc + nvir, ncor=1)
    want, tot, mism = O.run_system(s, "port", nthreads=4)
    assert mism == 0
    with T.Plan([s], mode=T.MODE_EMULATED, slices=8, batch=batch) as p:
        p.upload()
        p.execute()
        e4, e5 = p.energies()
        rec = p.triple_energies(0)
    assert_records_close(rec, want)
    assert_total_close(e4[0], tot[0], what="emp4")
    assert_total_close(e5[0], tot[1], what="emp5")


def test_a_sweep_of_an_odd_size(T, O):
    s = T.synth_system(3, 37, seed=8, a_count=3)
    with T.Plan([s], mode=T.MODE_EMULATED, slices=8) as p:
        p.upload()
        p.execute()
        rec = p.triple_energies(0)
    want = np.concatenate([O.run_system(s.a_view(a), "port", nthreads=4)[0] for a in range(3)])
    assert_records_close(rec, want)
