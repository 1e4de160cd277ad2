"""The fused kernel's last chunk of either contraction, by the number of its valid indices: a k4 step, a k8 step, both or
two (B200 only).  Every remainder of nvir with each kind of nocc, on ordinary, diagonal, packed and i == k items, against
the oracle at 1e-11 of a column's largest record."""
import pytest

from conftest import assert_records_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mma_k", [4, 8, 16])
@pytest.mark.parametrize("nvir", list(range(33, 49)) + [1, 4, 12, 68, 76])
def test_remainders_of_both_contractions(T, O, nvir, mma_k):
    for nocc in (3, 7, 10, 13):
        s = T.synth_system(nocc, nvir, seed=100 * nocc + nvir)
        want, _, mism = O.run_system(s, "port", nthreads=4)
        assert mism == 0
        with T.Plan([s], mode=T.MODE_FUSED, mma_k=mma_k) as p:
            p.upload()
            p.execute()
            assert_records_close(p.triple_energies(0), want)
