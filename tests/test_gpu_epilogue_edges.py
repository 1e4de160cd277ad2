"""Energies at the edge of the tiles (B200 only): positions past nvir add exactly nothing, also where the vectors of
the last virtual orbital are not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["MODE_FUSED", "MODE_EMULATED", "MODE_PLAIN"])
@pytest.mark.parametrize("nvir", [1, 15, 33, 48, 50])
def test_an_infinity_at_the_last_orbital_stays_in_its_records(T, mode, nvir):
    nocc, x = 3, 1
    s = T.synth_system(nocc, nvir, seed=11)

    def records():
        with T.Plan([s], mode=getattr(T, mode)) as p:
            p.upload()
            p.execute()
            return p.triple_energies(0), p.triples(0)

    base, triples = records()
    s.arrays["dintx"][x * nvir + nvir - 1] = np.inf
    got, _ = records()
    # e5 of a triple reads the vectors of its i (column 1) and k (column 3)
    hit = np.array([[False, t[0] == x + 1, False, t[2] == x + 1] for t in triples])
    assert np.array_equal(got[~hit], base[~hit])
    assert hit.any() and not np.isfinite(got[hit]).any()
