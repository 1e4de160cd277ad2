"""The plain path's running-pointer copies (B200 only), around the sizes where they begin (nvir 32 with 8-byte
copies, 64 with 16-byte ones) and at whole and ragged tiles of both widths, against the oracle at 1e-11 of a column's
largest record.  Even nvir with odd nocc also copies 8 bytes at a time."""
import pytest

from conftest import assert_records_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(12, 31), (12, 32), (7, 32), (7, 34), (2, 62), (12, 62), (2, 64), (3, 64), (12, 66),
                                   (2, 79), (3, 95), (2, 96), (6, 96), (4, 127), (4, 128), (2, 161), (5, 193)])
def test_sizes_around_the_first_running_copies(T, O, shape):
    nocc, nvir = shape
    s = T.synth_system(nocc, nvir, seed=nocc + nvir)
    want, _, mism = O.run_system(s, "port", nthreads=4)
    assert mism == 0
    with T.Plan([s], mode=T.MODE_PLAIN) as p:
        p.upload()
        p.execute()
        assert_records_close(p.triple_energies(0), want)
