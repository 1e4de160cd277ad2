"""The emulated form's recombination (B200 only): the level sums joined in int64, in int32 pairs or one by one, by the
width of the contraction and the slices; scales as exponent additions, or as multiplications where a result might
leave the range of normal numbers.  Records against the FP64 plan at 1e-11 of a column's largest: the digits dropped by
7 slices are below 2^-49 of a row's largest element each, the products of a contraction of 832 below 832 x 2^-46."""
import numpy as np
import pytest

from conftest import assert_records_close

pytestmark = pytest.mark.gpu


def _records(T, s, **kw):
    with T.Plan([s], **kw) as p:
        p.upload()
        p.execute()
        return p.triple_energies(0)


# widths (rounded up to 32) just inside and outside the limits: 503 and 811 for 7 slices, 579 for 8
@pytest.mark.parametrize("slices,shape", [(7, (3, 477)), (7, (2, 482)), (7, (2, 766)), (7, (3, 806)),
                                          (8, (2, 542)), (8, (2, 575)), (5, (3, 806)), (4, (2, 482))])
def test_widths_at_the_limits_of_the_joined_sums(T, slices, shape):
    nocc, nvir = shape
    s = T.synth_system(nocc, nvir, seed=nvir)
    want = _records(T, s, mode=T.MODE_FUSED)
    tol = {4: 1e-5, 5: 1e-7}.get(slices, 1e-11)  # 832 x 2^-(7 S - 3)
    assert_records_close(_records(T, s, mode=T.MODE_EMULATED, slices=slices), want, rtol=tol)


@pytest.mark.parametrize("power", [400, 600, -600])
@pytest.mark.parametrize("nvir", [40, 41])
def test_extreme_scales_give_the_same_bits(T, power, nvir):
    """A operands times 2^power and B operands times 2^-power: every f is the same number."""
    s = T.synth_system(4, nvir, seed=5)
    base = _records(T, s, mode=T.MODE_EMULATED, slices=7)
    for name, sign in (("jvv", 1), ("kvv", 1), ("tov", 1), ("xov", 1), ("t2", -1), ("jov", -1), ("kov", -1)):
        s.arrays[name] = np.ldexp(s.arrays[name], sign * power)
    assert np.array_equal(_records(T, s, mode=T.MODE_EMULATED, slices=7), base)
