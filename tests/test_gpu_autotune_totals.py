"""Autotuning a plan leaves the totals of its last execution alone (B200 only): trpdrv_plan_energies returns the same bits
before and after, and zeros where nothing has been executed.  The emulated form with target_digits samples records
with several numbers of slices, whose totals differ from those of the execution."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(T, mode, **kw):
    return T.Plan([T.synth_system(7, 64, seed=62), T.synth_system(4, 32, seed=63)], mode=mode, **kw)


@pytest.mark.parametrize("digits", [0, 8])
def test_totals_of_the_last_execution_survive_autotune(T, digits):
    modes = [(T.MODE_EMULATED, {"target_digits": digits})] + ([(T.MODE_FUSED, {})] if digits == 0 else [])
    for mode, kw in modes:
        with _plan(T, mode, **kw) as p:
            p.upload()
            p.execute()
            before = np.array(p.energies())
            p.autotune()
            assert np.array_equal(np.array(p.energies()), before)


@pytest.mark.parametrize("digits", [0, 8])
def test_autotune_alone_leaves_no_totals(T, digits):
    with _plan(T, T.MODE_EMULATED, target_digits=digits) as p:
        p.upload()
        p.autotune()
        assert not np.array(p.energies()).any()
