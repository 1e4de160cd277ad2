"""A call that fails for want of memory reports that and leaves nothing behind (B200 only): the same thread's next call
must not be refused for the error of the one before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fused", "plain", "emulated"])
def test_next_plan_runs_after_one_that_did_not_fit(T, mode):
    mode = {"fused": T.MODE_FUSED, "plain": T.MODE_PLAIN, "emulated": T.MODE_EMULATED}[mode]
    s = T.synth_system(3, 20, seed=4)
    want = T.run([s], mode=mode)
    huge = T.System(0, 200, 1500, 201)  # only the shape is read: 4 million triples, 1.1 TB of energy slots
    with pytest.raises(T.TrpdrvError) as e:
        T.Plan([huge], mode=T.MODE_FUSED)
    assert e.value.status == 3  # TRPDRV_ERR_NOMEM
    assert np.array_equal(T.run([s], mode=mode), want)
    assert T.cbody(s, 2, 1, 1, 1) == T.cbody(s, 2, 1, 1, 1)
