"""Plain plans where a full batch of f (96 MB) does not fit in the free device memory (B200 only): smaller batches, the same
bits; one triple at a time where only that fits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _records(T, s):
    with T.Plan([s], mode=T.MODE_PLAIN) as p:
        p.upload()
        p.execute()
        return p.triple_energies(0), p.last_launches()


@pytest.mark.parametrize("nvir,left", [(200, 60), (200, 24)])  # 2.6 MB of f a triple, 40 triples, 9 MB of tensors
def test_batches_that_fit(T, nvir, left):
    torch = pytest.importorskip("torch")
    s = T.synth_system(4, nvir, seed=6)
    torch.cuda.init()
    want, launches = _records(T, s)
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - left * MB, dtype=torch.uint8, device="cuda")
    try:
        got, more = _records(T, s)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert np.array_equal(got, want) and more > launches
