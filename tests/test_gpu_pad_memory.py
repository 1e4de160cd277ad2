"""Device memory that odd fused plans take beside their tensors (B200 only): padded copies out of plenty, none where they
would take more than a quarter of the free memory, so that an application that has planned with the rest still gets
it.  The records are the same bits either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _uploaded(T, torch, s):
    """Records, staging and the device memory that the upload took."""
    with T.Plan([s], mode=T.MODE_FUSED) as p:
        free0 = torch.cuda.mem_get_info()[0]
        p.upload()
        took = free0 - torch.cuda.mem_get_info()[0]
        p.execute()
        return p.triple_energies(0), p.staging(), took


def test_copies_only_out_of_plenty(T):
    torch = pytest.importorskip("torch")
    s = T.synth_system(13, 151, seed=13)
    padded = sum(s.arrays[n].nbytes for n in ("t2", "jvv", "kvv", "jov", "kov"))  # 41 MB, of 42 in all
    torch.cuda.init()
    _uploaded(T, torch, s)  # modules and kernels loaded
    plenty, staging, took = _uploaded(T, torch, s)
    assert staging == 1 and took >= s.nbytes() + padded
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - 160 * MB, dtype=torch.uint8, device="cuda")
    try:
        scarce, staging, took = _uploaded(T, torch, s)
        assert staging == 1 and took <= s.nbytes() + 2 * MB * len(s.arrays)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert np.array_equal(scarce, plenty)
