"""A plan of more systems than a grid has rows (65,535): every system's records and totals (B200 only).  The systems
share their device tensors and differ in the virtual index a."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,nocc,nvir", [("plain", 2, 4), ("fused", 1, 2)])
def test_more_systems_than_grid_rows(T, mode, nocc, nvir):
    import torch
    n = 65535 + 3
    mode = {"plain": T.MODE_PLAIN, "fused": T.MODE_FUSED}[mode]
    s = T.synth_system(nocc, nvir, seed=9)
    other = T.synth_system(nocc, nvir, seed=9, a=s.a + 1)
    t = {k: torch.from_numpy(v).cuda() for k, v in s.arrays.items()}
    ptrs = {k: v.data_ptr() for k, v in t.items()}
    want = []
    for q in (s, other):
        with T.Plan([q], mode=mode) as p:
            p.bind_device([ptrs])
            p.execute()
            want.append([float(x[0]) for x in p.energies()] + [p.triple_energies(0)])
    with T.Plan([s] * (n - 1) + [other], mode=mode, use_graph=0) as p:
        p.bind_device([ptrs] * n)
        p.execute()
        e4, e5 = p.energies()
        first, last = p.triple_energies(0), p.triple_energies(n - 1)
    assert np.all(e4[:-1] == want[0][0]) and np.all(e5[:-1] == want[0][1])
    assert e4[-1] == want[1][0] and e5[-1] == want[1][1]
    assert np.array_equal(first, want[0][2]) and np.array_equal(last, want[1][2])
