"""The fused kernel's cp.async staging and its i == k items against the oracle (B200 only).

Sizes sit at the edges of what the kernel distinguishes: 16-index chunks with one or two k-steps in either
phase, 32-wide tiles, packed edge tiles (at most 16 valid indices, three or more tiles), odd rows (read through
padded copies) and tensors that are not 16-byte aligned.  Every nocc >= 1 has triples with i == k, whose t
family is taken from the n family.  Bars as in the parity tests: 1e-11 of a column's largest record."""

import numpy as np
import pytest

from conftest import assert_records_close, assert_total_close

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 8), (2, 9), (3, 16), (3, 17), (8, 24), (9, 25), (5, 33), (2, 64), (4, 65), (7, 79), (16, 80),
          (17, 81), (6, 97)]


def _check(rec, e4, e5, want_rec, want_tot):
    assert_records_close(rec, want_rec)
    assert_total_close(e4, want_tot[0], what="emp4")
    assert_total_close(e5, want_tot[1], what="emp5")


@pytest.mark.parametrize("mma_k", [8, 4])
@pytest.mark.parametrize("shape", SHAPES)
def test_cpasync_staging_matches_the_oracle(T, O, shape, mma_k):
    nocc, nvir = shape
    s = T.synth_system(nocc, nvir, seed=1000 * nocc + nvir, ncor=nocc % 3)
    want, tot, mism = O.run_system(s, "port", nthreads=4)
    assert mism == 0
    with T.Plan([s], mode=T.MODE_FUSED, staging=T.STAGING_CPASYNC, mma_k=mma_k) as p:
        p.upload()
        p.execute()
        e4, e5 = p.energies()
        first = p.triple_energies(0)
        _check(first, e4[0], e5[0], want, tot)
        p.upload_execute(chunks=3)  # padded copies refilled span by span
        assert np.array_equal(p.triple_energies(0), first)


@pytest.mark.parametrize("shape", [(2, 10), (4, 34), (3, 33), (6, 80)])
def test_unaligned_device_tensors_match_the_oracle(T, O, shape):
    torch = pytest.importorskip("torch")
    nocc, nvir = shape
    s = T.synth_system(nocc, nvir, seed=77)
    want, tot, mism = O.run_system(s, "port", nthreads=4)
    assert mism == 0
    keep, ptrs = [], {}
    for n, name in enumerate(T.TENSOR_NAMES):
        a = s.arrays[name]
        buf = torch.zeros(a.size + 1, dtype=torch.float64, device="cuda")
        off = 1 if n % 2 else 0  # every other tensor starts 8 bytes past a 16-byte boundary
        buf[off:off + a.size] = torch.from_numpy(a).cuda()
        keep.append(buf)
        ptrs[name] = buf.data_ptr() + 8 * off
    torch.cuda.synchronize()
    with T.Plan([s], mode=T.MODE_FUSED) as p:
        p.bind_device([ptrs])
        p.execute()
        e4, e5 = p.energies()
        _check(p.triple_energies(0), e4[0], e5[0], want, tot)
        keep[T.T_T2].mul_(2.0)  # the bound tensors are read at every execution
        torch.cuda.synchronize()
        p.execute()
        assert abs(p.energies()[0][0]) > abs(e4[0])


@pytest.mark.parametrize("shape", [(2, 16), (4, 40), (8, 80), (10, 82), (6, 96)])
def test_i_equal_k_items_of_the_tma_kernel_match_the_oracle(T, O, shape):
    nocc, nvir = shape
    s = T.synth_system(nocc, nvir, seed=5 * nocc + nvir)
    want, tot, mism = O.run_system(s, "port", nthreads=4)
    assert mism == 0
    with T.Plan([s], mode=T.MODE_FUSED, staging=T.STAGING_TMA) as p:
        p.upload()
        p.execute()
        e4, e5 = p.energies()
        rec, ijk = p.triple_energies(0), p.triples(0)
    _check(rec, e4[0], e5[0], want, tot)
    same = ijk[:, 0] == ijk[:, 2]
    assert same.sum() == nocc * nocc
    assert_records_close(rec[same], want[same])
