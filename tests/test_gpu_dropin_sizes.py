"""The drop-in bodies at sizes their staging and tiles distinguish (B200 only): odd rows (padded in the staging
block), one and several tiles, slices larger than one transfer segment, calls in a k loop (only the k role
changes) and shapes that alternate.  Double precision against the oracle at 1e-11 of the call's magnitude; the
single-precision library against the same double-precision oracle at 2e-4 of the largest call (the bar of its
parity tests)."""
import ctypes as C
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (2, 15), (3, 17), (5, 32), (4, 33), (7, 63), (6, 64), (3, 97), (9, 130)]


def _k_loop(nocc):
    """(i, j, k, klo) of the reference driver's k loop for two (i, j)."""
    return [(i, j, k, 1 + (k > 2)) for i, j in ((nocc, 1), (1, nocc)) for k in range(1, i + 1)]


@pytest.mark.parametrize("shape", SHAPES)
def test_double_body_matches_the_oracle(T, O, shape):
    nocc, nvir = shape
    s = T.synth_system(nocc, nvir, seed=40 * nocc + nvir, ncor=nvir % 2)
    port = O.port_body_fn()
    for t in _k_loop(nocc):
        got, want = T.cbody(s, *t), T.body_call(port, s, *t)
        for g, w in zip(got, want):
            assert abs(g - w) <= 1e-11 * max(abs(want[0]), abs(want[1])), (t, got, want)


def test_alternating_shapes_and_large_slices(T, O):
    port = O.port_body_fn()
    systems = [T.synth_system(2, 301, seed=5), T.synth_system(3, 40, seed=6), T.synth_system(2, 301, seed=7)]
    for rep in range(2):
        for s in systems:
            for t in ((2, 1, 1, 1), (2, 1, 2, 1)):
                got, want = T.cbody(s, *t), T.body_call(port, s, *t)
                for g, w in zip(got, want):
                    assert abs(g - w) <= 1e-11 * max(abs(want[0]), abs(want[1])), (rep, t, got, want)


def _fp32_body(T):
    lib = C.CDLL(os.path.join(os.path.dirname(T.LIB_PATH), "libtrpdrv_b200_fp32.so"))
    fn = lib.ccsd_trpdrv_omp_cbody_
    fn.restype = None
    return fn


def _fp32_call(T, fn, s, f32, i, j, k, klo):
    s32 = T.System(s.ncor, s.nocc, s.nvir, s.a, f32)
    sl = T.triple_slices(s32, i, j, k, klo)
    fp = C.POINTER(C.c_float)
    f = np.zeros((8, s.nvir * s.nvir), dtype=np.float32)
    ints = [C.c_int(v) for v in (s.ncor, s.nocc, s.nvir)]
    idx = [C.c_int(v) for v in (s.a, i, j, k, klo)]
    e4, e5 = C.c_float(0.0), C.c_float(0.0)
    fn(*[f[q].ctypes.data_as(fp) for q in range(8)], f32["eorb"].ctypes.data_as(fp), *[C.byref(v) for v in ints],
       C.byref(e4), C.byref(e5), *[C.byref(v) for v in idx], *[sl[n].ctypes.data_as(fp) for n in T.BODY_ORDER])
    return e4.value, e5.value


@pytest.mark.parametrize("shape", SHAPES + [(2, 260)])
def test_float_body_matches_the_double_oracle(T, O, shape):
    nocc, nvir = shape
    s = T.synth_system(nocc, nvir, seed=90 * nocc + nvir, ncor=nvir % 2)
    f32 = {n: np.ascontiguousarray(a.astype(np.float32)) for n, a in s.arrays.items()}
    port, fn = O.port_body_fn(), _fp32_body(T)
    calls = _k_loop(nocc)
    got = np.array([_fp32_call(T, fn, s, f32, *t) for t in calls])
    want = np.array([T.body_call(port, s, *t) for t in calls])
    assert np.all(np.abs(got - want) <= 2e-4 * np.max(np.abs(want), axis=0)), (got, want)
