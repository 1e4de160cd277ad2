"""The pinned lines that plans share for their totals (host.c, res_take): every plan reads its own, whatever lives beside
it, also after lines were given back and taken again, after trpdrv_finalize and from several threads; plans of more
systems than the shared block holds pin their own.  Pinning memory per plan doubled the creation of small ones."""
import os
import re
import threading

import numpy as np
import pytest

from conftest import ROOT


def test_creating_a_plan_pins_no_memory_of_its_own():
    with open(os.path.join(ROOT, "nwchem-ccsd-trpdrv_b200", "csrc", "host.c")) as f:
        src = f.read()
    build = src[src.index("static int plan_build("):]
    build = build[:build.index("\n}\n")]
    assert not re.search(r"cudaHostRegister|cudaMallocHost|cudaHostAlloc", build)


def _plan(T, seed, n=1):
    s = T.synth_system(3, 18, seed=seed)
    p = T.Plan([s] * n, mode=T.MODE_FUSED)
    p.upload()
    p.execute()
    return p


@pytest.mark.gpu
def test_plans_side_by_side_and_reused_lines(T):
    want = {}
    for seed in range(6):
        with _plan(T, seed) as p:
            want[seed] = np.array(p.energies())
    assert len({w.tobytes() for w in want.values()}) == 6
    plans = [(seed, _plan(T, seed)) for seed in range(6)]
    for q in (4, 1):  # two holes, taken again by smaller and larger plans
        plans.pop(q)[1].close()
    plans += [(2, _plan(T, 2)), (5, _plan(T, 5))]
    wide = _plan(T, 3, n=40)  # 161 doubles
    large = _plan(T, 4, n=1100)  # 4,401 doubles: more than the shared block
    T.finalize()  # gives nothing back that a plan uses
    plans.append((0, _plan(T, 0)))
    for seed, p in plans:
        assert np.array_equal(np.array(p.energies()), want[seed])
    assert np.array_equal(np.array(wide.energies()), np.repeat(want[3], 40, axis=1))
    assert np.array_equal(np.array(large.energies()), np.repeat(want[4], 1100, axis=1))
    for p in [p for _, p in plans] + [wide, large]:
        p.close()
    T.finalize()
    with _plan(T, 1) as p:
        assert np.array_equal(np.array(p.energies()), want[1])


@pytest.mark.gpu
def test_never_executed_plans_read_zeros_on_reused_lines(T):
    with _plan(T, 1) as p:
        p.energies()
    with T.Plan([T.synth_system(3, 18, seed=1)], mode=T.MODE_FUSED) as p:
        assert not np.array(p.energies()).any()


@pytest.mark.gpu
def test_threads_with_plans_of_their_own(T):
    want = {}
    for seed in range(4):
        with _plan(T, seed) as p:
            want[seed] = np.array(p.energies())
    bad = []

    def work(seed):
        for _ in range(20):
            with _plan(T, seed) as p:
                if not np.array_equal(np.array(p.energies()), want[seed]):
                    bad.append(seed)

    threads = [threading.Thread(target=work, args=(seed,)) for seed in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
