"""Drop-in calls, which run the plain kernels, against the fused kernel's records of the same triples (B200 only): the two
share no product or energy code.  Bar as between the two paths elsewhere: 1e-12 of the largest total."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nocc,nvir", [(8, 64), (5, 33), (7, 80)])
@pytest.mark.parametrize("path", [None, "plain"])
def test_dropin_calls_agree_with_the_fused_kernel(T, monkeypatch, nocc, nvir, path):
    if path:
        monkeypatch.setenv("TRPDRV_DROPIN_PATH", path)
    s = T.synth_system(nocc, nvir, seed=91)
    with T.Plan([s], mode=T.MODE_FUSED, nkpass=3) as p:
        p.upload()
        p.execute()
        rec, ijk = p.triple_energies(0), p.triples(0)
    klo = {tuple(r[:3]): int(r[3]) for r in T.enumerate_triples(nocc, 3)}  # k-chunked: klo > 1 for most triples
    for t in range(0, len(ijk), 17):
        i, j, k = (int(v) for v in ijk[t])
        e4, e5 = T.cbody(s, i, j, k, klo[i, j, k], emp4=0.5, emp5=-0.25)
        w4 = 0.5 + rec[t, 0] + (rec[t, 2] if i != k else 0.0)
        w5 = -0.25 + rec[t, 1] + (rec[t, 3] if i != k else 0.0)
        assert abs(e4 - w4) <= 1e-12 * (abs(w4) + 1.0) and abs(e5 - w5) <= 1e-12 * (abs(w5) + 1.0)
