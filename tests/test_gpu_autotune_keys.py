"""Under which key the autotuner keeps a choice (B200 only): an a sweep apart from a single a, and no choices that a file
holds for other kernels."""
import pytest

pytestmark = pytest.mark.gpu


def test_a_sweep_and_a_single_a_are_timed_apart(T):
    one, two = T.synth_system(5, 38, seed=1), T.synth_system(5, 38, seed=1, a_count=2)
    for s in (one, two):
        with T.Plan([s], mode=T.MODE_FUSED) as p:
            p.upload()
            assert p.autotune()["from_cache"] == 0
        with T.Plan([s], mode=T.MODE_FUSED) as p:
            p.upload()
            assert p.autotune()["from_cache"] == 1


def test_choices_for_other_kernels_are_not_taken_from_the_file(T, tmp_path, monkeypatch):
    cache = tmp_path / "tune.txt"
    monkeypatch.setenv("TRPDRV_TUNE_CACHE", str(cache))

    def tune(nvir):
        with T.Plan([T.synth_system(4, nvir, seed=2)], mode=T.MODE_FUSED) as p:
            p.upload()
            return p.autotune()["from_cache"]

    assert tune(42) == 0
    line = cache.read_text().splitlines()[0]
    assert "shapes=4,42,1" in line
    key, choice = line.split(" -> ")
    version = key.split()[1]
    assert version == f"v{T.lib.trpdrv_version()}.2"
    older = key.replace(version, version.split(".")[0]).replace("4,42,1", "4,44,1").replace(" a=1", "")
    previous = key.replace(version, version[:-1] + "1").replace("4,42,1", "4,44,1")
    cache.write_text("".join(f"{k} -> {choice}\n" for k in (older, previous)))
    assert tune(44) == 0
    cache.write_text(f"{key.replace('4,42,1', '4,46,1')} -> {choice}\n")
    assert tune(46) == 2
