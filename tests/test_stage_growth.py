"""Device buffers of the drop-in entry points across a failed allocation (CPU only): after one, with errors returned
to the caller, the next call must not run on a buffer that is gone."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "nwchem-ccsd-trpdrv_b200", "csrc")


def test_a_failed_growth_leaves_no_capacity_behind(tmp_path):
    exe = tmp_path / "growth"
    subprocess.run(["gcc", "-std=c11", "-O1", "-Wall", "-Werror", "-fopenmp", "-I", CSRC, "-o", str(exe),
                    os.path.join(ROOT, "tests", "stage_growth.c")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_the_fp32_library_grows_its_buffers_that_way():
    with open(os.path.join(CSRC, "fp32.cu")) as f:
        src = f.read()
    grow = re.search(r"^int grow\(.*?^}", src, re.S | re.M).group(0)
    assert "stage_grow(" in grow and "cudaMalloc" not in grow
