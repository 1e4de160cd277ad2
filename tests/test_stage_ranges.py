"""What a drop-in call sends when only some of its slices lie in registered arrays (CPU only): the pieces that are staged,
not the unused slots between them (two blocks of nvir x nvir doubles with jvv and kvv registered and t2 and tov not)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_slots_left_out_are_not_sent(tmp_path):
    exe = tmp_path / "ranges"
    subprocess.run(["gcc", "-std=c11", "-O1", "-Wall", "-Werror", "-fopenmp",
                    "-I", os.path.join(ROOT, "nwchem-ccsd-trpdrv_b200", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "stage_ranges.c")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
