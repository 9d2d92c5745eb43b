"""Who writes which word of a staged tile along the box (mg_tile_box.cuh, the
kernels' own code compiled for the host): one writer between two barriers."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_one_writer_between_barriers(tmp_path):
    exe = tmp_path / "staging"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fno-strict-aliasing", "-Wno-unknown-pragmas",
                    "-I" + os.path.join(ROOT, "basilisk_b200", "csrc"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "tile_staging.cpp")], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
