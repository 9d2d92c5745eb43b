"""A decomposed solve after one whose device allocation failed, on a fake of
the CUDA runtime (no device)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.mark.parametrize("nth", [1, 2])
def test_solve_after_a_failed_allocation(tmp_path, nth):
    exe = tmp_path / "shard"
    subprocess.run(["gcc", "-std=gnu99", "-O1", "-Wall", "-o", str(exe),
                    os.path.join(ROOT, "tests", "shard_alloc.c"),
                    os.path.join(ROOT, "basilisk_b200", "csrc", "mg_shard.c"),
                    "-I" + os.path.join(ROOT, "basilisk_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(CUDA, "include"), "-lm"], check=True)
    r = subprocess.run([str(exe), str(nth)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
