"""A quadtree refined without device memory for the records of its cycle, on a
fake of the CUDA runtime (no device)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_refine_without_memory_for_the_cycle(tmp_path):
    exe = tmp_path / "tree"
    subprocess.run(["gcc", "-std=gnu99", "-O1", "-o", str(exe), os.path.join(ROOT, "tests", "tree_alloc.c"),
                    "-I" + os.path.join(ROOT, "basilisk_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(CUDA, "include"), "-lm",
                    # (the launches, which refining does not call)
                    "-no-pie", "-Wl,--unresolved-symbols=ignore-all"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
