"""The mesh arrays' copy over several host threads when memory runs out: no
exception leaves the C entry, and every byte is copied."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_copy_without_memory(tmp_path):
    exe, lib = str(tmp_path / "copy"), os.path.join(ROOT, "libfive_b200", "lib")
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-I" + os.path.join(ROOT, "include"),
                        os.path.join(ROOT, "tests", "capi", "copy_without_memory.cpp"), "-o", exe,
                        "-L" + lib, "-lfive", "-Wl,-rpath," + lib, "-pthread"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
