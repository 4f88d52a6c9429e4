"""The walk's dense lists, replayed on the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_dense_jobs_read_only_what_was_published(tmp_path):
    exe = tmp_path / "dense_slot_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "amt-bh-benchmark_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "dense_slot_check.cc"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr
