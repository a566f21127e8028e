"""The check that ends a render whose paths were lost, over sequences of round counters."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_round_progress(tmp_path):
    exe = str(tmp_path / "round_progress")
    subprocess.run(["/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++", "-std=c++17", "-O1", "-Wall", "-Werror",
                    "-I", os.path.join(ROOT, "gianduia_b200", "csrc", "cuda"),
                    os.path.join(ROOT, "tests", "cpp", "round_progress.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], timeout=20).returncode == 0
