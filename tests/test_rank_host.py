"""CPU-side check of the encoder's ranking: its window, exchange steps and limits
(shared with the kernel), compiled for the host and compared with a plain sort."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_ranking_on_host(tmp_path):
    exe = tmp_path / "rank_check"
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", os.path.join(ROOT, "gpz_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    "-o", str(exe), os.path.join(ROOT, "tests", "host", "rank_check.cu")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "bad=0" in out.stdout
