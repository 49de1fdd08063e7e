"""CPU-side checks of the look-back records: their fields against the words that
the atomics set, and the width in which the kernels read them."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gpz_b200", "csrc")


def test_fields_lie_in_single_words(tmp_path):
    exe = tmp_path / "look_check"
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC,
                    "-I", os.path.join(ROOT, "include"), "-o", str(exe),
                    os.path.join(ROOT, "tests", "host", "look_check.cu")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "bad=0" in out.stdout


def test_relaxed_loads_have_the_width_of_the_atomics():
    """A vector load is one access per element, in no order: its elements must be
    as wide as the words that `red ... .b64` sets."""
    src = "".join(open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cuh", ".cu")))
    widths = {int(w) for w in re.findall(r'"red\.relaxed\.gpu\.global\.or\.b(\d+)', src)}
    loads = re.findall(r'"ld\.relaxed\.gpu\.global\.(?:v\d\.)?[bu](\d+)', src)
    assert widths == {64} and loads
    assert all(int(w) == 64 for w in loads), loads
