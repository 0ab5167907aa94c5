"""The look-back words of the single-pass kernels (dcsr_b200/csrc/lookback.cuh),
compiled with nvcc and run on the CPU (tests/cpp/lookback_words_test.cu)."""
import os
import subprocess

from dcsr_b200 import build as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_lookback_words(tmp_path):
    exe = str(tmp_path / "lookback_words_test")
    subprocess.run([B.nvcc(), *B.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I" + B.CSRC,
                    os.path.join(ROOT, "tests", "cpp", "lookback_words_test.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    assert out.stdout.strip() == "ok"
