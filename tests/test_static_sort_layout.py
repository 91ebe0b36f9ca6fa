"""The static sort's scratch layout, checked by the compiler (no GPU needed):
every look-back word of a digit pass ends before the spare keys begin."""
import os
import subprocess

from merge_fusion_gb300 import build


def test_lookback_words_end_before_the_spare_keys(tmp_path):
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp", "static_sort_layout.cu")
    cmd = [build.nvcc()] + build.NVCC_FLAGS + ["-c", src, "-o", str(tmp_path / "layout.o")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
