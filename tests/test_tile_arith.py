"""The tile walk's integer additions and quotients (fs_bits.h, the functions the
kernels compile) replayed on the host against FP64: every result they accept
must be the hardware's, on random operands and on operands next to rounding
ties, midpoints and the ends of the binades."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_accepted_results_are_fp64(tmp_path, seed):
    exe = tmp_path / "tile_arith_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    str(ROOT / "tests" / "native" / "tile_arith_check.cpp"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe), "3000000", str(seed)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "all equal to FP64" in out.stdout
