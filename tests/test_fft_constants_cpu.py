"""The twiddle constants of the register transforms (rdft.cuh), evaluated on the host."""

import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

SOURCE = """
#include <cstdio>
#include "rdft.cuh"
int main() {
  for (int n = 2; n <= 128; ++n)
    for (int k = 0; k < n; ++k)
      std::printf("%.17g %.17g\\n", gwb::rdft_detail::cis(k, n, 0), gwb::rdft_detail::cis(k, n, 1));
}
"""


@pytest.mark.skipif(not Path(NVCC).exists(), reason="no nvcc")
def test_constants_are_nearest(tmp_path):
    """cos and sin of 2 pi k / n for every length: within half a unit of the last place (a few thousandths more,
    where the exact value lies next to the middle of two doubles)."""
    (tmp_path / "t.cu").write_text(SOURCE)
    subprocess.run([NVCC, "-std=c++17", "-arch=sm_100a", "--expt-relaxed-constexpr", "-I", str(ROOT / "gradwave_b200/csrc"), "-o",
                    str(tmp_path / "t"), str(tmp_path / "t.cu")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout
    got = np.array([[float(x) for x in line.split()] for line in out.splitlines()])
    pi = np.longdouble("3.14159265358979323846264338327950288")
    turns = [(k, n) for n in range(2, 129) for k in range(n)]
    # the angle reduced to an eighth of a turn exactly, so that zeros and ones are exact
    for i, (k, n) in enumerate(turns):
        q = (8 * k + n) // (2 * n)
        x = pi * (4 * k - q * n) / (2 * n)
        c, s = np.cos(x), np.sin(x)
        ref = [(c, s), (-s, c), (-c, -s), (s, -c)][q % 4]
        for g, e in zip(got[i], ref):
            assert abs(np.longdouble(g) - e) <= 0.503 * np.spacing(abs(g)), (k, n, g, e)
