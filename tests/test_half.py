"""The halved k = 0 rows of the derivative recurrences.  bits::half
(channel_flow_gb300/csrc/f64bits.cuh) against x * 0.5: infinities and NaN must not
come out finite; magnitudes below 2^-1021 stay what they are.  On the device, a NaN
among the odd coefficients of v has to be seen in row 0 of the mode's recovered u
and w (k_inc_recover64)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from channel_flow_gb300 import Channel, config, fields

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "f64bits.cuh"
using namespace chf::bits;
int main() {
  std::mt19937_64 rng(3);
  for (int i = 0; i < 1000000; ++i) {
    uint64_t u = rng();
    if (i % 4 == 1) u &= 0x801fffffffffffffull;  // exponents 0 and 1
    if (i % 4 == 2) u |= 0x7ff0000000000000ull;  // NaN
    if (i % 64 == 2) u &= 0xfff0000000000000ull;  // infinities
    const double x = u2d(u), a = half(x), b = std::fabs(x) < std::ldexp(1.0, -1021) ? x : x * 0.5;
    if (std::isnan(b) ? !std::isnan(a) : d2u(a) != d2u(b)) {
      std::printf("half(%a) = %a, not %a\n", x, a, b);
      return 1;
    }
  }
  return 0;
}
"""


def test_half_is_the_product_by_one_half(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src, exe = str(tmp_path / "half.cpp"), str(tmp_path / "half")
    with open(src, "w") as f:
        f.write(SOURCE)
    inc = os.path.join(HERE, "..", "channel_flow_gb300", "csrc")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I" + inc, "-o", exe, src], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nnx,nny", [(64, 40), (8, 8)])  # the digit solve and its recovery; k_solve
def test_nan_reaches_row_zero(chflow_lib, nnx, nny, precision):
    cfg = config.small(nnx=nnx, nny=nny, nnz=16, aphi=1.0, beta=0.5, dt=1e-4, re=180.0, re_p=1.0)
    st = fields.reference_like_state(cfg, seed=6, epsilon=0.3, noise=0.02, gamma=5.0)
    st["vnp1"][5, 3, 4:6] = np.nan  # an odd coefficient of v: D v is even
    with Channel(cfg, precision=precision) as g:
        g.set_launch_shape("recover_form", 0)
        g.upload_state(st)
        g.solve()
        out = g.download_state()
    for k in ("unp1", "wnp1"):
        assert np.isnan(out[k][0, 3, 4:6]).all(), k
        assert np.isfinite(out[k][:, 4, 4:6]).all(), k
