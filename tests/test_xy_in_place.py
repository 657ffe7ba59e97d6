"""The in-place x / y transforms (channel_flow_gb300/csrc/k_xy.cu).

CPU: the place and twiddle indices of fft_place_tables, restated here, give
NumPy's DFT for mixed radix orders.  GPU: a mixed step through the in-place
kernels equals the same step through the two-buffer kernels (a launch shape
set by name) bit for bit, since the stages, butterflies and twiddles are the
same and only their storage differs; line lengths cover every radix, last
radices on both sides of the fused products (up to 5, and 9), partial tiles
of modes and of rows, and packed planes."""
import numpy as np
import pytest

from channel_flow_gb300 import Channel, config, fields


def in_place_dft(x, radices):
    L = len(x)
    a = np.array(x, complex)
    Ns = 1
    for s, R in enumerate(radices):
        LO = L // (Ns * R)
        for hi in range(Ns):
            jm, h = 0, hi
            for i in range(s - 1, -1, -1):
                jm += (h % radices[i]) * int(np.prod(radices[:i], dtype=int))
                h //= radices[i]
            for lo in range(LO):
                at = hi * R * LO + lo + LO * np.arange(R)
                v = a[at] * np.exp(-2j * np.pi * np.arange(R) * jm / (Ns * R))
                a[at] = np.exp(-2j * np.pi * np.outer(np.arange(R), np.arange(R)) / R) @ v
        Ns *= R
    out = np.empty(L, complex)
    for k in range(L):
        at, n = 0, 1
        for R in radices:
            at += (k // n % R) * (L // (n * R))
            n *= R
        out[k] = a[at]
    return out


@pytest.mark.parametrize("radices", [(16, 9, 4), (16, 3), (9, 4, 3), (8, 9), (16, 3, 5), (3, 2), (2, 3, 4, 5)])
def test_place_tables_give_the_dft(radices):
    rng = np.random.default_rng(7)
    n = int(np.prod(radices))
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    # a DFT of length <= 576 in FP64: a few ulps per stage, relative to the line's norm
    assert np.abs(in_place_dft(x, radices) - np.fft.fft(x)).max() < 1e-13 * np.linalg.norm(x) * np.sqrt(n)


# nnx, nny, nnz: PX and PY = 6..576 (radices 3.2 | 8.9 | 16.3 | 16.9 | 9.4.5 | 16.9.4 ...); the
# second and third rows have planes enough for the in-place x kernel (32 rows per SM)
GRIDS = [(4, 4, 4), (32, 32, 16), (20, 72, 10), (160, 120, 6),
         (12, 384, 16), (48, 96, 24), (96, 72, 32), (160, 120, 30), (384, 64, 54), (20, 60, 60), (576, 120, 20),
         (24, 96, 32), (120, 64, 32)]  # the last two: an odd number of last butterflies


@pytest.mark.gpu
@pytest.mark.parametrize("nnx,nny,nnz", GRIDS)
def test_in_place_equals_two_buffer(chflow_lib, nnx, nny, nnz):
    cfg = config.small(nnx=nnx, nny=nny, nnz=nnz, aphi=1.0, beta=0.5, dt=1e-4, re=180.0, re_p=1.0)
    st = fields.turbulent_start_state(cfg, seed=9)
    rng = np.random.default_rng(3)
    for k in fields.FIELD_NAMES[:6]:  # every mode, so that no input slot is zero by chance
        st[k] = st[k] + 1e-3 * rng.standard_normal(st[k].shape)
    got = []
    for shape in (None, "xr"):
        with Channel(cfg, precision="mixed") as g:
            if shape:
                g.set_launch_shape(shape, 1)
            g.upload_state(st)
            g.step(2)
            got.append(g.download_state())
    for k in got[0]:
        assert np.array_equal(got[0][k], got[1][k]), k
    assert np.isfinite(got[0]["rhsvn"]).all() and np.abs(got[0]["rhsvn"]).max() > 0
