"""The explicit term of the FP64 solve in digits (channel_flow_gb300/csrc/
k_solve64.cu) against k_solve, which multiplies the same inverses in FP64
(CHF_MIXED_F64SOLVE keeps it, and its set-up inverts the same operators).

From a zero state v and omega_y are A^-1 r alone, so the two differ by the
roundings of that product.  Row by row, an FP64 sum of n terms a_q whose
roundings are independent and at most u = 2^-53 of a partial sum stays within
8 standard deviations, 8 u sqrt(n) |a|_2; two of them (and the roundings of r,
formed in both ways) give the bound below.  The digits have to be inside it
too, at wavenumbers up to the largest here, where the columns of A^-1 that
belong to the wall rows exceed the others a thousandfold and more and must not
take the row's bits: they meet zeros."""
import numpy as np
import pytest

from channel_flow_gb300 import Channel, config, fields

pytestmark = pytest.mark.gpu


def inverse_blocks(cfg, k2):
    """{(v?, even?): A^-1} of the operators, for the sizes of their rows."""
    N, dt, re = cfg.nnz, cfg.dt, cfg.re
    n, p = np.arange(N + 1), np.arange(N + 1)
    t0 = np.cos(np.pi * np.outer(p, n) / N)
    cheb = np.polynomial.chebyshev
    der = [t0]
    for k in (2, 4):
        m = np.zeros_like(t0)
        for j in n:
            c = cheb.chebder(np.eye(N + 1)[j], k)
            m[:, j] = t0[:, :len(c)] @ c
        der.append(m)
    t0, t2, t4 = der
    a = {True: -(t4 * dt / 2 / re) + (1 + k2 * dt / re) * t2 - k2 * (1 + k2 * dt / 2 / re) * t0,
         False: -(t2 * dt / 2 / re) + (1 + k2 * dt / 2 / re) * t0}
    out = {}
    for isv in (True, False):
        for par in (0, 1):
            j = np.arange(par, N + 1, 2)
            m = a[isv][:len(j), j].copy()
            m[0] = 1.0
            if isv:
                m[1] = j.astype(float) ** 2
            out[isv, par] = np.linalg.inv(m)
    return out


# nnx, nny, nnz, aphi, beta: k^2 up to 1e3, 3e4 and 1e5; 16 t + 1 rows in even blocks, 16 t in both, 16 t + 9
@pytest.mark.parametrize("nnx,nny,nnz,aphi,beta", [(48, 48, 128, 1.0, 0.5), (36, 40, 96, 0.1, 0.15), (48, 40, 48, 0.07, 0.1)])
def test_explicit_term_keeps_its_bits(chflow_lib, nnx, nny, nnz, aphi, beta):
    cfg = config.small(nnx=nnx, nny=nny, nnz=nnz, aphi=aphi, beta=beta, dt=2e-4, re=180.0, re_p=1.0)
    st = {k: np.zeros_like(v) for k, v in fields.laminar_state(cfg, gamma=1.0).items()}
    rng = np.random.default_rng(7)
    for k in ("rhsvn", "rhsomegayn", "unp1", "wnp1"):  # N^n and N^{n-1}
        st[k] = rng.standard_normal(st[k].shape)
    got = {}
    for precision in ("fp64", "mixed_fp64solve"):
        with Channel(cfg, precision=precision) as g:
            if precision == "fp64":
                assert g.kernels_per_step() >= 13  # the digit solve
            g.upload_state(st)
            g.solve()
            got[precision] = g.download_state()
    N, u = nnz, 2.0**-53
    worst = 0.0
    for ky in (0, 1, nny // 2 - 1):
        for kx in (0, 1, nnx // 2 - 1):
            k2 = (kx / aphi) ** 2 + (ky / beta) ** 2
            if k2 == 0.0:
                continue
            for (isv, par), x in inverse_blocks(cfg, k2).items():
                now, old = (("rhsvn", "unp1") if isv else ("rhsomegayn", "wnp1"))
                name, wall, n = ("vnp1", 2, len(x)) if isv else ("omegaynp1", 1, len(x))
                for c in (2 * kx, 2 * kx + 1):
                    h = cfg.dt * (1.5 * st[now][:, ky, c] - 0.5 * st[old][:, ky, c])
                    r = 0.5 * (h[:n] + (-1) ** par * h[N - np.arange(n)])
                    # |terms| also of the two points and histories that a row of r sums
                    a = cfg.dt * (1.5 * np.abs(st[now][:, ky, c]) + 0.5 * np.abs(st[old][:, ky, c]))
                    a = 0.5 * (a[:n] + a[N - np.arange(n)])
                    a[:wall] = r[:wall] = 0.0
                    bound = 16 * u * np.sqrt(n) * np.sqrt((x ** 2) @ (a ** 2))
                    both = [got[p][name][par::2, ky, c] for p in ("fp64", "mixed_fp64solve")]
                    assert np.abs(both[1] - x @ r).max() <= 1e-6 * np.abs(both[1]).max()  # the operator meant here
                    worst = max(worst, (np.abs(both[0] - both[1]) / bound).max())
    assert worst <= 1.0, worst
