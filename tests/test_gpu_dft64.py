"""The FP64 transforms as exact digit products (channel_flow_gb300/csrc/k_dft64.cu).

Against the oracle at the sizes where their tiles and steps can go wrong: the
smallest lines, output counts and k counts on both sides of a multiple of 8
and 16, an odd product grid, lines of more than 128 k (summed in two
segments), and lines on both sides of the longest that take this path (384 in
x and y, 512 in z), the other directions then still on it.
The bar is the FP64 path's own (1e-10, raised to 4x the oracle's
rounding-level spread where an array is ill-conditioned; 1e-7 for the plane
averages); above 128 wall-normal intervals, where the oracle itself is off by
more, an extended-precision evaluation takes its place.

A power-of-two factor on the whole state only moves the lines' exponents, so
the Lamb vector's histories scale by its square bit for bit.  Non-finite
values must stay visible."""
import numpy as np
import pytest

from channel_flow_gb300 import Channel, config, fields
from exact_lamb import nonlinear_histories
from parity import check, oracle_sensitivity, rel_l2, split

# digit bounds on the CPU ---------------------------------------------------


def digits(x):
    """Eight balanced base-256 digits of an integer below 2^62, top first, as
    the kernel cuts them."""
    y = x + 0x8080808080808080
    return [((y >> (8 * (7 - p))) & 0xff) - 128 for p in range(8)]


def test_digits_are_exact_and_level_sums_fit():
    rng = np.random.default_rng(0)
    xs = [0, 1, -1, 2**62, -2**62, 2**62 - 1, 128, -128, 127, 2**61] + \
        [int(v) for v in rng.integers(-2**62, 2**62, 200)]
    for x in xs:
        d = digits(x)
        assert sum(v * 256 ** (7 - p) for p, v in enumerate(d)) == x
        assert max(map(abs, d)) <= 128
    # 128 k of at most 8 products per level: an FP32 integer
    assert 8 * 128 * 128 * 128 <= 2**24


# nnx, nny, nnz, zpad (0: 2 nnz)
GRIDS = [(4, 4, 4, 0), (12, 20, 10, 16), (20, 40, 24, 0), (32, 60, 32, 50), (40, 36, 48, 75), (64, 24, 30, 48),
         (8, 8, 180, 288), (256, 4, 6, 0), (4, 256, 6, 0), (288, 8, 12, 0), (8, 288, 12, 20), (8, 8, 160, 512),
         (8, 8, 160, 540)]


def cfg_of(nnx, nny, nnz, re_p=1.0):
    return config.small(nnx=nnx, nny=nny, nnz=nnz, aphi=1.0, beta=0.5, dt=1e-4, re=180.0, re_p=re_p)


@pytest.mark.gpu
@pytest.mark.parametrize("nnx,nny,nnz,zpad", GRIDS)
def test_nonlinear_against_the_oracle(chflow_lib, oracle_mod, nnx, nny, nnz, zpad):
    cfg = cfg_of(nnx, nny, nnz)
    st = fields.reference_like_state(cfg, seed=5, epsilon=0.3, noise=0.02, gamma=5.0)
    o = oracle_mod.Oracle.from_config(cfg)
    o.setup()
    o.set_state(st)
    o.getnonlinear()
    with Channel(cfg, zpad=zpad) as g:
        g.upload_state(st)
        g.getnonlinear()
        out = g.download_state()
    ref = o.get_state()
    if nnz > 128:
        # the oracle's own histories are 1e-8 and more from exact on these
        # tall grids (the curl's derivative multiplies the products' rounding
        # by 2 nnz): held to an extended-precision evaluation instead, where
        # the digits have to be at least as accurate as the oracle
        for k, ex in zip(("rhsvn", "rhsomegayn"), nonlinear_histories(cfg, st)):
            e_g = rel_l2(split(out[k], k)[k], split(ex, k)[k])
            e_o = rel_l2(split(ref[k], k)[k], split(ex, k)[k])
            assert e_g <= max(e_o, 1e-12), (k, e_g, e_o)
        return
    check(out, ref, 1e-10, 1e-7, lambda: oracle_sensitivity(oracle_mod, cfg, st, lambda q: q.getnonlinear()))


@pytest.mark.gpu
@pytest.mark.parametrize("power", [-100, 100])
def test_powers_of_two_are_exact(chflow_lib, power):
    cfg = cfg_of(24, 20, 16, re_p=0.0)
    st = fields.reference_like_state(cfg, seed=8, epsilon=0.3, noise=0.02, gamma=5.0)
    big = {k: v * 2.0**power for k, v in st.items()}
    got = []
    for s in (st, big):
        with Channel(cfg) as g:
            g.upload_state(s)
            g.getnonlinear()
            got.append(g.download_state())
    for k in ("rhsvn", "rhsomegayn", "clamb1n", "clamb3n"):
        assert np.array_equal(got[0][k] * 4.0**power, got[1][k]), k


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_non_finite_values_stay_visible(chflow_lib, value):
    cfg = cfg_of(16, 8, 16)
    st = fields.reference_like_state(cfg, seed=8, epsilon=0.3, noise=0.02, gamma=5.0)
    st["vnp1"][3, 2, 4] = value
    with Channel(cfg) as g:
        g.upload_state(st)
        g.step(2)
        out = g.download_state()
        assert not g.diagnostics()["finite"]
    assert not np.isfinite(out["rhsvn"]).all() and not np.isfinite(out["unp1"]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("nnx,nny,nnz", [(16, 8, 16), (24, 12, 18), (36, 60, 20), (108, 20, 12), (12, 180, 30)])
def test_laminar_flow_stays_laminar(chflow_lib, nnx, nny, nnz):
    """Lines constant in x, y or z leak nothing into their other modes: a
    mean flow alone leaves every other mode exactly zero."""
    cfg = cfg_of(nnx, nny, nnz)
    st = fields.laminar_state(cfg, gamma=1.7)
    with Channel(cfg) as g:
        g.upload_state(st)
        g.getnonlinear()
        out = g.download_state()
    for k in ("rhsvn", "rhsomegayn"):
        assert not np.any(out[k]), k
    for k in ("omegaxnp1", "omegaznp1"):  # H1, H3 are left there; the mean mode's H1 holds -re_p
        assert not np.any(out[k][:, 1:, :]) and not np.any(out[k][:, 0, 2:]), k


@pytest.mark.gpu
@pytest.mark.parametrize("nnx,nny,nnz", [(4, 4, 4), (20, 36, 10), (60, 100, 32), (384, 12, 8), (12, 384, 250), (96, 64, 128)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_physical_velocity_equals_the_transform(chflow_lib, nnx, nny, nnz, precision):
    """The unpadded digit products (physical velocity, CFL numbers) against the
    FFT passes of chf_transform, which take one field at a time.  An FFT's
    rounding is at most a few ulp a stage of the line's norm, three lines in
    turn: 1e-12 of the largest value covers 30 stages."""
    cfg = config.small(nnx=nnx, nny=nny, nnz=nnz, aphi=1.0, beta=0.5, dt=1e-4, re=180.0, re_p=1.0)
    st = fields.reference_like_state(cfg, seed=2, epsilon=0.3, noise=0.02, gamma=3.0)
    with Channel(cfg, precision=precision) as g:
        g.upload_state(st)
        got = g.physical_velocity()
        ref = [g.transform(1, st[k]) for k in ("unp1", "wnp1", "vnp1")]
        cfl = g.cfl()
    for a, b in zip(got, ref):
        assert np.abs(a - b.reshape(a.shape)).max() <= 1e-12 * np.abs(b).max()
    umax = np.abs(ref[0]).max() * cfg.dt / (cfg.aphi * 2 * np.pi / nnx)
    assert abs(cfl["cfl_x"] - umax) <= 1e-12 * umax
