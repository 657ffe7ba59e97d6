"""The autotuner on CHF_FP64 grids whose lines go through digit products
(channel_flow_gb300/csrc/chf_tune.cu, k_dft64.cu): the radices and lines per CTA
of FFT kernels that no step launches are neither timed and chosen nor reported;
lines past the digits' range keep them."""
import pytest

from channel_flow_gb300 import Channel, config, fields

pytestmark = pytest.mark.gpu


# nnx, nny, nnz, zpad; whether x / y lines (up to 384 points) and z lines (up to 512 intervals) are digits
@pytest.mark.parametrize("nnx,nny,nnz,zpad,xy,z", [(24, 12, 20, 36, True, True), (288, 8, 12, 0, False, True),
                                                   (8, 8, 160, 540, True, False)])
def test_only_what_a_step_launches(chflow_lib, nnx, nny, nnz, zpad, xy, z):
    cfg = config.small(nnx=nnx, nny=nny, nnz=nnz, aphi=1.5, beta=0.75, dt=1e-5, re=300.0, re_p=1.0)
    st = fields.reference_like_state(cfg, seed=4, epsilon=0.3, noise=0.02, gamma=5.0)
    with Channel(cfg, precision="fp64", zpad=zpad) as g:
        g.upload_state(st)
        texts = [g.tuning(), g.autotune(reps=1)]
    for text in texts:
        assert ("x / y lines as digit products" in text) == xy, text
        assert ("z lines as digit products" in text) == z, text
        for name in ("py ", "px ", "kxb ", "xr "):
            assert (name in text) != xy, (name, text)
        for name in ("pzm ", "zl_c2v ", "zl_curl "):
            assert (name in text) != z, (name, text)
        assert "pz2 " in text
