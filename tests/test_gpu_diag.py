"""k_diag (channel_flow_gb300/csrc/k_solve.cu): the largest magnitude exactly, the
energy to rounding, and the spanwise Nyquist slot left out, on grids of one and
several CTAs along the modes and of fewer planes than CTAs along them."""
import numpy as np
import pytest

from channel_flow_gb300 import Channel, config, fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nnx,nny,nnz", [(4, 4, 4), (12, 20, 8), (32, 36, 16), (64, 64, 30)])
def test_diagnostics(chflow_lib, nnx, nny, nnz):
    cfg = config.small(nnx=nnx, nny=nny, nnz=nnz, aphi=1.0, beta=0.5, dt=1e-4, re=180.0, re_p=1.0)
    st = fields.reference_like_state(cfg, seed=5, epsilon=0.3, noise=0.02, gamma=3.0)
    rng = np.random.default_rng(0)
    six = ("unp1", "vnp1", "wnp1", "omegaxnp1", "omegaynp1", "omegaznp1")
    for k in six:
        st[k] = rng.standard_normal(st[k].shape)
        st[k][:, nny // 2] = 1e3  # the unused slot
    used = np.arange(nny) != nny // 2
    with Channel(cfg) as g:
        g.upload_state(st)
        d = g.diagnostics()
        assert d["finite"]
        assert d["max_abs"] == max(np.abs(st[k][:, used]).max() for k in six)
        energy = 0.5 * sum((st[k][:, used] ** 2).sum() for k in six[:3])
        assert abs(d["energy"] - energy) <= 1e-13 * energy  # sums of positive terms
        st["omegaznp1"][nnz // 2, 0, 1] = np.inf
        g.upload_state(st)
        assert not g.diagnostics()["finite"]
