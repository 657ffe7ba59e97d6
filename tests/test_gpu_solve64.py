"""The FP64 solve as exact digit products (channel_flow_gb300/csrc/k_solve64.cu).

Grids with enough modes for it (more of k_solve's CTAs than SMs) and
block sizes at its edges: 16 t + 1 rows (last row and column outside the
tiles) in the even or the odd blocks, 16 t, 16 t + 9, one tile with few rows,
and more than 64 rows (two pairs of columns per lane); k^2 groups of 1, 2 and
more than 4 modes.  One solve from a state with histories and non-zero wall
values against the oracle, to the FP64 path's bar (1e-10; v's operator is
ill-conditioned above 128 wall-normal intervals, 1e-8 there as in the parity
tests)."""
import numpy as np
import pytest

from channel_flow_gb300 import Channel, config, fields
from parity import check, oracle_sensitivity

pytestmark = pytest.mark.gpu

# nnx, nny, nnz, aphi, beta
GRIDS = [(64, 40, 4, 1.0, 0.5), (64, 64, 16, 1.0, 1.0), (48, 48, 32, 1.0, 0.5), (40, 64, 50, 1.3, 0.7),
         (60, 48, 64, 2.0, 0.5), (48, 64, 128, 2.0, 2.0 / 3.0), (64, 36, 160, 1.0, 0.5)]


@pytest.mark.parametrize("nnx,nny,nnz,aphi,beta", GRIDS)
def test_solve_against_the_oracle(chflow_lib, oracle_mod, nnx, nny, nnz, aphi, beta):
    cfg = config.small(nnx=nnx, nny=nny, nnz=nnz, aphi=aphi, beta=beta, dt=1e-4, re=180.0, re_p=1.0)
    st = fields.reference_like_state(cfg, seed=6, epsilon=0.3, noise=0.02, gamma=5.0)
    rng = np.random.default_rng(2)
    for k in ("rhsvn", "rhsomegayn", "unp1", "wnp1"):  # N^n and N^{n-1} as getnonlinear leaves them
        st[k] = rng.standard_normal(st[k].shape)
    o = oracle_mod.Oracle.from_config(cfg)
    o.setup()
    o.set_state(st)
    o.solve()
    with Channel(cfg) as g:
        assert g.kernels_per_step() >= 13  # solve, recovery and (0,0) mode apart: this path
        g.upload_state(st)
        g.solve()
        out = g.download_state()
    check(out, o.get_state(), 1e-10 if nnz <= 128 else 1e-8, 1e-7,
          lambda: oracle_sensitivity(oracle_mod, cfg, st, lambda q: q.solve()))


def test_non_finite_history_stays_visible(chflow_lib):
    cfg = config.small(nnx=64, nny=40, nnz=16, aphi=1.0, beta=0.5, dt=1e-4, re=180.0, re_p=1.0)
    st = fields.reference_like_state(cfg, seed=6, epsilon=0.3, noise=0.02, gamma=5.0)
    for value in (np.inf, np.nan):
        bad = {k: v.copy() for k, v in st.items()}
        bad["rhsvn"][5, 3, 4] = value
        with Channel(cfg) as g:
            g.upload_state(bad)
            g.solve()
            out = g.download_state()
            assert not g.diagnostics()["finite"]
        assert not np.isfinite(out["vnp1"][:, 3, 4:6]).all()
        assert np.isfinite(out["vnp1"][:, 4, 4:6]).all()  # the other modes are not touched
