"""Warps some of whose lanes have no line, mode or row to store, in the kernels
whose tensor-core instructions take whole warps (ldmatrix and mma.sync in
k_dft64.cu and k_solve64.cu, tcgen05.ld in k_tcgemm.cu): the lanes leave the
stores of one tile early and have to be back for the next one.

The grids leave 2 and 6 of a warp's 8 spanwise lines, 1 or 2 of a run's 4
modes and 1 of 8 rows of the product grid to the last warps, with several tiles
per warp after them.  Results against the oracle (the FP64 path's bar; the
histories against an extended-precision evaluation, which they have to be as
close to as the oracle's, for those are up to 7e-11 off it) and the mixed paths'
(1e-5 of the velocity), and the same bits on every handle."""
import numpy as np
import pytest

from channel_flow_gb300 import Channel, config, fields
from channel_flow_gb300.fields import FIELD_NAMES, MEAN_NAMES
from exact_lamb import nonlinear_histories
from parity import bad_parts, compare, rel_l2, split

pytestmark = pytest.mark.gpu

# nnx, nny, nnz, aphi, beta: k^2 groups of 1 and 2 modes in these boxes
GRIDS = [(20, 40, 60, 1.3, 0.7), (60, 36, 72, 1.3, 0.7), (36, 20, 96, 1.7, 0.6)]
HIST = ("rhsvn", "rhsomegayn")


def advance(g, state):
    """Two steps and the nonlinear term and solve before them; the state that
    the last nonlinear term started from, and the last one."""
    g.getnonlinear()
    g.solve()
    g.step(1)
    before = state()
    g.step(1)
    return before, state()


def history_errors(cfg, before, after):
    return [rel_l2(split(after[k], k)[k], split(ex, k)[k]) for k, ex in zip(HIST, nonlinear_histories(cfg, before))]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nnx,nny,nnz,aphi,beta", GRIDS)
def test_lanes_without_work(chflow_lib, oracle_mod, nnx, nny, nnz, aphi, beta, precision):
    cfg = config.small(nnx=nnx, nny=nny, nnz=nnz, aphi=aphi, beta=beta, dt=1e-4, re=180.0, re_p=1.0)
    st = fields.reference_like_state(cfg, seed=6, epsilon=0.3, noise=0.02, gamma=5.0)
    outs = []
    for _ in range(3):
        with Channel(cfg, precision=precision) as g:
            g.upload_state(st)
            outs.append(advance(g, g.download_state))
    got = outs[0]
    for out in outs[1:]:
        for k in FIELD_NAMES + MEAN_NAMES:
            assert np.array_equal(got[1][k], out[1][k]), k
    o = oracle_mod.Oracle.from_config(cfg)
    o.setup()
    o.set_state(st)
    ref = advance(o, o.get_state)
    if precision == "fp64":
        errs = {k: e for k, e in compare(got[1], ref[1]).items() if k not in HIST}
        assert not bad_parts(errs, 1e-10, 1e-7), errs
        for e_g, e_o in zip(history_errors(cfg, *got), history_errors(cfg, *ref)):
            assert e_g <= e_o
        return
    used = np.arange(nny) != nny // 2
    err = sum(((got[1][k] - ref[1][k])[:, used] ** 2).sum() for k in ("unp1", "vnp1", "wnp1"))
    size = sum((ref[1][k][:, used] ** 2).sum() for k in ("unp1", "vnp1", "wnp1"))
    assert err <= 1e-10 * size
