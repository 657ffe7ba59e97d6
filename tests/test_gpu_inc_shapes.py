"""The increment solve of the mixed path at the edges of its launch rules
(channel_flow_gb300/csrc/k_solve_mixed.cu): wall-normal sizes around 160 rows
(2 or 4 modes per CTA by the rule), around 224 rows (blocks of 224 or 256
threads), one row more than whole warps, and the largest.  Every shape gives
the same bits, and the result agrees with the FP64 solve to FP32 rounding of
the O(dt) term (1e-6 of the field's largest value)."""
import numpy as np
import pytest

from channel_flow_gb300 import Channel, config, fields
from channel_flow_gb300.fields import FIELD_NAMES, MEAN_NAMES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nnz", [6, 32, 150, 160, 216, 240, 250])
def test_shapes_and_rules(chflow_lib, nnz):
    cfg = config.small(nnx=16, nny=12, nnz=nnz, aphi=1.0, beta=1.0, dt=1e-4, re=180.0, re_p=1.0)
    st = fields.turbulent_start_state(cfg, seed=4)
    outs = []
    for shape in (None, (2, 4, 1), (4, 4, 1), (2, 3, 2), (4, 2, 2)):
        with Channel(cfg, precision="mixed") as g:
            if shape:
                g.set_launch_shape("inc_rows", 1)
                for name, value in zip(("inc_modes", "inc_columns", "inc_rows"), shape):
                    g.set_launch_shape(name, value)
            g.upload_state(st)
            g.getnonlinear()
            g.solve()
            outs.append(g.download_state())
    for out in outs[1:]:
        for k in FIELD_NAMES + MEAN_NAMES:
            assert np.array_equal(outs[0][k], out[k]), k
    with Channel(cfg, precision="fp64") as g:
        g.upload_state(st)
        g.getnonlinear()
        g.solve()
        ref = g.download_state()
    for k in ("vnp1", "omegaynp1"):
        assert np.abs(outs[0][k] - ref[k]).max() <= 1e-6 * np.abs(ref[k]).max(), k
