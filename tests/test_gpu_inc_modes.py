"""Modes per CTA of the increment solve (channel_flow_gb300/csrc/
k_solve_mixed.cu: inc_modes), as chf_tuning reports them."""
import pytest

from channel_flow_gb300 import Channel, config

pytestmark = pytest.mark.gpu


def modes(g):
    return int(g.tuning().split("increment solve ")[1].split()[0])


@pytest.mark.parametrize("nnz", [32, 216])
def test_back_to_the_rule(chflow_lib, nnz):
    cfg = config.small(nnx=16, nny=12, nnz=nnz, aphi=1.0, beta=1.0, dt=1e-4, re=180.0, re_p=1.0)
    with Channel(cfg, precision="mixed") as g:
        rule = modes(g)
        for m in (2, 4):
            g.set_launch_shape("inc_modes", m)
            assert modes(g) == m
        g.set_launch_shape("inc_modes", 6 - rule)
        g.set_launch_shape("inc_modes", 0)
        assert modes(g) == rule
