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
        g.set_launch_shape("inc_modes", 0)  # the handle may start from a cached choice
        rule = modes(g)
        for m in (2, 4):
            g.set_launch_shape("inc_modes", m)
            assert modes(g) == m
        g.set_launch_shape("inc_modes", 6 - rule)
        g.set_launch_shape("inc_modes", 0)
        assert modes(g) == rule


# square boxes fill the runs of four (n2 / n4 = 1.97 and 1.89), 4 pi x 4/3 pi does not (1.24 and 1.14)
@pytest.mark.parametrize("nnx,nny,nnz,box,want", [
    (128, 128, 128, (1.0, 1.0), 4), (128, 128, 144, (1.0, 1.0), 4), (128, 128, 128, (2.0, 2 / 3), 2),
    (128, 128, 180, (2.0, 2 / 3), 2), (128, 128, 192, (2.0, 2 / 3), 4), (128, 128, 120, (2.0, 2 / 3), 4),
    (32, 32, 180, (2.0, 2 / 3), 2), (32, 32, 180, (1.0, 1.0), 4), (32, 32, 32, (1.0, 1.0), 2)])
def test_rule(chflow_lib, nnx, nny, nnz, box, want):
    cfg = config.small(nnx=nnx, nny=nny, nnz=nnz, aphi=box[0], beta=box[1], dt=1e-4, re=180.0, re_p=1.0)
    with Channel(cfg, precision="mixed") as g:
        g.set_launch_shape("inc_modes", 0)  # the handle may start from a cached choice
        assert modes(g) == want
