"""Values around 2^-1022 in the digit products (channel_flow_gb300/csrc/
digits64.cuh, k_dft64.cu): subnormal numbers and lines whose power
of two is no double take part like all others, as they do in an FP64 FFT or
matrix product.

The physical velocity is linear in the state, so a state times 2^-1030, brought back
by 2^1030 after that rounding, gives the results to compare with.  Rounding to
the units u = 2^-1074 of a subnormal result adds u / 2 per real part and stage;
the y and x transforms sum those of KY and 2 KX values of at most sqrt(2) u / 2
of modulus."""
import numpy as np
import pytest

from channel_flow_gb300 import Channel, config, fields

pytestmark = pytest.mark.gpu

U = 2.0**-1074
TINY = 2.0**-515  # twice


def tiny_state(cfg, names):
    """A state whose arrays `names` are 2^-1030 of O(1) numbers, and the same before the factor."""
    st = {k: np.zeros_like(v) for k, v in fields.laminar_state(cfg, gamma=1.0).items()}
    rng = np.random.default_rng(11)
    big = {k: v.copy() for k, v in st.items()}
    for k in names:
        st[k] = rng.standard_normal(st[k].shape) * TINY * TINY
        big[k] = st[k] / TINY / TINY
    return st, big


def test_physical_velocity(chflow_lib):
    cfg = config.small(nnx=16, nny=12, nnz=20, aphi=1.0, beta=0.5, dt=1e-4, re=180.0, re_p=1.0)
    out = []
    for st in tiny_state(cfg, ("unp1", "vnp1", "wnp1")):
        with Channel(cfg) as g:
            g.upload_state(st)
            out.append(g.physical_velocity())
    modulus = np.sqrt(2) / 2  # of u, after z
    modulus = np.sqrt(2) * (cfg.nny * modulus) + np.sqrt(2) / 2  # after y
    bound = 2 * (cfg.nnx // 2) * modulus + 0.5
    want = out[1] * TINY * TINY
    assert np.abs(want).max() > 1e6 * bound * U  # or the test would show nothing
    assert np.abs(out[0] - want).max() <= (bound + 1) * U
