"""Set-up that the first statistics, CFL, physical-velocity or pressure call does
on a handle, when it fails (channel_flow_gb300/csrc/k_dft64.cu: build_tf;
chf_phys.cu: ensure_phys).  A stream under capture refuses the set-up's
synchronisation, so the call returns an error; the next one has to do the
set-up again and give what an untouched handle gives."""
import ctypes

import numpy as np
import pytest

from channel_flow_gb300 import Channel, ChannelError, config, fields

pytestmark = pytest.mark.gpu

CFG = config.small(nnx=24, nny=12, nnz=20, aphi=1.5, beta=0.75, dt=5e-4, re=300.0, re_p=1.0)
RELAXED = 2  # CU_STREAM_CAPTURE_MODE_RELAXED
CALLS = {
    "statistics": lambda g: g.statistics(),
    "cfl": lambda g: g.cfl(),
    "physical_velocity": lambda g: g.physical_velocity(),
    "pressure": lambda g: g.pressure(),
}


def flat(x):
    if isinstance(x, dict):
        return [v for k in sorted(x) for v in flat(x[k])]
    if isinstance(x, (list, tuple)):
        return [v for y in x for v in flat(y)]
    return [np.asarray(x)]


def captured(g, call):
    """call on g while its stream is being captured; the capture is dropped."""
    cu = ctypes.CDLL("libcuda.so.1")
    s, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert cu.cuStreamCreate(ctypes.byref(s), 1) == 0
    g.set_stream(s.value)
    assert cu.cuStreamBeginCapture_v2(s, RELAXED) == 0
    with pytest.raises(ChannelError):
        call(g)
    assert cu.cuStreamEndCapture(s, ctypes.byref(graph)) != 0  # invalidated: there is no graph
    assert not graph.value


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", sorted(CALLS))
def test_a_failed_first_call_is_repeated(chflow_lib, name, precision):
    st = fields.reference_like_state(CFG, seed=3, epsilon=0.3, noise=0.02, gamma=3.0)
    call = CALLS[name]
    with Channel(CFG, precision=precision) as g:
        g.upload_state(st)
        want = call(g)
        transformed = g.transform(1, st["vnp1"])
    with Channel(CFG, precision=precision) as g:
        g.upload_state(st)
        captured(g, call)
        for a, b in zip(flat(call(g)), flat(want)):
            assert np.array_equal(a, b)
        assert np.array_equal(g.transform(1, st["vnp1"]), transformed)
