"""CHF_FP64 on a device that its optional buffers do not fit: the solve's
operators as digits (k_solve64.cu) and the work space of the in-plane
transforms (k_dft64.cu).  The handle is created all the same and runs the
kernels that need neither, to the accuracy that both are held to against the
oracle (1e-10 each); the FP64 inverses go once the digits are cut from them.

The memory is taken by one allocation that leaves what the handle cannot do
without plus a margin, and nothing here is allocated until it fails."""
import numpy as np
import pytest

from channel_flow_gb300 import Channel, config, fields

pytestmark = pytest.mark.gpu

MB = 1 << 20
CFG = config.small(nnx=96, nny=96, nnz=128, aphi=1.3, beta=0.77, dt=1e-4, re=180.0, re_p=1.0)
KX, KY, NZ, MP, PX, PY = 48, 96, 129, 257, 144, 144
GROUPS = KX * (KY // 2) - 1  # one per (kx, |ky|) but (0, 0) in this box
FIELD = 16 * KX * KY * NZ
MUST = 8 * FIELD + 6 * 16 * MP * KX * (KY + PY)  # state, work space after the z and y transforms
INVERSES = 8 * GROUPS * 2 * (65**2 + 64**2)
DIGITS = 2 * INVERSES
PHYSICAL = 6 * 8 * MP * PX * PY
NAMES = ("vnp1", "omegaynp1", "unp1", "wnp1", "omegaxnp1", "omegaznp1")


def run():
    st = fields.reference_like_state(CFG, seed=6, epsilon=0.3, noise=0.02, gamma=5.0)
    with Channel(CFG) as g:
        kernels = g.kernels_per_step()
        g.upload_state(st)
        g.getnonlinear()
        g.solve()
        g.step(2)
        out = g.download_state()
        return kernels, [out[k] for k in NAMES] + [np.asarray(g.pressure()), np.array(list(g.cfl().values()))]


def test_digits_replace_the_inverses(chflow_lib):
    import torch
    with Channel(CFG):
        pass  # the library is loaded
    before = torch.cuda.mem_get_info()[0]
    with Channel(CFG) as g:
        assert g.kernels_per_step() == 13
        used = before - torch.cuda.mem_get_info()[0]
    assert used <= MUST + 1.03 * DIGITS + PHYSICAL + 64 * MB  # the digits' planes, exponents and edges


# margin over what the handle needs with its inverses; kernels of a step
@pytest.mark.parametrize("margin,kernels", [(400 * MB, 9), (750 * MB, 11)])
def test_little_memory(chflow_lib, margin, kernels):
    import torch
    n, want = run()
    assert n == 13
    free = torch.cuda.mem_get_info()[0]
    ballast = torch.empty(free - (MUST + INVERSES + margin), dtype=torch.uint8, device="cuda")
    try:
        n, got = run()
    finally:
        del ballast
        torch.cuda.empty_cache()
    assert n == kernels
    for a, b in zip(got, want):
        assert np.linalg.norm(a - b) <= 2e-10 * np.linalg.norm(b)
