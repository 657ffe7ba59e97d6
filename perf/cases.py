"""Timed cases of the channel-flow library: what a DNS program has it do.

A program creates a channel (or an ensemble), loads a state and then calls
the time step over and over, with the statistics in between.  The cases are
those calls, at the sizes of the repository's own workloads
(channel_flow_gb300.config.CONFIGS), their ragged neighbours and their
precisions:

  kind "step"     Channel.step(steps): the resident time step, chf_step
  kind "host"     Channel.step_host(steps): the step of a driver whose arrays
                  live in (page-locked) host memory, chf_step_host
  kind "batch"    Batch.step(steps) of an ensemble of channels, chf_batch_step
  kind "monitor"  what a program prints between steps: diagnostics,
                  statistics and CFL numbers

States are seeded: a laminar or wall-law mean profile with a divergence-free
perturbation in every resolved mode, exponentially decaying over the
spectrum, that satisfies the wall conditions, and histories of the size that
advection by the mean gives them, as a restarted run has.
"""
import math

import numpy as np
import torch

from channel_flow_gb300 import Batch, Channel
from channel_flow_gb300.config import ChannelConfig

FIELDS = ("vnp1", "omegaynp1", "unp1", "wnp1", "omegaxnp1", "omegaznp1", "rhsvn", "rhsomegayn")
MEANS = ("clamb1n", "clamb1nm1", "clamb3n", "clamb3nm1", "au0", "w0")


def _smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


def _exact_grid(nnz):
    """The smallest product grid in z that dealiases exactly."""
    m = 3 * nnz // 2 + 1
    while not _smooth(2 * m):
        m += 1
    return m


def _case(name, kind, precision, nnx, nny, nnz, steps, aphi=1.0, beta=0.5, dt=2e-4, re=180.0, re_p=1.0,
          exact_zpad=True, amp=0.1, channels=0):
    return {"name": name, "kind": kind, "precision": precision, "nnx": nnx, "nny": nny, "nnz": nnz,
            "steps": steps, "aphi": aphi, "beta": beta, "dt": dt, "re": re, "re_p": re_p,
            "zpad": _exact_grid(nnz) if exact_zpad else 0, "amp": amp, "channels": channels}


def listed():
    box = {"aphi": 2.0, "beta": 2.0 / 3.0}
    return [
        # the Orr-Sommerfeld box, a driver that calls one step at a time: all launches and latency
        _case("os_16x65x4_fp64_1", "step", "fp64", 16, 4, 64, 1, beta=1.0, dt=1e-3, re=7500.0, re_p=2.0 / 7500.0,
              exact_zpad=False, amp=0.01),
        # the 32^3 Poiseuille box, ten steps between outputs, in the two precisions a small run uses
        _case("poiseuille_32_fp64", "step", "fp64", 32, 32, 32, 10, dt=1e-3, re=2000.0, re_p=1e-3,
              exact_zpad=False, amp=0.02),
        _case("poiseuille_32_mixed", "step", "mixed", 32, 32, 32, 10, dt=1e-3, re=2000.0, re_p=1e-3,
              exact_zpad=False, amp=0.02),
        # ragged grids: lines of 144 and 108 points, 81 planes, the reference's own product grid
        _case("ragged_96x81x72_fp64", "step", "fp64", 96, 72, 80, 4, exact_zpad=False, amp=0.05),
        # lines of 240 and 180 points, 97 planes
        _case("ragged_160x97x120_mixed", "step", "mixed", 160, 120, 96, 4, amp=0.05),
        # the Re_tau 180 channel in every precision
        _case("retau180_128_mixed", "step", "mixed", 128, 128, 128, 4, **box),
        _case("retau180_128_f64solve", "step", "mixed_fp64solve", 128, 128, 128, 2, **box),
        _case("retau180_128_fp64", "step", "fp64", 128, 128, 128, 2, **box),
        # the Re_tau 550 channel, the largest
        _case("retau550_384_mixed", "step", "mixed", 384, 384, 192, 2, dt=5e-5, re=550.0, amp=0.1),
        # an ensemble of small channels at different Reynolds numbers on two grids
        _case("ensemble_24_mixed", "batch", "mixed", 64, 64, 64, 10, amp=0.1, channels=24),
        # the reference driver's structure: host arrays up and down every step
        _case("host_128_mixed", "host", "mixed", 128, 128, 128, 1, **box),
        # what is printed between steps
        _case("monitor_128", "monitor", "fp64", 128, 128, 128, 1, **box),
    ]


_COST = {"fp64": 10.0, "mixed_fp64solve": 2.5, "mixed": 1.0}  # time per grid point, mixed = 1
_PLANE = [n for n in range(12, 321, 4) if _smooth(3 * n // 2)]
_WALL = [n for n in range(12, 201, 2) if _smooth(2 * n)]


def _near(rng, sizes, lo, hi):
    """One of `sizes`, spread over the logarithm of lo .. hi."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(sizes, key=lambda n: abs(n - x))


def draw(rng):
    kind = rng.choice(["step"] * 7 + ["batch", "host", "monitor"])
    precision = rng.choice(["fp64", "mixed", "mixed", "mixed_fp64solve"])
    if kind in ("batch",):
        precision = rng.choice(["mixed", "mixed_fp64solve"])
    while True:
        top = 64 if kind == "batch" else 320
        nnx, nny = _near(rng, _PLANE, 12, top), _near(rng, _PLANE, 12, top)
        nnz = _near(rng, _WALL, 16, 96 if kind == "batch" else 200)
        points = nnx * nny * (nnz + 1)
        steps = 1 if kind in ("host", "monitor") else rng.choice([1, 2, 4, 10])
        channels = rng.choice([4, 8, 16]) if kind == "batch" else 0
        if points * _COST[precision] * steps * max(1, channels) <= 4e7 and points <= 8e6:
            break
    n = max(nnx, nny, nnz)
    return _case("", kind, precision, nnx, nny, nnz, steps, aphi=rng.choice([1.0, 1.5, 2.0]),
                 beta=rng.choice([0.5, 2.0 / 3.0, 1.0]), dt=2e-4 * min(1.0, (96.0 / n) ** 2),
                 re=round(rng.uniform(100.0, 400.0), 1), exact_zpad=rng.random() < 0.5, amp=0.05, channels=channels)


# --------------------------------------------------------------------------
# states
# --------------------------------------------------------------------------
def _config(case, re=None, nnx=None, nny=None, nnz=None):
    return ChannelConfig(nnx or case["nnx"], nny or case["nny"], nnz or case["nnz"], case["aphi"], case["beta"],
                         case["dt"], re or case["re"], case["re_p"])


def _zpad(case, cfg):
    return _exact_grid(cfg.nnz) if case["zpad"] else 0


def _wavenumbers(cfg, dev):
    a = torch.arange(cfg.nnx // 2, dtype=torch.float64, device=dev) / cfg.aphi
    j = torch.arange(cfg.nny, dtype=torch.float64, device=dev)
    b = torch.where(j <= cfg.nny // 2, j, j - cfg.nny) / cfg.beta
    return a[None, None, :], b[None, :, None]


def _cos_matrix(points, coefs, intervals, dev):
    """T_n(z_p) = cos(pi n p / intervals), p < points, n < coefs."""
    p = torch.arange(points, device=dev)[:, None] * torch.arange(coefs, device=dev)[None, :]
    return torch.cos(math.pi * (p % (2 * intervals)).double() / intervals)


def _derivative(nz, dev):
    """d/dz of a Chebyshev series of nz + 1 coefficients."""
    i, j = torch.arange(nz + 1, device=dev)[:, None], torch.arange(nz + 1, device=dev)[None, :]
    D = torch.where((j > i) & ((i + j) % 2 == 1), 2.0 * j.double(), torch.zeros((), dtype=torch.float64, device=dev))
    D[0] *= 0.5
    return D


def _times(M, f):
    """A real matrix times a complex field along its first axis."""
    r = torch.view_as_real(f.contiguous()).reshape(f.shape[0], -1)
    return torch.view_as_complex((M @ r).reshape(M.shape[0], *f.shape[1:], 2))


def _wall_series(nz, ncoef, power, dev):
    """Column j: the Chebyshev series of (1 - z^2)^power T_j."""
    from numpy.polynomial import chebyshev
    B = np.zeros((nz + 1, ncoef))
    wall = [0.5, 0.0, -0.5] if power == 1 else list(chebyshev.chebmul([0.5, 0.0, -0.5], [0.5, 0.0, -0.5]))
    for j in range(ncoef):
        c = chebyshev.chebmul(wall, [0.0] * j + [1.0])
        B[:len(c), j] = c
    return torch.from_numpy(B).to(dev)


def _state(cfg, seed, amp):
    """The 8 fields (complex, on the GPU) and 6 mean arrays of a restart."""
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(seed)
    N, KX, KY = cfg.nnz, cfg.nnx // 2, cfg.nny
    nyq = KY // 2
    al, be = _wavenumbers(cfg, dev)
    k2 = al * al + be * be
    ncoef = max(2, min(N // 2, N - 4))
    jx = torch.arange(KX, device=dev)[None, None, :].double() / KX
    jy = torch.arange(KY, device=dev).double()
    jy = (torch.minimum(jy, KY - jy) / nyq)[None, :, None]
    decay = torch.exp(-9.0 * torch.sqrt(jx * jx + jy * jy)) \
        * torch.exp(-9.0 * torch.arange(ncoef, device=dev).double() / ncoef)[:, None, None]

    def series(power):
        c = torch.randn((ncoef, KY, KX), dtype=torch.complex128, device=dev, generator=g) * decay
        f = _times(_wall_series(N, ncoef, power, dev), c)
        f[:, nyq] = 0.0
        f[:, 0, 0] = 0.0
        if KY > 2:  # a real field: kx = 0 modes satisfy f(-ky) = conj f(ky)
            f[:, nyq + 1:, 0] = torch.conj(torch.flip(f[:, 1:nyq, 0], dims=(1,)))
        return f

    v, oy = series(2), series(1)
    D, T0 = _derivative(N, dev), _cos_matrix(N + 1, N + 1, N, dev)
    u, w, ox, oz = _recover(v, oy, al, be, k2, D)
    # mean profile: laminar, or a flat turbulent one at the larger Reynolds number
    zc = torch.zeros(N + 1, dtype=torch.float64, device=dev)
    lam = cfg.re * cfg.re_p / 2.0
    uc = lam if lam <= 2.0 else 2.5 * math.log(cfg.re) + 5.5
    if cfg.re >= 500.0 and lam > 2.0:
        z = np.cos(np.pi * np.arange(N + 1) / N)
        c = np.polynomial.chebyshev.chebfit(z, uc * (1.0 - z ** 8), 8)
        c[1::2] = 0.0
        zc[:9] = torch.from_numpy(c).to(dev)
    else:
        zc[0], zc[2] = 0.5 * uc, -0.5 * uc
    ms = sum(float((torch.abs(_times(T0, f)) ** 2).sum()) for f in (u, v, w)) / (N + 1)
    scale = amp * uc / math.sqrt(max(ms, 1e-300) / 3.0)
    for f in (v, oy, u, w, ox, oz):
        f *= scale
    u[:, 0, 0] = zc.to(torch.complex128)
    oz[:, 0, 0] = -(D @ zc).to(torch.complex128)
    # histories at the Gauss-Lobatto points: advection by the mean profile
    adv = -1j * al * (0.5 * uc)
    rv = adv * _times(T0, _times(D @ D, v) - k2 * v)
    rg = adv * _times(T0, oy)
    rv[:, nyq] = 0.0
    rg[:, nyq] = 0.0
    fields = dict(zip(FIELDS, (v, oy, u, w, ox, oz, rv, rg)))
    zero = torch.zeros((N + 1, 2), dtype=torch.float64, device=dev)
    means = {k: zero.clone() for k in MEANS}
    means["clamb1n"][:, 0] = means["clamb1nm1"][:, 0] = -cfg.re_p
    means["au0"][:, 0] = zc
    return fields, means


class _Device:
    """A resident field as an array for torch; it keeps its owner alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


def _fields(ch, owner, views):
    """The channel's resident fields as torch tensors (no copies)."""
    import ctypes
    out = []
    p = ctypes.c_void_p()
    for i in range(len(FIELDS)):
        ch._check(ch.L.chf_device_field(ch.h, i, ctypes.byref(p)))
        t = views.get((id(ch), p.value))
        if t is None:
            t = torch.as_tensor(_Device(owner, p.value, ch.shape), device="cuda")
            views[(id(ch), p.value)] = t
        out.append(t)
    return out


def _load(ch, owner, cfg, seed, amp, views):
    fields, means = _state(cfg, seed, amp)
    ch.upload_state({k: m.cpu().numpy() for k, m in means.items()})
    for t, name in zip(_fields(ch, owner, views), FIELDS):
        t.copy_(torch.view_as_real(fields[name]).reshape(t.shape))


def _members(case, seed):
    """The ensemble: half of the channels on the case's grid, half on one of
    three quarters of its wall-normal points, Reynolds numbers spread."""
    r = np.random.default_rng(seed)
    small = min(_WALL, key=lambda n: abs(n - 3 * case["nnz"] / 4))
    return [_config(case, re=float(r.uniform(100.0, 300.0)), nnz=case["nnz"] if i % 2 == 0 else small)
            for i in range(case["channels"])]


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "steps": case["steps"], "views": {}}
    if kind == "batch":
        cfgs = _members(case, seed)
        b = Batch(cfgs, precision=case["precision"], zpad=[_zpad(case, c) for c in cfgs])
        s = torch.cuda.Stream()
        for i, c in enumerate(cfgs):
            _load(b[i], b, c, seed + 1000 * (i + 1), case["amp"], state["views"])
            b[i].set_stream(s.cuda_stream)
        state.update(batch=b, stream=s)
    else:
        cfg = _config(case)
        ch = Channel(cfg, precision=case["precision"], zpad=case["zpad"])
        state["channel"] = ch
        if kind == "host":
            fields, means = _state(cfg, seed, case["amp"])
            host = {}
            for k, f in list(fields.items()) + list(means.items()):
                f = torch.view_as_real(f).reshape(ch.shape) if f.is_complex() else f
                p = torch.empty(f.shape, dtype=torch.float64, pin_memory=True)
                p.copy_(f)
                host[k] = p.numpy()
            state["host"] = host
        else:
            _load(ch, ch, cfg, seed, case["amp"], state["views"])
    torch.cuda.synchronize()
    return state


def run(state):
    kind = state["kind"]
    if kind == "host":
        return state["channel"].step_host(state["host"], state["steps"])
    if kind == "batch":
        b = state["batch"]
        b.step(state["steps"])
        with torch.cuda.stream(state["stream"]):  # the ensemble's state, one array per field
            each = [_fields(ch, b, state["views"]) for ch in b.channels]
            return [torch.cat([f[i].reshape(-1) for f in each]) for i in range(len(FIELDS))]
    ch = state["channel"]
    if kind == "monitor":
        d, s, c = ch.diagnostics(), ch.statistics(), ch.cfl()
        return {"diagnostics": d, "statistics": s, "cfl": c}
    ch.step(state["steps"])
    return _fields(ch, ch, state["views"])


def _step_work(cfg, zpad):
    KX, KY, NZ, MP = cfg.nnx // 2, cfg.nny, cfg.nnz + 1, (zpad or 2 * cfg.nnz) + 1
    PX, PY = 3 * cfg.nnx // 2, 3 * cfg.nny // 2
    modes = KX * KY
    al = np.arange(KX)[None, :] / cfg.aphi
    j = np.arange(KY)
    be = (np.where(j <= KY // 2, j, j - KY) / cfg.beta)[:, None]
    groups = len(np.unique(al * al + be * be))
    blocks = 2 * ((NZ // 2 + 1) ** 2 + (NZ // 2) ** 2)  # the even and odd inverses of v and omega_y
    # fields in and out, and each inverse once
    nbytes = 16 * 16.0 * NZ * modes + 8.0 * groups * blocks
    lg = lambda n: 5.0 * n * math.log2(n)  # noqa: E731
    # nine fields through z, y and x on the product grid, the two Gauss-Lobatto
    # transforms, the products, and per mode the four block products (re, im)
    flops = (9 * modes * lg(MP) + 2 * modes * lg(NZ) + 9.0 * MP * (KX * lg(PY) + PY * lg(PX) / 2)
             + 15.0 * MP * PX * PY + 4.0 * modes * blocks)
    return nbytes, flops


def work(case):
    cfg = _config(case)
    kind = case["kind"]
    field = 16.0 * (cfg.nnz + 1) * cfg.nny * (cfg.nnx // 2)
    if kind == "monitor":
        n = cfg.nnx * cfg.nny * (cfg.nnz + 1)
        return {"bytes": 6.0 * field, "flops": 3 * 2.5 * n * math.log2(n) + 20.0 * n}
    if kind == "batch":
        each = [_step_work(c, _zpad(case, c)) for c in _members(case, 0)]
        out = (sum(e[0] for e in each), sum(e[1] for e in each))
    else:
        out = _step_work(cfg, case["zpad"])
    return {"bytes": case["steps"] * out[0] + (16.0 * field if kind == "host" else 0.0), "flops": case["steps"] * out[1]}


# --------------------------------------------------------------------------
# the same in 64 bits with torch alone: dense wall-normal matrices, torch.fft
# in the plane, dense inverses of the collocation operators
# --------------------------------------------------------------------------
def _recover(v, oy, al, be, k2, D):
    k2 = torch.where(k2 == 0.0, torch.ones_like(k2), k2)
    dv = _times(D, v)
    u = (1j * al * dv - 1j * be * oy) / k2
    w = (1j * be * dv + 1j * al * oy) / k2
    return u, w, _times(D, w) - 1j * be * v, -_times(D, u) + 1j * al * v


def _lamb(cfg, f, MZ, al, be, D):
    """Chebyshev coefficients of the Lamb vector's three components."""
    dev = "cuda"
    KX, KY, N, MP = cfg.nnx // 2, cfg.nny, cfg.nnz, MZ + 1
    PX, PY, nyq = 3 * cfg.nnx // 2, 3 * cfg.nny // 2, cfg.nny // 2
    T1 = _cos_matrix(MP, N + 1, MZ, dev)
    vals = [_times(T1, f[k]) for k in ("unp1", "vnp1", "wnp1", "omegaxnp1", "omegaynp1", "omegaznp1")]
    out = [torch.empty((MP, KY, KX), dtype=torch.complex128, device=dev) for _ in range(3)]
    chunk = max(1, int(2e8 // (PX * PY)))
    for p in range(0, MP, chunk):
        phys = []
        for x in vals:
            x = x[p:p + chunk]
            pad = torch.zeros((x.shape[0], PY, KX), dtype=torch.complex128, device=dev)
            pad[:, :nyq] = x[:, :nyq]
            pad[:, PY - nyq + 1:] = x[:, nyq + 1:]
            pad = torch.fft.ifft(pad, dim=1, norm="forward")
            pad[:, :, 0].imag.zero_()
            phys.append(torch.fft.irfft(pad, n=PX, dim=2, norm="forward"))
        u, v, w, ox, oy, oz = phys
        for i, h in enumerate((oy * w - cfg.re_p - oz * v, oz * u - ox * w, ox * v - oy * u)):
            s = torch.fft.fft(torch.fft.rfft(h, dim=2, norm="forward")[:, :, :KX], dim=1, norm="forward")
            out[i][p:p + chunk, :nyq + 1] = s[:, :nyq + 1]
            out[i][p:p + chunk, nyq + 1:] = s[:, PY - nyq + 1:]
    W = _cos_matrix(N + 1, MP, MZ, dev) * (2.0 / MZ)
    W[:, 0] *= 0.5
    W[:, MZ] *= 0.5
    W[0] *= 0.5
    return [_times(W, h) for h in out]


def _operators(cfg, k2u, T, dev):
    """Inverses of the collocation operators of v and omega_y at each k^2."""
    T0, T2, T4 = T
    N, s = cfg.nnz, cfg.dt * 0.5 / cfg.re
    j = torch.arange(N + 1, device=dev).double()
    sign = 1.0 - 2.0 * (j % 2)
    k = k2u[:, None, None]
    A = -s * T4 + (1.0 + 2.0 * k * s) * T2 - k * (1.0 + k * s) * T0
    A[:, 0], A[:, 1], A[:, N - 1], A[:, N] = torch.ones_like(j), j * j, -sign * j * j, sign
    B = -s * T2 + (1.0 + k * s) * T0
    B[:, 0], B[:, N] = torch.ones_like(j), sign
    return torch.linalg.inv(A), torch.linalg.inv(B)


def _exact_steps(cfg, zpad, mixed, fields, means, steps):
    dev = "cuda"
    f, m = dict(fields), dict(means)
    N, KX, KY = cfg.nnz, cfg.nnx // 2, cfg.nny
    nyq, dt = KY // 2, cfg.dt
    al, be = _wavenumbers(cfg, dev)
    k2 = al * al + be * be
    D = _derivative(N, dev)
    D2 = D @ D
    T0 = _cos_matrix(N + 1, N + 1, N, dev)
    T = (T0, T0 @ D2, T0 @ (D2 @ D2))
    k2u, group = torch.unique(k2.reshape(-1), return_inverse=True)
    modes = KX * KY
    live = torch.ones((KY, KX), dtype=torch.bool, device=dev)
    live[nyq] = False
    live[0, 0] = False
    live = live.reshape(-1)
    s = dt * 0.5 / cfg.re
    for _ in range(steps):
        H1, H2, H3 = _lamb(cfg, f, zpad or 2 * N, al, be, D)
        hv = k2 * H2 + _times(D, 1j * al * H1 + 1j * be * H3)
        hg = 1j * al * H3 - 1j * be * H1
        for name, h in (("clamb1n", H1), ("clamb3n", H3)):
            m[name + "m1"] = m[name]
            m[name] = torch.view_as_real(T0.to(torch.complex128) @ h[:, 0, 0]).contiguous()
        hv[:, 0, 0] = 0.0
        hg[:, 0, 0] = 0.0
        if not mixed:
            f["omegaxnp1"], f["omegaznp1"] = H1.clone(), H3.clone()
        old_v, old_g = f["rhsvn"], f["rhsomegayn"]
        f["rhsvn"], f["rhsomegayn"] = _times(T0, hv), _times(T0, hg)
        del H1, H2, H3, hv, hg
        # right-hand sides at the Gauss-Lobatto points, wall rows zero
        v, oy = f["vnp1"], f["omegaynp1"]
        rhs_v = (s * _times(T[2], v) + (1.0 - 2.0 * k2 * s) * _times(T[1], v) - k2 * (1.0 - k2 * s) * _times(T0, v)
                 + dt * (1.5 * f["rhsvn"] - 0.5 * old_v))
        rhs_g = s * _times(T[1], oy) + (1.0 - k2 * s) * _times(T0, oy) + dt * (1.5 * f["rhsomegayn"] - 0.5 * old_g)
        rhs_v[:2], rhs_v[N - 1:], rhs_g[:1], rhs_g[N:] = 0.0, 0.0, 0.0, 0.0
        rhs_v = rhs_v.reshape(N + 1, modes).t().contiguous()
        rhs_g = rhs_g.reshape(N + 1, modes).t().contiguous()
        vn, gn = v.reshape(N + 1, modes).clone(), oy.reshape(N + 1, modes).clone()
        order = torch.argsort(group)
        order = order[live[order]]
        size = max(1, int(4e8 // ((N + 1) ** 2)))
        for lo in range(0, order.numel(), size):
            i = order[lo:lo + size]
            g0, g1 = int(group[i[0]]), int(group[i[-1]])
            Av, Ag = _operators(cfg, k2u[g0:g1 + 1], T, dev)
            at = group[i] - g0
            for inv, rhs, dst in ((Av, rhs_v, vn), (Ag, rhs_g, gn)):
                x = torch.bmm(inv[at], torch.view_as_real(rhs[i]))
                dst[:, i] = torch.view_as_complex(x.contiguous()).t()
            del Av, Ag
        f["vnp1"], f["omegaynp1"] = vn.reshape(N + 1, KY, KX), gn.reshape(N + 1, KY, KX)
        u, w, ox, oz = _recover(f["vnp1"], f["omegaynp1"], al, be, k2, D)
        mask = live.reshape(1, KY, KX)
        f["unp1"], f["wnp1"] = torch.where(mask, u, old_v), torch.where(mask, w, old_g)
        f["omegaxnp1"] = torch.where(mask, ox, f["omegaxnp1"])
        f["omegaznp1"] = torch.where(mask, oz, f["omegaznp1"])
        # the (0,0) mode
        _, A0 = _operators(cfg, torch.zeros(1, dtype=torch.float64, device=dev), T, dev)
        for mean, now, vel, vort, sg in (("au0", "clamb1n", "unp1", "omegaznp1", -1.0),
                                         ("w0", "clamb3n", "wnp1", "omegaxnp1", 1.0)):
            r = s * (T[1] @ m[mean]) + T0 @ m[mean] - 0.5 * dt * (3.0 * m[now] - m[now + "m1"])
            r[0], r[N] = 0.0, 0.0
            m[mean] = (A0[0] @ r).contiguous()
            f[vel][:, 0, 0] = torch.view_as_complex(m[mean])
            f[vort][:, 0, 0] = torch.view_as_complex((sg * (D @ m[mean])).contiguous())
    return f, m


def _exact_monitor(cfg, f, m):
    dev = "cuda"
    N, KX, KY, nyq = cfg.nnz, cfg.nnx // 2, cfg.nny, cfg.nny // 2
    keep = torch.ones(KY, dtype=torch.bool, device=dev)
    keep[nyq] = False
    six = [torch.view_as_real(f[k][:, keep]) for k in FIELDS[:6]]
    au0 = m["au0"][:, 0]
    n = torch.arange(N + 1, device=dev).double()
    top, bottom = float((n * n * au0).sum()), float(((2.0 * (n % 2) - 1.0) * n * n * au0).sum())
    diag = {"energy": 0.5 * sum(float((six[i] ** 2).sum()) for i in (2, 0, 3)), "wall_shear_top": top,
            "wall_shear_bottom": bottom, "max_abs": max(float(x.abs().max()) for x in six), "finite": True}
    T0 = _cos_matrix(N + 1, N + 1, N, dev)
    gl = [_times(T0, f[k]) for k in ("unp1", "vnp1", "wnp1")]
    z = torch.cos(math.pi * n / N)
    wt = torch.full((1, KY, KX), 2.0, dtype=torch.float64, device=dev)
    wt[:, :, 0] = 1.0
    wt[:, nyq] = 0.0
    total = sum((wt * torch.abs(x) ** 2).sum() for x in gl)
    wt[:, 0, 0] = 0.0
    cov = lambda a, b: (wt * (a * b.conj()).real).sum(dim=(1, 2)).cpu().numpy()  # noqa: E731
    U, V, W = gl
    um = U[:, 0, 0].real
    ut, ub = math.sqrt(abs(top / cfg.re)), math.sqrt(abs(bottom / cfg.re))
    even = n % 2 == 0
    half = range(N // 2, N)
    stats = {"u_tau_top": ut, "u_tau_bottom": ub, "re_tau_top": ut * cfg.re, "re_tau_bottom": ub * cfg.re,
             "re_centre": float(um[N // 2]) * cfg.re,
             "re_bulk": 2.0 * cfg.re * sum(float(um[k] * abs(z[k + 1] - z[k])) for k in half),
             "bulk_velocity": float((au0[even] / (1.0 - n[even] ** 2)).sum()),
             "energy": 0.5 * cfg.nnx * cfg.nny * float(total)}
    stats.update(z=z.cpu().numpy(), u=um.cpu().numpy(), v=V[:, 0, 0].real.cpu().numpy(), w=W[:, 0, 0].real.cpu().numpy(),
                 uu=cov(U, U), vv=cov(V, V), ww=cov(W, W), uv=cov(U, V), uw=cov(U, W), vw=cov(V, W))
    dy = torch.zeros(N + 1, dtype=torch.float64, device=dev)
    for k in range(1, N // 2 + 1):
        dy[k] = dy[N - k] = math.cos((k - 1) * math.pi / N) - math.cos(k * math.pi / N)
    peak = []
    for x in gl:
        x = x.clone()
        x[:, nyq] = 0.0
        x = torch.fft.ifft(x, dim=1, norm="forward")
        x[:, :, 0].imag.zero_()
        peak.append(torch.fft.irfft(x, n=cfg.nnx, dim=2, norm="forward").abs().amax(dim=(1, 2)))
    cfl = {"cfl_x": float(peak[0].max()) * cfg.dt / (2 * math.pi * cfg.aphi / cfg.nnx),
           "cfl_y": float((peak[1][1:N] / dy[1:N]).max()) * cfg.dt,
           "cfl_z": float(peak[2].max()) * cfg.dt / (2 * math.pi * cfg.beta / cfg.nny)}
    return {"diagnostics": diag, "statistics": stats, "cfl": cfl}


def _real(f):
    return torch.view_as_real(f.contiguous()).reshape(f.shape[0], f.shape[1], -1)


def exact(case, seed):
    mixed = case["precision"] != "fp64"
    if case["kind"] == "batch":
        each = []
        for i, c in enumerate(_members(case, seed)):
            f, m = _state(c, seed + 1000 * (i + 1), case["amp"])
            f, _ = _exact_steps(c, _zpad(case, c), mixed, f, m, case["steps"])
            each.append([_real(f[k]).reshape(-1) for k in FIELDS])
        return [torch.cat([e[i] for e in each]) for i in range(len(FIELDS))]
    cfg = _config(case)
    f, m = _state(cfg, seed, case["amp"])
    if case["kind"] == "monitor":
        return _exact_monitor(cfg, f, m)
    f, m = _exact_steps(cfg, case["zpad"], mixed, f, m, case["steps"])
    if case["kind"] == "host":
        out = {k: _real(f[k]).cpu().numpy() for k in FIELDS}
        out.update({k: m[k].cpu().numpy() for k in MEANS})
        return out
    return [_real(f[k]) for k in FIELDS]
