"""The work a user of this package has it do, as timed cases.

Four kinds of call, each through the package's public entry points:

* ``steps``     ``Channel.step_host_ptr``: u, v, w, theta in page-locked host memory (the reference
  driver's ownership of U), n RK3 steps on the GPU, the fields back.  n = 1 is the drop-in call of a
  driver that keeps the loop; larger n is a run between two outputs.
* ``ensemble``  ``ensemble_step`` over independent channels of uneven sizes, then every channel's
  fields read back (``kmm_download_state``).
* ``adjoint``   ``control_objective`` and its ``backward``: the wall-stress objective of n steps and
  its gradients with respect to the control amplitude and the per-mode gains.
* ``blocks``    one RK3 step of a caller that holds the fields on the GPU in the reference layout:
  ``y_to_x``, ``dft_x_realspace``, ``x_to_y`` and ``wavespace`` for substeps 1 to 3.

``exact`` restates the step in plain torch with dense FP64 operators (and differentiates it for the
adjoint).  A case names its grid, box (``lx_over_pi``, ``lz_over_pi``), spline order, wall-normal map,
precision, time step (``dt`` > 0 fixed, 0 the CFL rule), control amplitude and scalars.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from channel_passive_b200 import Channel, Config, _lib
from channel_passive_b200.autograd import control_objective
from channel_passive_b200.solver import ensemble_step

RK = {"alpha": (29 / 96, -3 / 40, 1 / 6), "beta": (37 / 160, 5 / 24, 1 / 6),
      "gamma": (8 / 15, 5 / 12, 3 / 4), "zeta": (0.0, -17 / 60, -5 / 12)}
DT_START = 1e-3   # the dt a CFL run starts from (its first substep replaces it)

# the uneven ensemble of independent channels: (nx, ny, nz) and how many of each
ENSEMBLE = {"wide": (((64, 65, 64), 6), ((96, 97, 96), 6), ((128, 97, 128), 4)),
            "small": (((32, 49, 32), 3), ((64, 65, 48), 3), ((48, 65, 64), 2))}


def _case(name, kind, nx, ny, nz, **kw):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": 1, "precision": "fp64", "dt": 0.0, "cfl": 1.0,
         "control": 0.0, "scalars": 1, "labs_k": 6, "map": "sine", "stretch": 0.9, "lx_over_pi": 2.0,
         "lz_over_pi": 1.0, "re_bulk": 2800.0, "re_tau": 180.0}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    re180 = dict(lx_over_pi=4.0, lz_over_pi=4.0 / 3.0, control=-0.5, dt=0.005)
    return [
        # the smallest call: one step of a test-sized channel, where launches and latency count (a
        # Reynolds number that this grid resolves, so that any number of steps stays bounded)
        _case("tiny_fp64_step", "steps", 16, 33, 16, re_bulk=200.0),
        # the plain Re_tau 180 small channel: no control, fixed time step
        _case("small_fp64_20", "steps", 64, 65, 64, steps=20, dt=0.01),
        # a member of the ensemble alone: mixed precision, control, the CFL time step
        _case("medium_mixed_cfl_10", "steps", 96, 97, 96, steps=10, precision="mixed", control=-0.5),
        # the benchmark grid with opposition control, a stretch of the run between two outputs
        _case("re180_mixed_20", "steps", 192, 129, 192, steps=20, precision="mixed", **re180),
        _case("re180_fp64_20", "steps", 192, 129, 192, steps=20, **re180),
        # the same grid under a host driver that keeps U and asks for one step at a time
        _case("re180_mixed_host_step", "steps", 192, 129, 192, precision="mixed", **re180),
        # grids off the tuned sizes: padded lengths with a factor 5, kx counts that are no multiple
        # of 8, an even ny, another spline order
        _case("ragged_fp64_cfl_10", "steps", 100, 82, 90, steps=10, labs_k=4),
        _case("ragged_mixed_10", "steps", 160, 111, 108, steps=10, precision="mixed", dt=0.005),
        # the Re_tau 590 production grid with two scalars
        _case("production_mixed_5", "steps", 384, 257, 384, steps=5, precision="mixed", scalars=2, cfl=0.8,
              control=-1.0, map="tanh", stretch=2.0, re_bulk=10850.0, re_tau=590.0),
        # sixteen independent channels of uneven sizes stepped together
        _case("ensemble_16_mixed", "ensemble", 0, 0, 0, members="wide", steps=10, precision="mixed", control=-0.9),
        # the control gradient of a short horizon, one checkpoint per step
        _case("adjoint_128", "adjoint", 128, 97, 128, steps=4, control=-0.5, dt=0.01),
        # a device-resident caller that strings the building blocks together
        _case("blocks_128_fp64", "blocks", 128, 97, 128, dt=0.005),
    ]


def _smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


FOUR_STEP = (12, 24, 36, 48, 72, 96, 144, 192, 288, 384, 576)
EVEN = [n for n in range(16, 257, 2) if _smooth(3 * n // 2)]
TUNED = [n for n in EVEN if 3 * n // 2 in FOUR_STEP]


def draw(rng):
    def pick(values, lo, hi):
        x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return min(values, key=lambda v: abs(math.log(v / x)))

    kind = rng.choice(("steps",) * 9 + ("blocks", "adjoint", "ensemble"))
    precision = rng.choice(("fp64", "mixed"))
    control = rng.choice((0.0, round(rng.uniform(-0.6, -0.2), 2)))
    if kind == "ensemble":
        return _case(None, kind, 0, 0, 0, members="small", steps=rng.randint(2, 12), precision=precision,
                     control=round(rng.uniform(-1.0, -0.2), 2))
    if kind == "adjoint":
        n = rng.choice((32, 48, 64, 96))
        return _case(None, kind, n, rng.randint(33, 97), rng.choice((32, 48, 64)), steps=rng.randint(1, 5),
                     control=round(rng.uniform(-0.6, -0.2), 2), dt=0.005)
    scalars = rng.choice((1, 1, 1, 2)) if kind == "steps" else 1
    lengths = TUNED if scalars == 2 or rng.random() < 0.5 else EVEN
    nx, nz = pick(lengths, 16, 256), pick(lengths, 16, 256)
    ny = round(math.exp(rng.uniform(math.log(25), math.log(193))))
    steps = 1 if kind == "blocks" else rng.choice((1, 2, 5, 10, 20))
    dt = rng.choice((0.0, 0.002)) if kind == "steps" else 0.002
    return _case(None, kind, nx, ny, nz, steps=steps, precision=precision, control=control, scalars=scalars, dt=dt,
                 labs_k=rng.choice((4, 5, 6, 6, 7)), cfl=rng.choice((0.8, 1.0)), re_bulk=500.0)


# ---- inputs ------------------------------------------------------------------------------

def _box(c):
    return c["lx_over_pi"] / 2.0, c["lz_over_pi"] / 2.0   # LMFx, LMFz


def _y_detect(c):
    return -1.0 + 15.0 / c["re_tau"]


def _config(c):
    lmfx, lmfz = _box(c)
    return Config(nx=c["nx"], ny=c["ny"], nz=c["nz"], labs_k=c["labs_k"], lmfx=lmfx, lmfz=lmfz, stretch=c["stretch"],
                  grid=_lib.KMM_GRID_TANH if c["map"] == "tanh" else _lib.KMM_GRID_SINE, nu=1.0 / c["re_bulk"],
                  cfl=c["cfl"], fixed_dt=int(c["dt"] > 0), n_scalar=c["scalars"],
                  precision=_lib.KMM_PREC_MIXED if c["precision"] == "mixed" else _lib.KMM_PREC_FP64,
                  control_amp=c["control"], control_yd=_y_detect(c))


def _points(c):
    """Knots of the clamped splines of order labs_k + 1 and their Greville points."""
    k, n = c["labs_k"] + 1, c["ny"]
    s = np.linspace(-1.0, 1.0, n - k + 2)
    a = c["stretch"]
    b = np.tanh(a * s) / math.tanh(a) if c["map"] == "tanh" else np.sin(a * math.pi / 2 * s) / math.sin(a * math.pi / 2)
    t = np.concatenate([np.full(k - 1, b[0]), b, np.full(k - 1, b[-1])])
    y = np.array([t[i + 1:i + k].mean() for i in range(n)])
    return t, y


def _nf(c):
    return 11 if c["scalars"] == 2 else 7


def _slots(c):
    return (0, 1, 2, 6, 10) if c["scalars"] == 2 else (0, 1, 2, 6)


def _fields(c, seed, out):
    """Laminar flow and scalar plus a divergence-free random-phase perturbation of the modes up to
    8, root mean square 0.1 of the bulk velocity, into out (nf, nz, nxh, ny)."""
    rng = np.random.default_rng(seed)
    lmfx, lmfz = _box(c)
    _, y = _points(c)
    q = 1.0 - y * y
    jx, jz = min(8, c["nx"] // 2 - 1), min(8, c["nz"] // 2 - 1)
    kx = np.arange(jx + 1)[None, :, None] / lmfx
    kz = np.concatenate([np.arange(jz + 1), np.arange(-jz, 0)])[:, None, None] / lmfz
    shape = (2 * jz + 1, jx + 1, 1)
    a, b = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape) for _ in range(2))
    a[0, 0] = b[0, 0] = 0.0
    k2 = kx * kx + kz * kz
    k2[0, 0] = 1.0
    v, f, g = q * q * a, -4.0 * y * q * a, q * b
    low = np.stack([1j * (kx * f - kz * g) / k2, v, 1j * (kz * f + kx * g) / k2])
    for j in range(1, jz + 1):   # the kx = 0 plane is Hermitian: the physical field is real
        low[:, -j, 0] = np.conj(low[:, j, 0])
    weight = np.where(np.arange(jx + 1) == 0, 1.0, 2.0)[None, None, :, None]
    low *= 0.1 / math.sqrt((weight * np.abs(low) ** 2).sum() / (3 * len(y)))
    rows = list(range(jz + 1)) + list(range(c["nz"] - jz, c["nz"]))
    out[:3, rows, :jx + 1] = torch.from_numpy(low)
    for s in (0,) + _slots(c)[3:]:
        out[s, 0, 0] = torch.from_numpy(1.5 * q + 0j)
    return out


def _host_fields(c, seed, pinned):
    shape = (_nf(c), c["nz"], c["nx"] // 2, c["ny"])
    return _fields(c, seed, torch.zeros(shape, dtype=torch.complex128, pin_memory=pinned))


def _gains(c, seed):
    rng = np.random.default_rng(seed + 1)
    return (1.0 + 0.05 * rng.standard_normal((c["nz"], c["nx"] // 2))).astype(np.float32)


def _members(c):
    grids = [g for g, n in ENSEMBLE[c["members"]] for _ in range(n)]
    return [dict(c, kind="steps", nx=g[0], ny=g[1], nz=g[2], control=c["control"] * (i + 1) / len(grids))
            for i, g in enumerate(grids)]


def prepare(case, seed):
    c, pinned = case, torch.cuda.is_available()
    if c["kind"] == "ensemble":
        members = _members(c)
        channels, fields = [Channel(_config(m)) for m in members], []
        for i, (m, ch) in enumerate(zip(members, channels)):
            fields.append(_host_fields(m, seed * 97 + i, pinned))
            ch.set_initial_data_uvw(fields[-1].numpy(), DT_START)
        return {"case": c, "channels": channels, "fields": fields}
    channel, U = Channel(_config(c)), _host_fields(c, seed, pinned)
    state = {"case": c, "channel": channel, "U": U}
    if c["kind"] == "steps":
        channel.dt = c["dt"] or DT_START
    elif c["kind"] == "adjoint":
        state["amp"] = torch.tensor(c["control"], dtype=torch.float64, requires_grad=True)
        state["gains"] = torch.from_numpy(_gains(c, seed)).requires_grad_()
    else:
        nxh, ny, nz, nz32 = c["nx"] // 2, c["ny"], c["nz"], c["nz"] * 3 // 2
        line = torch.float32 if c["precision"] == "mixed" else torch.float64
        dev = torch.zeros((10, nz, nxh, ny), dtype=torch.complex128, device="cuda")
        dev[:7] = U.cuda()
        channel.set_initial_data_uvw(U.numpy(), c["dt"])
        state.update(U=dev, stores=torch.from_numpy(channel.download_state()[1]).cuda(),
                     work=torch.zeros((10, nz, nxh, ny), dtype=torch.complex128, device="cuda"),
                     pencil=torch.zeros((10, ny, nz32, nxh, 2), dtype=line, device="cuda"))
    return state


# ---- one pass -----------------------------------------------------------------------------

def _scalars(out):
    return {"dt": out["dt"], "velmax": out["velmax"], "dpdx": out["phi_dpdx"][3], "tau_w": out["wall_shear_stress"],
            "q_w": out["wall_theta_stress"]}


def run(state):
    return {"steps": _run_steps, "ensemble": _run_ensemble, "adjoint": _run_adjoint,
            "blocks": _run_blocks}[state["case"]["kind"]](state)


def _run_steps(state):
    c, U = state["case"], state["U"]
    out = state["channel"].step_host_ptr(U.data_ptr(), _nf(c), None, c["steps"])
    return {"fields": [U[s] for s in _slots(c)], "scalars": _scalars(out)}


def _run_ensemble(state):
    outs = ensemble_step(state["channels"], state["case"]["steps"])
    lib = _lib.load()
    for ch, U in zip(state["channels"], state["fields"]):
        _lib.check(lib.kmm_download_state(ch._h, _lib.C.cast(U.data_ptr(), _lib._D), 7, None))
    dts = np.array([o["dt"] for o in outs])
    tau = np.array([o["wall_shear_stress"] for o in outs])
    return {"fields": list(state["fields"]), "dt": dts, "tau_w": tau}   # U as read back, whole


def _run_adjoint(state):
    c, amp, gains = state["case"], state["amp"], state["gains"]
    amp.grad = gains.grad = None
    J = control_objective(amp, gains, state["channel"], state["U"].numpy(), c["steps"], c["dt"], 1.0, 0.5)
    J.backward()
    return {"J": J.detach(), "dJ_damp": amp.grad, "dJ_dgains": gains.grad}


def _run_blocks(state):
    c, ch, U, W, X = state["case"], state["channel"], state["U"], state["work"], state["pencil"]
    for s in (1, 2, 3):
        for f in (0, 1, 2, 6):
            ch.y_to_x(U[f], X[f])
        ch.dft_x_realspace(X, s)
        for f in (0, 1, 2, 3, 4, 6, 7, 8):
            ch.x_to_y(X[f], W[f])
        W[9] = U[1]   # the starting v, which opposition control reads
        out = ch.wavespace(W, state["stores"], s, c["dt"])
        for f in (0, 1, 2, 6):
            U[f] = W[f]
    return {"fields": [U[f] for f in (0, 1, 2, 6)], "stores": state["stores"], "tau_w": out["wall_shear_stress"]}


# ---- what a pass cannot do without ----------------------------------------------------------

def _points_of(c):
    return c["nx"] // 2 * c["nz"] * c["ny"]


def work(case):
    """Bytes: the fields in and out, and per substep the state and the RK stores read and written
    once (they do not fit on the chip from one substep to the next).  Operations: the padded
    transforms at 5/2 N log2 N a real line, and the banded solves and products."""
    c = case
    if c["kind"] == "ensemble":
        parts = [work(m) for m in _members(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    ns, x32, z32, nsc = _points_of(c), c["nx"] * 3 // 2, c["nz"] * 3 // 2, c["scalars"]
    nfld, nprod, nst = 3 + nsc, 5 + 3 * nsc, 2 + nsc
    sub = 3 * c["steps"] * (4 if c["kind"] == "adjoint" else 1)   # forward, recomputed forward, transpose (twice the lines)
    lines = (nfld + nprod) * c["ny"] * (c["nx"] // 2 * 5.0 * z32 * math.log2(z32) + z32 * 2.5 * x32 * math.log2(x32))
    bw = (c["labs_k"] + 2) // 2
    solves = ns * ((4 + nst + nsc) * 4.0 * (4 * bw + 1) + (8 + 2 * nst) * 4.0 * (2 * bw + 1))
    return {"bytes": 16.0 * ns * (2 * nfld + sub * 2 * (nfld + nst)), "flops": sub * (lines + solves)}


def tolerance(case):
    """Against the dense FP64 step, FP32 transforms and products leave up to 6e-7 in the fields after
    ten steps and three times that over the passes of a state that marches on, and the FP64 path up to
    4e-13 on these grids (the second derivatives of the splines amplify the rounding of its sums, more
    so on finer grids); the gains and their gradient are FP32 numbers (2.5e-8)."""
    if case["kind"] == "adjoint":
        return {"rel": 1e-7, "max": 1e-5}
    if case["precision"] == "mixed":
        return {"rel": 6e-6, "max": 1e-3}
    return {"rel": 1e-11, "max": 1e-8}


# ---- the same step in dense FP64 torch --------------------------------------------------------

def _basis(t, k, x, d):
    """d-th derivatives of all order-k splines on the knots t at the points x: (len(x), n)."""
    if k == 1:
        last = np.max(np.nonzero(t[:-1] < t[1:])[0])
        B = (t[None, :-1] <= x[:, None]) & (x[:, None] < t[None, 1:])
        B[x >= t[-1], last] = True
        return B.astype(np.float64) if d == 0 else np.zeros(B.shape)
    n = len(t) - k
    left, right = t[k - 1:k - 1 + n] - t[:n], t[k:k + n] - t[1:1 + n]
    il, ir = (np.divide(1.0, w, out=np.zeros(n), where=w > 0) for w in (left, right))
    if d == 0:
        B = _basis(t, k - 1, x, 0)
        return (x[:, None] - t[:n]) * il * B[:, :n] + (t[k:k + n] - x[:, None]) * ir * B[:, 1:n + 1]
    B = _basis(t, k - 1, x, d - 1)
    return (k - 1) * (il * B[:, :n] - ir * B[:, 1:n + 1])


class _Dense:
    """The RK3 step of one channel with dense operators; fields are (nz, nxh, ny) tensors."""

    def __init__(self, c, device):
        self.c, self.device = c, device
        k = c["labs_k"] + 1
        t, y = _points(c)
        as_t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=device)
        D = [_basis(t, k, y, d) for d in range(3)]
        inv = np.linalg.inv(D[0])
        self.D0, self.D1, self.D2 = (as_t(m) for m in D)
        self.M1, self.M2 = as_t(D[1] @ inv), as_t(D[2] @ inv)
        self.integ = as_t((t[k:] - t[:-k]) / k)
        yd = _y_detect(c)
        self.probe = as_t(_basis(t, k, np.array([yd, -yd]), 0) @ inv)
        gap = np.diff(y)
        self.dyr = as_t(1.0 / np.minimum(np.concatenate([gap[:1], gap]), np.concatenate([gap, gap[-1:]])))
        lmfx, lmfz = _box(c)
        nz, nxh, nh = c["nz"], c["nx"] // 2, c["nz"] // 2
        self.kx = as_t(np.arange(nxh) / lmfx)[None, :, None]
        self.kz = as_t(np.concatenate([np.arange(nh + 1), np.arange(nh + 1 - nz, 0)]) / lmfz)[:, None, None]
        self.k2 = self.kx ** 2 + self.kz ** 2
        self.k2[0, 0] = 1.0   # the mean mode is solved apart
        self.nu, self.dxr, self.dzr = 1.0 / c["re_bulk"], c["nx"] / (2 * math.pi * lmfx), nz / (2 * math.pi * lmfz)
        self.visc = [self.nu / 0.71, self.nu / 0.2][:c["scalars"]]
        self.kept = {}

    def op(self, M, f):
        return torch.view_as_complex(torch.einsum("ij,zxjc->zxic", M, torch.view_as_real(f)).contiguous())

    def apply(self, A, f):
        """A (modes, ny, ny) on f (nz, nxh, ny)."""
        r = torch.view_as_real(f)
        return torch.view_as_complex(torch.bmm(A, r.reshape(-1, f.shape[-1], 2)).reshape(r.shape))

    def _inverse(self, a, b, wall):
        """Inverses of a D0 - b D2 per mode, its wall rows replaced by wall (per mode) on the diagonal."""
        n, out = self.c["ny"], []
        for i in range(0, a.numel(), 4096):
            s = slice(i, min(i + 4096, a.numel()))
            A = a.reshape(-1, 1, 1)[s] * self.D0 - b.reshape(-1, 1, 1)[s] * self.D2
            A[:, 0] = A[:, -1] = 0.0
            A[:, 0, 0], A[:, -1, -1] = wall.reshape(-1)[s], wall.reshape(-1)[s]
            out.append(torch.linalg.inv(A))
        return torch.cat(out)

    def inverse(self, beta):
        """(alpha D0 - beta D2)^-1 per mode; kept while dt is fixed."""
        if beta in self.kept:
            return self.kept[beta]
        a = 1.0 + beta * self.k2
        wall = a * self.D0[0, 0] - beta * self.D2[0, 0]
        inv = self._inverse(a, torch.full_like(a, beta), wall)
        if self.c["dt"] > 0:
            self.kept[beta] = inv
        return inv

    def v_inverse(self):
        if "v" not in self.kept:
            a = -self.k2
            self.kept["v"] = self._inverse(a, torch.full_like(a, -1.0), torch.full_like(a, float(self.D0[0, 0])))
        return self.kept["v"]

    def physical(self, f):
        nz, nh, nxh, n32 = self.c["nz"], self.c["nz"] // 2, self.c["nx"] // 2, self.c["nx"] * 3 // 2
        z = torch.zeros((nz * 3 // 2 - (nz - 1),) + f.shape[1:], dtype=f.dtype, device=f.device)
        f = torch.fft.ifft(torch.cat([f[:nh], z, f[nh + 1:]]), dim=0, norm="forward")
        f = torch.cat([f[:, :1].real + 0j, f[:, 1:], torch.zeros((f.shape[0], n32 // 2 + 1 - nxh, f.shape[2]),
                                                                 dtype=f.dtype, device=f.device)], dim=1)
        return torch.fft.irfft(f, n=n32, dim=1, norm="forward")

    def spectral(self, f):
        nz, nh, nxh = self.c["nz"], self.c["nz"] // 2, self.c["nx"] // 2
        g = torch.fft.fft(torch.fft.rfft(f, dim=1, norm="forward")[:, :nxh], dim=0, norm="forward")
        return torch.cat([g[:nh], torch.zeros_like(g[:1]), g[g.shape[0] - (nz - nh - 1):]])

    def start(self, U):
        u, v, w = U[:3]
        return [1j * self.kz * u - 1j * self.kx * w, self.op(self.M2, v) - self.k2 * v] + list(U[3:]), \
            [u[0, 0], w[0, 0]] + [t[0, 0] for t in U[3:]]

    def step(self, U, stores, means, dt, amp=None, gains=None):
        """One RK3 step; returns the fields, the stores, the mean stores, dt and the diagnostics."""
        info = {"phi": 0.0}
        for s in (1, 2, 3):
            U, stores, means, dt = self.substep(U, stores, means, dt, s, amp, gains, info)
        return U, stores, means, dt, {"dt": dt, "velmax": info["velmax"], "dpdx": info["phi"] / dt,
                                      "tau_w": info["tau"], "q_w": info["q"]}

    def substep(self, U, stores, means, dt, s, amp, gains, info):
        c, kx, kz, k2 = self.c, self.kx, self.kz, self.k2
        p = [self.physical(f) for f in U]
        u, v, w = p[:3]
        if s == 1:
            info["velmax"] = float((u.abs() * self.dxr + v.abs() * self.dyr + w.abs() * self.dzr).detach().max())
            dt = c["dt"] or c["cfl"] / math.pi / info["velmax"]
        f1, f2, f3, f4, f5 = (self.spectral(f) for f in (u * u - v * v, u * v, w * w - v * v, v * w, u * w))
        flux = [[self.spectral(q * t) for q in (u, v, w)] for t in p[3:]]
        co = lambda name, i=s: dt * RK[name][i - 1]
        hg = kx * kz * (f1 - f3) + (kz ** 2 - kx ** 2) * f5 + self.op(self.M1, 1j * kx * f4 - 1j * kz * f2)
        hv = self.op(self.M1, -kx ** 2 * f1 - 2 * kx * kz * f5 - kz ** 2 * f3) \
            + 1j * k2 * (kx * f2 + kz * f4) + self.op(self.M2, 1j * kz * f4 + 1j * kx * f2)
        ht = [-(1j * kx * a + 1j * kz * b + self.op(self.M1, m)) for a, m, b in flux]

        def rhs(store, h, visc):
            r = store + co("gamma") * h
            if s == 1:
                r = r + co("alpha") * visc * (self.op(self.M2, store) - k2 * store)
            return torch.cat([torch.zeros_like(r[..., :1]), r[..., 1:-1], torch.zeros_like(r[..., :1])], dim=-1)

        def new_store(f, d2f, h, visc):
            return f if s == 3 else co("zeta", s + 1) * h + f + co("alpha", s + 1) * visc * (d2f - k2 * f)

        def helmholtz(store, h, visc):
            x = self.apply(self.inverse(co("beta") * visc), rhs(store, h, visc))
            f, d2f = self.op(self.D0, x), self.op(self.D2, x)
            return f, new_store(f, d2f, h, visc)

        g, sg = helmholtz(stores[0], hg, self.nu)
        phi, sphi = helmholtz(stores[1], hv, self.nu)
        scal = [helmholtz(st, h, visc) for st, h, visc in zip(stores[2:], ht, self.visc)]
        # the wall velocities of the opposition control, with the projection the padded transforms apply
        wall = [torch.zeros_like(phi[..., :1])] * 2
        if c["control"] != 0.0:
            wall = []
            for row in self.probe:
                d = torch.einsum("i,zxi->zx", row + 0j, U[1])
                nyq = torch.ones(c["nz"], 1, device=self.device, dtype=d.dtype)
                nyq[c["nz"] // 2] = 0.0
                flip = torch.cat([d[:1, :1], d[1:, :1].flip(0)])
                d = nyq * torch.cat([0.5 * (d[:, :1] + flip.conj()), d[:, 1:]], dim=1)
                wall.append(((c["control"] if amp is None else amp) * (d if gains is None else gains * d))[..., None])
        # particular and unit-wall solutions of phi and v, combined so that dv/dy vanishes at the walls
        n = c["ny"]
        beta = co("beta") * self.nu
        p0 = (1.0 + beta * k2) * self.D0[0, 0] - beta * self.D2[0, 0]
        ch = (p0 * self.inverse(beta)[:, :, 0].reshape(c["nz"], -1, n))   # real
        real = lambda M, x: torch.einsum("ij,zxj->zxi", M, x)
        ph, d2ph = real(self.D0, ch), real(self.D2, ch)
        vinv = self.v_inverse()
        cv = self.apply(vinv, torch.cat([wall[0], phi[..., 1:-1], wall[1]], dim=-1))
        ph0 = ph.clone()
        ph0[..., 0] = ph0[..., -1] = 0.0
        chv = torch.bmm(vinv, ph0.reshape(-1, n, 1)).reshape(ph.shape)
        vp, dvp, vh, dvh = self.op(self.D0, cv), self.op(self.D1, cv), real(self.D0, chv), real(self.D1, chv)
        a, b = dvh[..., :1], dvh[..., -1:]
        den = a * a - b * b
        C1, C2 = (b * dvp[..., -1:] - a * dvp[..., :1]) / den, (a * dvp[..., -1:] - b * dvp[..., :1]) / den
        v = vp + C1 * vh + C2 * vh.flip(-1)
        dv = dvp + C1 * dvh - C2 * dvh.flip(-1)
        hs = ph if s == 3 else ph + co("alpha", s + 1) * self.nu * (d2ph - k2 * ph)
        sphi = sphi + C1 * hs + C2 * hs.flip(-1)
        u, w = (1j * kx * dv - 1j * kz * g) / k2, (1j * kx * g + 1j * kz * dv) / k2

        # the mean mode: U and the scalars forced to their bulk values, W not
        def mean(store, f, visc, forced):
            d = self.M1 @ f.real
            r = store.real - co("gamma") * d
            if s == 1:
                r = r + co("alpha") * visc * (self.M2 @ store.real)
            A = self.D0 - co("beta") * visc * self.D2
            A[0], A[-1] = 0.0, 0.0
            A[0, 0] = A[-1, -1] = self.D0[0, 0] - co("beta") * visc * self.D2[0, 0]
            inner = torch.ones_like(r)
            inner[0] = inner[-1] = 0.0
            x = torch.linalg.solve(A, torch.stack([r * inner, inner], dim=1))
            phi = (1.0 - 0.5 * self.integ @ x[:, 0]) / (0.5 * self.integ @ x[:, 1]) if forced else 0.0 * r[0]
            x = x[:, 0] + phi * x[:, 1]
            prof = self.D0 @ x
            st = prof if s == 3 else prof + co("alpha", s + 1) * visc * (self.D2 @ x) - co("zeta", s + 1) * d
            return prof, st, phi, 0.5 * visc * ((self.D1 @ x)[0] - (self.D1 @ x)[-1])

        m = [mean(means[0], f2[0, 0], self.nu, True), mean(means[1], f4[0, 0], self.nu, False)]
        m += [mean(st, f[1][0, 0], visc, True) for st, f, visc in zip(means[2:], flux, self.visc)]
        info["phi"] = info["phi"] + m[0][2]
        info["tau"], info["q"] = m[0][3], m[2][3]
        first = torch.zeros((c["nz"], c["nx"] // 2, 1), dtype=torch.bool, device=self.device)
        first[0, 0] = True
        put = lambda f, line: torch.where(first, line + 0j, f)
        U = [put(u, m[0][0]), put(v, 0.0 * m[0][0]), put(w, m[1][0])] + [put(f[0], x[0]) for f, x in zip(scal, m[2:])]
        return U, [sg, sphi] + [f[1] for f in scal], [x[1] for x in m], dt


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _as_scalars(info):
    return {k: float(v) for k, v in info.items()}


def _march(c, seed):
    D, U = _Dense(c, _device()), _host_fields(c, seed, False)
    U = [U[s].to(_device()) for s in _slots(c)]
    stores, means = D.start(U)
    dt = c["dt"]
    for _ in range(c["steps"]):
        U, stores, means, dt, info = D.step(U, stores, means, dt)
    stores = [s.clone() for s in stores]
    for s, line in zip([stores[0], stores[1]] + stores[2:], means):
        s[0, 0] = line + 0j
    return U, stores, _as_scalars(info)


def exact(case, seed):
    c = case
    if c["kind"] == "ensemble":
        got = [_march(m, seed * 97 + i) for i, m in enumerate(_members(c))]
        empty = lambda U: [torch.zeros_like(U[0])] * 3   # fields 4 to 6 hold nothing between steps
        return {"fields": [torch.stack(U[:3] + empty(U) + U[3:]).cpu() for U, _, _ in got],
                "dt": np.array([i["dt"] for _, _, i in got]), "tau_w": np.array([i["tau_w"] for _, _, i in got])}
    # dense operators of this many modes take minutes: the time goes with modes x ny^3
    if _points_of(c) * c["ny"] ** 2 * (c["steps"] if c["dt"] == 0 else 2) > 1e12:
        return None
    if c["kind"] == "adjoint":
        D, U = _Dense(c, _device()), _host_fields(c, seed, False)
        U = [U[s].to(_device()) for s in _slots(c)]
        amp = torch.tensor(c["control"], dtype=torch.float64, device=_device(), requires_grad=True)
        gains = torch.from_numpy(_gains(c, seed)).to(_device(), torch.float64).requires_grad_()
        stores, means = D.start(U)
        J = 0.0
        for _ in range(c["steps"]):
            U, stores, means, _, info = D.step(U, stores, means, c["dt"], amp, gains)
            J = J + (info["tau_w"] + 0.5 * info["q_w"]) / c["steps"]
        J.backward()
        return {"J": J.detach().cpu(), "dJ_damp": amp.grad.cpu(), "dJ_dgains": gains.grad.cpu()}
    U, stores, info = _march(c, seed)
    if c["kind"] == "blocks":
        return {"fields": [f.cpu() for f in U], "stores": torch.stack(stores).cpu(), "tau_w": info["tau_w"]}
    return {"fields": [f.cpu() for f in U], "scalars": info}
