"""Performance cases of the channel-flow time step: what a program that uses
the framework has it do, through the public Python entry points (`cdns`).

A case is a dict of plain values.  `kind` says which entry points a pass goes
through:

  steps      a running simulation advanced by `steps` steady time steps
             (Context.run), its velocity read into a device buffer;
  sampled    the same with a statistics sample after every step and the running
             means read at the end (a production run past its spin-up);
  restart    velocity handed over from pinned host memory, the first `steps`
             iterations (both solver setups among them), velocity, pressure and
             pressure gradient read back: a short job, or a disturbance study;
  gradient   the wall-shear objective of `steps` steps and its gradient with
             respect to the initial velocity and the wall blowing/suction
             (Context.adjoint_run), forward and backward;
  ensemble   `members` independent channels of mixed sizes advanced together
             (Batch.run);
  synthesis  one field brought to the product grid on caller-owned buffers and
             the caller's stream (fine_backward_noalloc), the smallest call.

`exact` is the same computation in 64 bits in plain torch, written from the
equations: Fourier in x and z, Chebyshev-tau in y, the influence-matrix and tau
corrections of the pressure, second-order extrapolated multistep.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "channel-dns_b200"))

import cdns  # noqa: E402

PI = math.pi
# product lengths of x and z: 2^a 3^b 5^c 7^d, what an FFT user picks
SMOOTH = sorted({2 ** a * 3 ** b * 5 ** c * 7 ** d for a in range(9) for b in range(5) for c in range(3)
                 for d in range(3) if 24 <= 2 ** a * 3 ** b * 5 ** c * 7 ** d <= 400})
# product lengths the mixed-precision step takes (include/cdns.h, cdns_precision)
MIXED = (32, 48, 64, 72, 96, 128, 144, 192, 196)
MEMBER_SIZES = (32, 48, 64, 96)   # ensemble members (cdns.ensemble)


def _channel(name, kind, nx, ny, nz, steps, nx2=None, ny2=None, nz2=None, precision="fp64", flow="gradient", **more):
    """A channel of nx x (ny + 1) x nz points with NXS = nx/2, NZS = nz/2 and
    NYS = ny - 2 retained modes and a 3/2 product grid unless given."""
    c = {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "nx2": nx2 or 3 * nx // 2,
         "ny2": ny2 or 3 * ny // 2, "nz2": nz2 or 3 * nz // 2, "steps": steps, "precision": precision, "flow": flow}
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: one field to physical space inside another program
        _channel("synthesis_48", "synthesis", 48, 48, 48, 1),
        # the repository's example channel (32 x 33 x 32, constant flow rate): launches and latency
        _channel("steps_32_flowrate", "steps", 32, 32, 32, 20, flow="rate"),
        # a parameter study's channel (64 x 65 x 64, 96^3 product grid)
        _channel("steps_64", "steps", 64, 64, 64, 10),
        # a grid chosen by its resolution and not by its factors: 90, 75 and 100 points
        _channel("steps_60_ragged", "steps", 60, 50, 66, 10, nx2=90, ny2=76, nz2=100),
        # the headline channel, Re_tau 180 (128 x 129 x 128, 196 x 193 x 196 product grid)
        _channel("steps_retau180", "steps", 128, 128, 128, 10, nx2=196, ny2=192, nz2=196),
        # the same in the mixed FP32/FP64 form
        _channel("steps_retau180_mixed", "steps", 128, 128, 128, 10, nx2=196, ny2=192, nz2=196, precision="mixed"),
        # a well-resolved higher Reynolds number: 256 x 193 x 192, 384 x 289 x 288 product grid
        _channel("steps_256x193x192", "steps", 256, 192, 192, 3, re=395.0),
        # the headline channel past its spin-up: statistics of every step
        _channel("sampled_retau180", "sampled", 128, 128, 128, 5, nx2=196, ny2=192, nz2=196),
        # a short job from a host field, both setups included
        _channel("restart_96", "restart", 96, 96, 96, 10),
        # drag gradient, 64 x 65 x 64, checkpoints every 5 steps
        _channel("gradient_64", "gradient", 64, 64, 64, 20, interval=5),
        # an ensemble of uneven channels, both precisions
        {"name": "ensemble_24", "kind": "ensemble", "members": 24, "steps": 5, "precision": "fp64", "draw": 3},
        {"name": "ensemble_24_mixed", "kind": "ensemble", "members": 24, "steps": 5, "precision": "mixed", "draw": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _product(rng, n, lengths=SMOOTH):
    """A product length of at least 3/2 n: the next one, or one a little longer."""
    ok = [m for m in lengths if 2 * m >= 3 * n]
    return rng.choice(ok[:2])


def draw(rng):
    kind = rng.choice(["steps"] * 5 + ["sampled", "restart", "gradient", "ensemble", "synthesis"])
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(4, 16), "steps": rng.randint(2, 4),
                "precision": rng.choice(["fp64", "mixed"]), "draw": rng.randint(0, 10 ** 6)}
    precision = rng.choice(["fp64", "fp64", "mixed"]) if kind in ("steps", "sampled", "restart") else "fp64"
    top = {"synthesis": 60, "gradient": 72, "restart": 128}.get(kind, 192)
    lengths = SMOOTH
    if precision == "mixed":
        lengths, top = MIXED, 128
    elif kind == "synthesis":
        lengths = [m for m in SMOOTH if m <= 90]
    nx, nz = (2 * _log_int(rng, 12, top // 2) for _ in range(2))
    if kind == "sampled":   # the statistics' coarse grid is transformed too
        nx, nz = (min(m for m in SMOOTH if m >= n and m % 2 == 0) for n in (nx, nz))
    ny = 2 * _log_int(rng, 12, min(top, 160) // 2)
    nx2, nz2 = _product(rng, nx, lengths), _product(rng, nz, lengths)
    ny2 = 3 * ny // 2 + rng.choice([0, 0, 1, 4])
    ny2 += ny2 % 2
    flow = "gradient" if kind == "gradient" else rng.choice(["gradient", "gradient", "rate"])
    steps = min(rng.randint(3, 8), max(1, 80_000_000 // (nx2 * ny2 * nz2)))
    if kind in ("synthesis", "sampled", "restart"):
        steps = {"synthesis": 1, "sampled": max(1, steps // 2), "restart": max(2, steps)}[kind]
    more = {}
    if kind == "gradient":
        steps, more = rng.randint(8, 20), {"interval": rng.randint(2, 6)}
    c = _channel("", kind, nx, ny, nz, steps, nx2=nx2, ny2=ny2, nz2=nz2, precision=precision, flow=flow, **more)
    del c["name"]
    return c


def _mesh(c):
    lx, lz = (10.0, 10.0) if c["flow"] == "rate" else (4.0 * PI, 2.0 * PI)
    return cdns.Mesh(c["nx"], c["ny"], c["nz"], c["nx"] // 2, c["ny"] - 2, c["nz"] // 2, c["nx2"], c["ny2"],
                     c["nz2"], lx, lz)


def _params(c):
    if c["flow"] == "rate":   # the example configuration
        return cdns.Params(Re=2800.0, DT=3e-3, INDEX_GRAD_PRE=0, V_Microblow0=1e-3)
    return cdns.Params(Re=c.get("re", 180.0), DT=5e-5)


def _members(c):
    """The ensemble's channels: sizes and Re_tau from the case's own draw."""
    rng = np.random.default_rng(c["draw"])
    sizes = rng.choice(MEMBER_SIZES, size=c["members"])
    res = rng.uniform(100.0, 180.0, size=c["members"])
    return [_channel("", "steps", int(n), int(n), int(n), c["steps"], precision=c["precision"], re=float(r))
            for n, r in zip(sizes, res)]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _chebyshev_coeffs(values, ncy):
    """First ncy Chebyshev coefficients of samples on Gauss-Lobatto points (last axis)."""
    n = values.shape[-1] - 1
    j = torch.arange(n + 1, dtype=torch.float64, device=values.device)
    C = torch.cos(PI * torch.outer(j, j[:ncy]) / n)
    w = torch.full((n + 1,), 2.0, dtype=torch.float64, device=values.device)
    w[0] = w[-1] = 1.0
    a = (values * w).to(values.dtype) @ C.to(values.dtype) / n
    a[..., 0] = a[..., 0] * 0.5
    return a


def _field(mesh, params, seed):
    """Seeded velocity [nkz][ncy][nkx][3]: mean profile plus a solenoidal no-slip
    perturbation with a k^-5/3 energy envelope at 10 % of the centreline velocity."""
    dev = _device()
    nkz, ncy, nkx = mesh.spectral_shape
    g = torch.Generator().manual_seed(int(seed))
    nq = min(8, max(ncy - 5, 1))
    q = torch.randn((2, 2, nkz, nkx, nq), generator=g, dtype=torch.float64).to(dev)
    kz = torch.arange(-mesh.NZS, mesh.NZS + 1, dtype=torch.float64, device=dev)
    kx = torch.arange(nkx, dtype=torch.float64, device=dev)
    k2 = kx[None, :] ** 2 + kz[:, None] ** 2
    scale = torch.where(k2 > 0, k2.clamp(min=1.0) ** (-5.0 / 12.0), torch.zeros_like(k2))
    npts = 2 * ncy
    y = torch.cos(PI * torch.arange(npts, dtype=torch.float64, device=dev) / (npts - 1))
    T = torch.cos(torch.outer(torch.arange(nq, dtype=torch.float64, device=dev), torch.arccos(y.clamp(-1, 1))))
    shape = _chebyshev_coeffs((1.0 - y * y) ** 2 * T, ncy)             # [nq][ncy]
    A, B = (torch.complex(q[i, 0], q[i, 1]) * scale[..., None] @ shape.to(torch.complex128) for i in range(2))
    ax, az = kx * (2.0 * PI / mesh.XL), kz * (2.0 * PI / mesh.ZL)
    iax, iaz = 1j * ax[None, :, None], 1j * az[:, None, None]
    dB = B @ _derivative_matrix(ncy, dev).T.to(torch.complex128)
    v = torch.stack((-iaz * A + iax * dB, (ax[None, :, None] ** 2 + az[:, None, None] ** 2) * B,
                     iax * A + iaz * dB))                              # [3][nkz][nkx][ncy]
    v[:, :, 0] = 0.5 * (v[:, :, 0] + v[:, :, 0].flip(1).conj())        # a real field
    wx = torch.full((nkx,), 2.0, dtype=torch.float64, device=dev)
    wx[0] = 1.0
    k, j = torch.arange(ncy, dtype=torch.float64, device=dev), torch.arange(npts, dtype=torch.float64, device=dev)
    C = torch.cos(PI * torch.outer(k, j) / (npts - 1)).to(torch.complex128)
    rms = torch.sqrt((wx[None, None, :, None] * (v @ C).abs() ** 2).sum() / (3 * npts))
    if params.INDEX_GRAD_PRE == 1:   # Reichardt's law of the wall
        yp = (1.0 - y.abs()) * params.Re
        mean = torch.log1p(0.41 * yp) / 0.41 + 7.8 * (1.0 - torch.exp(-yp / 11.0) - yp / 11.0 * torch.exp(-yp / 3.0))
    else:
        mean = 1.5 * (1.0 - y * y)
    v = v * (0.1 * mean.max() / rms)
    a = _chebyshev_coeffs(mean, ncy)
    sign = (-1.0) ** torch.arange(ncy, device=dev)
    top, bottom = a.sum(), (a * sign).sum()
    a[0] -= 0.5 * (top + bottom)
    a[1] -= 0.5 * (top - bottom)
    v[:, mesh.NZS, 0] = 0.0
    v[0, mesh.NZS, 0] = a.to(torch.complex128)
    return v.permute(1, 3, 2, 0).contiguous()


def _control(mesh, seed):
    """Seeded blowing/suction of the |k| <= 8 modes, wall data [nkz][2][nkx][3]."""
    rng = np.random.default_rng(seed)
    nkz, _, nkx = mesh.spectral_shape
    bc = np.zeros((nkz, 2, nkx, 3), dtype=np.complex128)
    z, mz, mx = mesh.NZS, min(8, mesh.NZS), min(8, mesh.NXS)
    v = 0.01 * (rng.standard_normal((2 * mz + 1, 2, mx + 1)) + 1j * rng.standard_normal((2 * mz + 1, 2, mx + 1)))
    v[:, :, 0] = 0.5 * (v[:, :, 0] + v[::-1, :, 0].conj())
    v[mz, :, 0] = 0.0
    bc[z - mz:z + mz + 1, :, :mx + 1, 1] = v
    return bc


def _spectrum(mesh, seed):
    """A spectral field of a real signal with a decaying spectrum, [nkz][ncy][nkx]."""
    return _field(mesh, cdns.Params(Re=180.0, DT=5e-5), seed)[..., 0].contiguous()


def _context(c, u):
    """A simulation past its two first-order setup steps."""
    ctx = cdns.Context(_mesh(c), _params(c),
                       precision=cdns.PRECISION_MIXED if c["precision"] == "mixed" else cdns.PRECISION_FP64)
    torch.cuda.synchronize()
    ctx.set_velocity_device(u.data_ptr())
    ctx.run(1, 2)
    ctx.synchronize()
    return ctx


def prepare(case, seed):
    c, kind = dict(case), case["kind"]
    s = {"case": c}
    if kind == "ensemble":
        members = _members(c)
        fields = [_field(_mesh(m), _params(m), seed + 1000 * i) for i, m in enumerate(members)]
        torch.cuda.synchronize()
        s["batch"] = cdns.Batch([_mesh(m) for m in members], [_params(m) for m in members],
                                precision=cdns.PRECISION_MIXED if c["precision"] == "mixed" else cdns.PRECISION_FP64)
        for ctx, u in zip(s["batch"].members, fields):
            ctx.set_velocity_device(u.data_ptr())
        s["batch"].run(1, 2)
        s["batch"].synchronize()
        s["it"], s["out"] = 3, fields
        return s
    mesh = s["mesh"] = _mesh(c)
    if kind == "synthesis":   # the embedding program steps a channel of that mesh, too
        s["ctx"] = cdns.Context(mesh, _params(c))
        s["in"] = _spectrum(mesh, seed)
        s["out"] = torch.empty(mesh.fine_shape, dtype=torch.float64, device="cuda")
        return s
    u = _field(mesh, _params(c), seed)
    if kind in ("steps", "sampled"):
        s["ctx"], s["it"], s["out"] = _context(c, u), 3, u
        return s
    s["ctx"] = cdns.Context(mesh, _params(c),
                            precision=cdns.PRECISION_MIXED if c["precision"] == "mixed" else cdns.PRECISION_FP64)
    if kind == "gradient":
        s["u"], s["control"] = u, _control(mesh, seed)
        torch.cuda.synchronize()
        return s
    s["u"] = u.cpu().pin_memory()
    s["v"] = torch.empty_like(s["u"]).pin_memory()
    s["p"] = torch.empty(mesh.spectral_shape, dtype=torch.complex128).pin_memory()
    return s


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    n = c["steps"]
    if kind == "synthesis":
        cdns.fine_backward_noalloc(state["mesh"], state["in"].data_ptr(), state["out"].data_ptr(),
                                   torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "ensemble":
        state["batch"].run(state["it"], n)
        state["it"] += n
        for ctx, out in zip(state["batch"].members, state["out"]):
            ctx.get_velocity_device(out.data_ptr())
        return state["out"]
    ctx = state["ctx"]
    if kind == "steps":
        ctx.run(state["it"], n)
        state["it"] += n
        ctx.get_velocity_device(state["out"].data_ptr())
        return state["out"]
    if kind == "sampled":
        ctx.statistics_reset()
        for _ in range(n):
            ctx.step(state["it"])
            ctx.statistics_sample()
            state["it"] += 1
        ctx.get_velocity_device(state["out"].data_ptr())
        _, dp, means = ctx.statistics_read()
        return state["out"], np.array(dp), means
    if kind == "gradient":
        ctx.set_velocity_device(state["u"].data_ptr())
        J, gu, gb = ctx.adjoint_run(n, c["interval"], control=state["control"])
        return np.array(J), gu, gb
    ctx.set_velocity(state["u"].numpy())
    ctx.run(1, n)
    ctx.synchronize()
    return ctx.get_velocity(state["v"].numpy()), ctx.get_pressure(state["p"].numpy()), np.array(ctx.dpdx())


def work(case):
    """Bytes: the multistep state read and written once a step (u, u_prev, N_prev
    in; u, N out; the pressure); flops: the nine 3-D transforms, u x omega and
    the four column solves of a step."""
    if case["kind"] == "ensemble":
        ws = [work(m) for m in _members(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    m = _mesh(case)
    nkz, ncy, nkx = m.spectral_shape
    ns, ny2 = nkz * ncy * nkx, m.NY2 + 1

    def transform():
        return (5.0 * m.NY2 * math.log2(m.NY2) * nkz * nkx + 5.0 * m.NZ2 * math.log2(m.NZ2) * ny2 * nkx
                + 2.5 * m.NX2 * math.log2(m.NX2) * ny2 * m.NZ2)

    if case["kind"] == "synthesis":
        return {"bytes": 16.0 * ns + 8.0 * ny2 * m.NZ2 * m.NX2, "flops": transform()}
    step_bytes = 16.0 * ns * 16
    step_flops = 9 * transform() + 9.0 * ny2 * m.NZ2 * m.NX2 + 4 * 24.0 * ns
    if case["kind"] == "sampled":
        step_flops += 4 * 0.3 * transform() + 40.0 * m.NX * m.NY * m.NZ
    if case["kind"] == "gradient":   # forward and transposed step
        return {"bytes": 2.0 * case["steps"] * step_bytes, "flops": 2.7 * case["steps"] * step_flops}
    return {"bytes": case["steps"] * step_bytes + 16.0 * 6 * ns, "flops": case["steps"] * step_flops}


def tolerance(case):
    # About four times what passes differ by from `exact`, after up to three passes.
    # FP64: 1e-13 for velocities and gradients, 3e-13 to 1e-12 for the pressure
    # (its sigma correction divides by a difference that cancels to 1e-6).  Mixed:
    # 1e-8 to 4e-8 of the field; a single coefficient, far below the mean profile,
    # may be off by more of the field's root mean square.
    if case.get("precision") == "mixed":
        return {"rel": 2e-7, "max": 3e-4}
    return {"rel": 4e-12, "max": 4e-10}


# ---- the same computation in plain torch, 64 bits -------------------------
def _derivative_matrix(n, dev):
    """(D f)_k = sum_{j > k, j + k odd} 2 j f_j, halved at k = 0."""
    k = torch.arange(n, device=dev)
    D = torch.where((k[None, :] > k[:, None]) & ((k[None, :] + k[:, None]) % 2 == 1), 2.0 * k[None, :].double(), 0.0)
    D[0] *= 0.5
    return D


class _Exact:
    """One channel; columns [nkz][nkx] with y first: arrays [ncy][nkz][nkx]."""

    def __init__(self, mesh, params):
        self.m, self.p, self.dev = mesh, params, _device()
        m, dev = mesh, self.dev
        self.nkz, self.ncy, self.nkx = m.spectral_shape
        self.ax = torch.arange(self.nkx, dtype=torch.float64, device=dev)[None, :] * (2 * PI / m.XL)
        self.az = torch.arange(-m.NZS, m.NZS + 1, dtype=torch.float64, device=dev)[:, None] * (2 * PI / m.ZL)
        self.D = _derivative_matrix(self.ncy, dev).to(torch.complex128)
        n = m.NYS
        self.WL, self.WD, self.WR = [0.0] * (n + 3), [0.0] * (n + 3), [0.0] * (n + 3)
        for y in range(2, n + 1):
            self.WL[y] = (2.0 if y == 2 else 1.0) / (4.0 * y * (y - 1))
            self.WD[y] = 0.0 if y >= n - 1 else -1.0 / (2.0 * (y * y - 1))
            self.WR[y] = 0.0 if y >= n - 3 else 1.0 / (4.0 * y * (y + 1))

    def dy(self, f):
        return torch.einsum("kj,jzx->kzx", self.D, f)

    def points(self, n):
        """[n + 1][ncy]: Chebyshev polynomials on the Gauss-Lobatto points."""
        j = torch.arange(n + 1, dtype=torch.float64, device=self.dev)
        return torch.cos(PI * torch.outer(j, torch.arange(self.ncy, dtype=torch.float64, device=self.dev)) / n)

    def physical(self, f, nx, ny, nz, coarse=False):
        """[ncy][nkz][nkx] -> [ny + 1][nz][nx]."""
        zs, xs = self.m.NZS, self.m.NXS
        P = self.points(ny).to(torch.complex128)
        if ny < self.ncy:
            raise ValueError("fewer points than coefficients")
        F = torch.einsum("jk,kzx->jzx", P, f)
        Z = torch.zeros((ny + 1, nz, nx // 2 + 1), dtype=torch.complex128, device=self.dev)
        Z[:, :zs + 1, :xs + 1] = F[:, zs:]
        if coarse and nz == 2 * zs:   # both Nyquist coefficients share a slot
            Z[:, nz - zs + 1:, :xs + 1] = F[:, 1:zs]
            Z[:, zs, :xs + 1] = F[:, 2 * zs] + F[:, 0]
        elif zs:
            Z[:, nz - zs:, :xs + 1] = F[:, :zs]
        Z = torch.fft.ifft(Z, dim=1, norm="forward")
        if coarse and nx == 2 * xs:
            Z = torch.cat((Z[..., :xs], 2.0 * Z[..., xs:]), dim=2)
        return torch.fft.irfft(Z, n=nx, dim=2, norm="forward")

    def spectral(self, g):
        """[NY2 + 1][NZ2][NX2] -> [ncy][nkz][nkx]."""
        m, zs = self.m, self.m.NZS
        X = torch.fft.rfft(g, dim=2, norm="forward")[:, :, :self.nkx]
        Z = torch.fft.fft(X, dim=1, norm="forward")
        K = torch.cat((Z[:, m.NZ2 - zs:], Z[:, :zs + 1]), dim=1)
        w = torch.full((m.NY2 + 1,), 2.0 / m.NY2, dtype=torch.float64, device=self.dev)
        w[0] = w[-1] = 1.0 / m.NY2
        A = self.points(m.NY2).T * w[None, :]
        A = torch.cat((0.5 * A[:1], A[1:])).to(torch.complex128)
        return torch.einsum("kj,jzx->kzx", A, K)

    def wall_sums(self, f):
        s = ((-1.0) ** (torch.arange(self.ncy, device=self.dev) + 1)).to(torch.complex128)
        return f.sum(0), (s[:, None, None] * f).sum(0)

    def nonlinear(self, u):
        iax, iaz = 1j * self.ax, 1j * self.az
        o = (self.dy(u[2]) - iaz * u[1], iaz * u[0] - iax * u[2], iax * u[1] - self.dy(u[0]))
        m = self.m
        a = [self.physical(f, m.NX2, m.NY2, m.NZ2) for f in u]
        b = [self.physical(f, m.NX2, m.NY2, m.NZ2) for f in o]
        N = [self.spectral(a[(k + 1) % 3] * b[(k + 2) % 3] - a[(k + 2) % 3] * b[(k + 1) % 3]) for k in range(3)]
        return N, self.wall_sums((iax * o[2] - iaz * o[0]) / self.p.Re + N[1])

    def pivots(self, g):
        n, w = self.m.NYS, -(self.ax ** 2 + self.az ** 2 + g)
        ad = [torch.zeros_like(w)] * (n + 3)
        for y in (n, n - 1):
            ad[y] = 1.0 / (1.0 + self.WD[y] * w)
        for y in range(n - 2, 1, -1):
            ad[y] = 1.0 / (1.0 + (self.WD[y] - self.WR[y] * self.WL[y + 2] * w * ad[y + 2]) * w)
        return w, ad

    def tau(self, g, a, b, lower, upper, wad, r):
        """(D^2 - k^2 - g) f = r with a f + b f' given at y = +1 and y = -1."""
        w, ad = wad
        n, z = self.m.NYS, self.m.NZS
        r = list(r.unbind(0))
        zero = torch.zeros_like(r[0])
        singular = g == 0.0 and a == 0.0
        if singular:   # the zero mode: closed by the mean, its even chain starts at zero
            corr = sum(r[y] / (y * y - 1.0) for y in range(2, n + 1, 2))
            if b != 0.0:
                corr = corr + (lower + upper) / (2.0 * b)
            at = torch.zeros(zero.shape, dtype=torch.bool, device=self.dev)
            at[z, 0] = True
            r[0] = torch.where(at, corr, r[0])
        r = r + [zero, zero]
        x = [(lower + upper) / 2.0, (lower - upper) / 2.0]
        x += [self.WL[y] * r[y - 2] + self.WD[y] * r[y] + self.WR[y] * r[y + 2] for y in range(2, n + 1)]
        for y in range(n - 2, 1, -1):
            x[y] = x[y] - self.WR[y] * w * ad[y + 2] * x[y + 2]

        def row(y):
            return float((1 - y % 2) * y * y + y % 2) if a == 0.0 and b == 0.0 else a + b * y * y

        piv = [None, None]
        for y in (n, n - 1):
            piv[y % 2] = torch.full_like(w, row(y))
        for y in range(n - 2, -1, -1):
            q = y % 2
            x[q] = x[q] - piv[q] * ad[y + 2] * x[y + 2]
            piv[q] = row(y) - self.WL[y + 2] * w * piv[q] * ad[y + 2]
        if singular:
            x[0] = torch.where(at, zero, x[0])
            piv[0] = torch.where(at, torch.ones_like(w), piv[0])
        x[0], x[1] = x[0] / piv[0], x[1] / piv[1]
        for y in range(2, n + 1):
            x[y] = (x[y] - self.WL[y] * w * x[y - 2]) * ad[y]
        return torch.stack(x)

    def base(self, pa, pb, rp, bp, R, bv):
        """Pressure and the three velocities without the corrections."""
        p = self.p
        P = self.tau(p.G_pre, pa, pb, bp[0], bp[1], self.adp, rp)
        grad = (1j * self.ax * P, self.dy(P), 1j * self.az * P)
        return P, [self.tau(self.g, p.a_V[k], p.b_V[k], bv[k][0], bv[k][1], self.adv, p.Re * (grad[k] - R[k]))
                   for k in range(3)]

    def wall_divergence(self, v):
        y = torch.arange(self.ncy, dtype=torch.float64, device=self.dev)
        s = (-1.0) ** y
        t = 1j * self.ax * v[0] + 1j * self.az * v[2]
        w = (y * y)[:, None, None] * v[1]
        return (t + w).sum(0), (s[:, None, None] * (t - w)).sum(0)

    def influence(self, v):
        d0, d1 = self.wall_divergence(v)
        (i00, i01), (i10, i11) = self.inf_div
        return d1 * i10 - d0 * i11, d0 * i01 - d1 * i00

    def setup(self, g):
        self.g, p, n, z = g, self.p, self.m.NYS, self.m.NZS
        self.adp, self.adv = self.pivots(p.G_pre), self.pivots(g)
        zero = torch.zeros((self.ncy, self.nkz, self.nkx), dtype=torch.complex128, device=self.dev)
        none = (zero[0], zero[0])
        one = torch.ones_like(zero[0])
        res = [self.base(1.0, 0.0, zero, bp, [zero] * 3, [none] * 3) for bp in ((one, zero[0]), (zero[0], one))]
        div = [self.wall_divergence(v) for _, v in res]
        den = div[0][0] * div[1][1] - div[0][1] * div[1][0]
        root = 1.0 if p.a_V[1] == 0.0 else 0.25 / div[0][0][z, 0]
        self.inf_div = []
        for i in range(2):
            w0, w1 = div[i][0] / den, div[i][1] / den
            w0[z, 0], w1[z, 0] = root, 0.0
            self.inf_div.append((w0, w1))
        self.inf = res
        rp = zero.clone()
        rp[0] = float(n - 1)
        for y in range(1, n):
            rp[y] = float(2 * (n - (y + 1) % 2))
        P, v = self.base(1.0, 0.0, rp, none, [zero] * 3, [none] * 3)
        c = self.influence(v)
        self.pb = P + c[0] * res[0][0] + c[1] * res[1][0]
        self.vb = [v[k] + c[0] * res[0][1][k] + c[1] * res[1][1][k] for k in range(3)]
        w = self.adv[0]
        s1 = p.Re + w * self.vb[1][n - 1] - 2.0 * n * p.Re * self.pb[n]
        s1[z, 0] = 1.0
        self.sigma0 = (p.Re + w * self.vb[1][n], s1)
        r = zero.clone()
        r[0, z, 0] = p.Re
        self.unit = [self.tau(g, p.a_V[k], p.b_V[k], none[0], none[0], self.adv, r)[:, z, 0].real for k in (0, 2)]

    def flow(self, column):
        y = torch.arange(0, self.ncy, 2, dtype=torch.float64, device=self.dev)
        return -(column[::2] / (y * y - 1.0)).sum()

    def start(self, u, bc=None):
        """u: [nkz][ncy][nkx][3]; bc: velocity wall data [nkz][2][nkx][3]."""
        self.u = [u[..., k].permute(1, 0, 2) for k in range(3)]
        zero = torch.zeros_like(self.u[0])
        self.u1, self.N1, self.B1 = [zero] * 3, [zero] * 3, (zero[0], zero[0])
        if bc is None:
            bc = torch.zeros((self.nkz, 2, self.nkx, 3), dtype=torch.complex128, device=self.dev)
            bc[self.m.NZS, :, 0, 1] = self.p.V_Microblow0
        self.bv = [(bc[:, 0, :, k], bc[:, 1, :, k]) for k in range(3)]
        self.it = 0

    def step(self):
        p, n, z = self.p, self.m.NYS, self.m.NZS
        self.it += 1
        e = min(self.it, 2)
        a0, a1, b0, b1 = e / p.DT, (1 - e) / (2.0 * p.DT), float(e), float(1 - e)
        if self.it < 3:
            with torch.no_grad():
                self.setup((a0 + a1) * p.Re)
        N, B = self.nonlinear(self.u)
        bp = [b0 * B[i] + b1 * self.B1[i] for i in range(2)]
        R = [a0 * self.u[k] + a1 * self.u1[k] + b0 * N[k] + b1 * self.N1[k] for k in range(3)]
        rp = 1j * self.ax * R[0] + self.dy(R[1]) + 1j * self.az * R[2]
        P, v = self.base(p.a_pre0, p.b_pre0, rp, bp, R, self.bv)
        c0, c1 = self.influence(v)
        (q0, w0), (q1, w1) = self.inf
        P = P + c0 * q0 + c1 * q1
        v = [v[k] + c0 * w0[k] + c1 * w1[k] for k in range(3)]
        w = self.adv[0]
        s0 = (-w * v[1][n] - p.Re * R[1][n]) / self.sigma0[0]
        s1 = (-w * v[1][n - 1] + p.Re * (2.0 * n * P[n] - R[1][n - 1])) / self.sigma0[1]
        odd = (torch.arange(self.ncy, device=self.dev) % 2 == 1)[:, None, None]
        same, other = torch.where(odd, s0, s1), torch.where(odd, s1, s0)
        P = P + same * self.pb
        v = [v[k] + (other if k == 1 else same) * self.vb[k] for k in range(3)]
        zero_mode = torch.zeros(v[0].shape, dtype=torch.bool, device=self.dev)
        zero_mode[:, z, 0] = True
        keep = torch.zeros_like(v[1][:, z, 0])
        keep = torch.cat(((0.5 * (self.bv[1][0][z, 0] + self.bv[1][1][z, 0])).reshape(1), keep[1:]))
        v[1] = torch.where(zero_mode, keep[:, None, None], v[1])
        if p.INDEX_GRAD_PRE == 1:
            self.dp = [-math.cos(p.THETA * PI / 180.0), -math.sin(p.THETA * PI / 180.0)]
        else:
            want = (math.cos(p.THETA * PI / 180.0), math.sin(p.THETA * PI / 180.0))
            self.dp = [float((want[i] - self.flow(v[2 * i][:, z, 0].real)) / self.flow(self.unit[i])) for i in (0, 1)]
        for i in (0, 1):
            v[2 * i] = v[2 * i] + torch.where(zero_mode, (self.dp[i] * self.unit[i])[:, None, None], 0.0)
        self.u1, self.u, self.N1, self.B1, self.P = self.u, v, N, B, P

    def velocity(self):
        return torch.stack([f.permute(1, 0, 2) for f in self.u], dim=-1)

    def wall_shear(self):
        y = torch.arange(0, self.ncy, 2, dtype=torch.float64, device=self.dev)
        return -(y * y * self.u[0][::2, self.m.NZS, 0].real).sum() / self.p.Re

    def moments(self):
        """Plane means [20][NY + 1] in the order the running means are read."""
        m = self.m
        u, v, w, p = (self.physical(f, m.NX, m.NY, m.NZ, coarse=True) for f in self.u + [self.P])
        p = p - 0.5 * (u * u + v * v + w * w)
        terms = (u, v, w, p, u * u, v * v, w * w, u * v, v * w, w * u, p * p, p * u, p * v, p * w,
                 u ** 3, v ** 3, w ** 3, u ** 4, v ** 4, w ** 4)
        return torch.stack([t.mean(dim=(1, 2)) for t in terms])


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "ensemble":
        if c["members"] > 12:   # the whole ensemble takes too long: its first members
            pick = 4
        else:
            pick = c["members"]
        out = []
        for i, m in enumerate(_members(c)):
            if i >= pick:
                out.append(None)
                continue
            e = _Exact(_mesh(m), _params(m))
            e.start(_field(_mesh(m), _params(m), seed + 1000 * i))
            for _ in range(2 + c["steps"]):
                e.step()
            out.append(e.velocity())
        return out
    mesh, params = _mesh(c), _params(c)
    e = _Exact(mesh, params)
    if kind == "synthesis":
        f = _spectrum(mesh, seed).permute(1, 0, 2)
        return e.physical(f, mesh.NX2, mesh.NY2, mesh.NZ2).permute(1, 0, 2).contiguous()
    u = _field(mesh, params, seed)
    if kind == "gradient":
        u.requires_grad_(True)
        bc = torch.from_numpy(_control(mesh, seed)).to(e.dev).requires_grad_(True)
        e.start(u, bc)
        J = 0.0
        for _ in range(c["steps"]):
            e.step()
            J = J + e.wall_shear() / c["steps"]
        gu, gb = torch.autograd.grad(J, (u, bc))
        return J.detach(), gu, gb
    e.start(u)
    if kind == "restart":
        for _ in range(c["steps"]):
            e.step()
        return e.velocity(), e.P.permute(1, 0, 2).contiguous(), np.array(e.dp)
    for _ in range(2):
        e.step()
    means, dp = 0.0, np.zeros(2)
    for _ in range(c["steps"]):
        e.step()
        if kind == "sampled":
            means = means + e.moments() / c["steps"]
            dp += np.array(e.dp) / c["steps"]
    return (e.velocity(), dp, means) if kind == "sampled" else e.velocity()
