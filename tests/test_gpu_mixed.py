"""Mixed-precision step (CDNS_PRECISION_MIXED): FP32 fine-grid stages and FFTs,
FP64 curl, Chebyshev accumulation, tau solves, corrections and mean flow.
Compared against the FP64 path of the same library (itself pinned to the
reference at 1e-10): the nonlinear term to FP32 round-off, time steps to
relative L2 <= 1e-6 per velocity component at 48^3, and the Re_tau180 bound
of the precision form after 1000 steps: velocity field relative L2 <= 1e-6,
the errors of the mean profile and Reynolds stresses reported and bounded,
and the per-component bound as a strict expected failure at the measured
floor of FP32 FFT arithmetic."""
import numpy as np
import pytest

import cdns
from oracle_cases import channel_case, divergence_free_field, orc, retau180_case
from test_gpu_parity import ODD_RADIX_MESHES, ctx_for, odd_radix_case

pytestmark = pytest.mark.gpu


def mixed_ctx_for(m, p):
    mesh = cdns.Mesh(m.NX, m.NY, m.NZ, m.NXS, m.NYS, m.NZS, m.NX2, m.NY2, m.NZ2, m.XL, m.ZL)
    params = cdns.Params(Re=p.Re, DT=p.DT, G_pre=p.G_pre, a_pre0=p.a_pre0, b_pre0=p.b_pre0,
                         a_V=p.a_V, b_V=p.b_V, INDEX_GRAD_PRE=p.INDEX_GRAD_PRE, THETA=p.THETA,
                         V_Microblow0=p.V_Microblow0)
    return cdns.Context(mesh, params, precision=cdns.PRECISION_MIXED)


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def run(ctx, u0, nsteps):
    ctx.set_velocity(np.stack(u0, axis=-1))
    ctx.run(1, nsteps)
    ctx.synchronize()
    return ctx.get_velocity()


def test_mixed_nonlinear_term_48():
    m, p = channel_case(32)
    u0 = divergence_free_field(m, p, seed=0, amp=0.05, kmax=4)
    u = np.stack(u0, axis=-1)
    N64, B64 = ctx_for(m, p).nonlinear(u)
    N32, B32 = mixed_ctx_for(m, p).nonlinear(u)
    for k in range(3):
        assert rel_l2(N32[..., k], N64[..., k]) <= 1e-5
    # B cancels to round-off here: scale by the N_y endpoint sums it is made of
    scale = max(np.abs(B64).max(), np.abs(N64[..., 1]).max() * (m.NYS + 1))
    assert np.abs(B32 - B64).max() <= 1e-5 * scale


def test_mixed_stage_buffers_are_fp32_rounded(monkeypatch):
    """The synthesised vorticity of the mixed path is the FP64 one rounded to
    FP32 (fields 3-5 of the synthesis buffer; 0-2 are reused by the forward z
    transform), except the (kz, kx) = (0, 0) mean profile, which stays FP64
    outside the FP32 stages and is zero there.  Both synthesise in the matrix
    form (the FP32 stages have no FFT form)."""
    monkeypatch.setenv("CDNS_Y_TRANSFORM", "matrix")
    m, p = channel_case(32)
    u = np.stack(divergence_free_field(m, p, seed=2, amp=0.05, kmax=4), axis=-1)
    c64, c32 = ctx_for(m, p), mixed_ctx_for(m, p)
    c64.nonlinear(u)
    c32.nonlinear(u)
    f64 = c64.debug_buffer(0)
    f32 = c32.debug_buffer(0)
    expect = f64[3:].astype(np.complex64).astype(np.complex128)
    expect[:, :, m.NZS, 0] = 0.0
    assert np.array_equal(f32[3:], expect)


def test_mixed_steps_48():
    m, p = channel_case(32)
    u0 = divergence_free_field(m, p, seed=0, amp=0.05, kmax=4)
    v64 = run(ctx_for(m, p), u0, 50)
    v32 = run(mixed_ctx_for(m, p), u0, 50)
    for k in range(3):
        assert rel_l2(v32[..., k], v64[..., k]) <= 1e-6


def run_sampled(ctx, u0, nsteps):
    """nsteps steps from u0 with a statistics sample after every step
    (Simulation::run with Nstat = 0); returns (velocity, running means)."""
    ctx.set_velocity(np.stack(u0, axis=-1))
    ctx.statistics_reset()
    for it in range(1, nsteps + 1):
        ctx.step(it)
        ctx.statistics_sample()
    ctx.synchronize()
    return ctx.get_velocity(), ctx.statistics_read()[2]


def statistics_errors(means32, means64):
    """Relative L2 errors over y of the mean profile U and of the Reynolds
    stresses <u_i u_j> - <u_i><u_j> (uu, vv, ww, uv), from the running means
    in Statistics::write's order (u v w, p, uu vv ww uv vw wu, ...)."""
    def stresses(mn):
        u, v, w = mn[0], mn[1], mn[2]
        return {"uu": mn[4] - u * u, "vv": mn[5] - v * v, "ww": mn[6] - w * w, "uv": mn[7] - u * v}
    out = {"U": rel_l2(means32[0], means64[0])}
    r32, r64 = stresses(means32), stresses(means64)
    for k in r64:
        out[k] = rel_l2(r32[k], r64[k])
    return out


@pytest.fixture(scope="module")
def retau180_1000():
    m, p = retau180_case()
    u0 = divergence_free_field(m, p, seed=1, amp=0.1, spectrum="k53", mean="loglaw")
    v64, s64 = run_sampled(ctx_for(m, p), u0, 1000)
    v32, s32 = run_sampled(mixed_ctx_for(m, p), u0, 1000)
    return m, p, v64, s64, v32, s32


def test_mixed_retau180_1000_steps(retau180_1000):
    """The precision form after 1000 Re_tau180 steps against the FP64 path:
    relative L2 of the whole velocity field <= 1e-6, every component's error
    below 1e-6 of the field norm, the mean profile and the Reynolds stresses
    (running means of a statistics sample after every step) within 1e-6
    relative L2 over y, and a finite, divergence-free field."""
    m, p, v64, s64, v32, s32 = retau180_1000
    assert rel_l2(v32, v64) <= 1e-6
    norm = np.linalg.norm(v64)
    for k in range(3):
        assert np.linalg.norm(v32[..., k] - v64[..., k]) <= 1e-6 * norm
    errs = statistics_errors(s32, s64)
    print("mixed vs fp64 after 1000 steps:", {k: f"{v:.2e}" for k, v in errs.items()},
          "per component", [f"{rel_l2(v32[..., k], v64[..., k]):.2e}" for k in range(3)])
    assert all(v <= 1e-6 for v in errs.values())   # measured: U 4.8e-10, stresses 1.7e-8 to 2.1e-7
    cst = orc.make_constants(m, p.Re)
    div = orc.divergence(cst, [v32[..., k] for k in range(3)])
    assert np.abs(div).max() <= 1e-12 * max(1.0, np.abs(v32).max())


@pytest.mark.xfail(strict=True, reason="floor of FP32 FFT arithmetic: per-component relative L2 after 1000 "
                                       "steps measured u 1.3e-7, v 2.7e-6, w 3.8e-6")
def test_mixed_retau180_1000_steps_per_component(retau180_1000):
    """The precision form's stated bound taken per velocity component:
    relative L2 of each of u, v, w <= 1e-6 after 1000 steps.  v and w, whose
    norms are 10-30x smaller than u's, do not meet it: FP32 FFT arithmetic
    leaves 3e-7 to 5e-7 relative error in each evaluation of u x omega (in
    its x and z components), and the difference to the FP64 path grows about
    linearly with the steps.  Moving the mean-flow terms M x omega' and
    u' x M_omega of the product into FP64 lowers only the y component's error,
    so the floor is that of the fluctuation products' FP32 transforms."""
    _, _, v64, _, v32, _ = retau180_1000
    for k in range(3):
        assert rel_l2(v32[..., k], v64[..., k]) <= 1e-6


@pytest.mark.parametrize("key", sorted(ODD_RADIX_MESHES))
def test_mixed_rejects_meshes_without_register_form(key):
    m, p = odd_radix_case(key)
    with pytest.raises(cdns.CdnsError, match="mixed precision"):
        mixed_ctx_for(m, p)


@pytest.mark.parametrize("shape", [(48, 84, 112, 72, 126, 192), (120, 64, 60, 192, 98, 96), (32, 32, 32, 48, 48, 48)])
@pytest.mark.parametrize("flow", ["rate", "gradient"])
def test_mixed_pressure_and_gradient(shape, flow):
    """What the mixed form gives beside the velocity, eight steps: dp/dx of a constant flow
    rate divides FP32 noise of the mean flux by the flux of a unit gradient over one step
    and is good to 1e-5 (1e-6 to 6e-6 seen over 24 to 128 points a side), the pressure to
    3e-6 (1e-7 to 8e-7 seen); the velocity to 1e-7 (1e-9 to 3e-8 seen)."""
    nx, ny, nz, nx2, ny2, nz2 = shape
    box = (10.0, 10.0) if flow == "rate" else (4.0 * np.pi, 2.0 * np.pi)
    m = orc.Mesh(nx, ny, nz, nx // 2, ny - 2, nz // 2, nx2, ny2, nz2, *box)
    p = orc.Parm(Re=2800.0, DT=3e-3, INDEX_GRAD_PRE=0, V_Microblow0=1e-3) if flow == "rate" else orc.Parm(Re=180.0, DT=5e-5)
    u0 = divergence_free_field(m, p, seed=3, amp=0.1, spectrum="k53", mean="laminar" if flow == "rate" else "loglaw")
    ctxs = [ctx_for(m, p), mixed_ctx_for(m, p)]
    u64, u32 = (run(c, u0, 8) for c in ctxs)
    (g64, p64), (g32, p32) = ((np.array(c.dpdx()), c.get_pressure()) for c in ctxs)
    assert rel_l2(u32, u64) <= 1e-7
    assert rel_l2(p32, p64) <= 3e-6
    assert rel_l2(g32, g64) <= 1e-5


@pytest.mark.parametrize("form", ["matrix", "fft"])
def test_mixed_chebyshev_forms(form, monkeypatch):
    """Both forms of the Chebyshev transforms on the FP32 stage buffers (the
    FFT form writes FP32 rows and keeps the mean profiles in FP64; its analysis
    widens FP32 input and applies 1/(NX2 NZ2)): the mixed nonlinear term
    against the FP64 one, at the bound of test_mixed_nonlinear_term_48."""
    m, p = channel_case(32)
    u = np.stack(divergence_free_field(m, p, seed=0, amp=0.05, kmax=4), axis=-1)
    N64, B64 = ctx_for(m, p).nonlinear(u)
    monkeypatch.setenv("CDNS_Y_TRANSFORM", form)
    c32 = mixed_ctx_for(m, p)
    assert c32.tuning()["y_synthesis"] == form and c32.tuning()["y_analysis"] == form
    N32, B32 = c32.nonlinear(u)
    for k in range(3):
        assert rel_l2(N32[..., k], N64[..., k]) <= 1e-5
    scale = max(np.abs(B64).max(), np.abs(N64[..., 1]).max() * (m.NYS + 1))
    assert np.abs(B32 - B64).max() <= 1e-5 * scale
