"""The column solve's chains (csrc/solver.cu) at the ends of their row groups: the
smallest NYS and some up to the largest, column counts that do not fill a block, both
forcings, wall conditions that differ between u and w, and the curl that the
solve leaves for the next step (changes of the velocity between steps).  Time
steps against the oracle's loop at the step tolerance (relative L2 <= 1e-10)."""
import numpy as np
import pytest

from oracle_cases import divergence_free_field, orc
from test_gpu_parity import ctx_for

pytestmark = pytest.mark.gpu

PI = float(np.pi)


def channel(NYS, NXS=6, NZS=5, **parm):
    NY2 = max(3 * NYS // 2 + 1, 8)
    m = orc.Mesh(2 * NXS, NYS + 2, 2 * NZS, NXS, NYS, NZS, 3 * NXS + 2, NY2, 3 * NZS + 1, 4.0 * PI, 2.0 * PI)
    p = dict(Re=180.0, DT=1e-4, INDEX_GRAD_PRE=1)
    p.update(parm)
    return m, orc.Parm(**p)


def compare(m, p, nsteps=4, poke=None):
    u0 = divergence_free_field(m, p, seed=7, amp=0.05, kmax=3)
    sim = orc.Simulation(m, p, u0)
    ctx = ctx_for(m, p)
    ctx.set_velocity(np.stack(u0, axis=-1))
    for it in range(1, nsteps + 1):
        with np.errstate(all="ignore"):
            sim.step()
        ctx.step(it)
        if poke:
            poke(it, sim, ctx)
    ctx.synchronize()
    got, pres = ctx.get_velocity(), ctx.get_pressure()
    norm = np.sqrt(sum(np.sum(np.abs(u) ** 2) for u in sim.u))
    for k in range(3):
        assert np.linalg.norm(got[..., k] - sim.u[k]) <= 1e-10 * norm
    assert np.linalg.norm(pres - sim.pressure) <= 1e-9 * np.linalg.norm(sim.pressure)
    return sim, ctx


@pytest.mark.parametrize("NYS", [8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 31, 32, 33, 47])
def test_rows(NYS):
    compare(*channel(NYS))


@pytest.mark.parametrize("NYS", [4, 5, 6, 7, 254, 255])
def test_rows_smallest_and_largest(NYS):
    """4 to 7: no full group of rows, the two top rows next to y = 2, row groups without a
    row.  254 and 255: the largest tile and every held pivot."""
    compare(*channel(NYS, NXS=4, NZS=3))


@pytest.mark.parametrize("NXS,NZS", [(0, 3), (1, 1), (3, 0), (4, 2), (8, 9)])
def test_columns(NXS, NZS):
    compare(*channel(12, NXS=NXS, NZS=NZS))


@pytest.mark.parametrize("a_V,b_V", [((1.0, 1.0, 1.0), (0.0, 0.0, 0.5)), ((1.0, 1.0, 0.7), (0.2, 0.0, 0.1)),
                                     ((0.0, 1.0, 0.0), (1.0, 0.0, 1.0)), ((1.0, 0.8, 1.0), (0.1, 0.05, 0.1))])
@pytest.mark.parametrize("NYS", [13, 16])
def test_wall_conditions(NYS, a_V, b_V):
    compare(*channel(NYS, a_V=a_V, b_V=b_V))


@pytest.mark.parametrize("NYS", [12, 17])
def test_constant_flow_rate(NYS):
    compare(*channel(NYS, INDEX_GRAD_PRE=0, DT=1e-3, Re=500.0, V_Microblow0=1e-3))


@pytest.mark.parametrize("a_V,b_V", [((1.0, 1.0, 1.0), (0.0, 0.0, 0.0)), ((1.0, 1.0, 0.7), (0.2, 0.0, 0.1))])
@pytest.mark.parametrize("NYS", [4, 5, 31, 32, 63, 64, 127, 128, 255])
def test_flux_column(NYS, a_V, b_V):
    """The zero-mode column whose flux gives dp/dx, at the ends of its rows per lane (1,
    2, 4 and 8), u and w together and apart.  dp/dx = (Q - q) / q_unit, q_unit some dt Q:
    a last bit of q is 2.2e-16 / dt = 2.2e-13; 1e-11 for 45 of them after four steps of
    another order.  With 5 or 6 coefficients the column itself loses four digits (every
    order of the solve, warp scans and chains, is 1e-10 to 1e-9 off the oracle's): 1e-8."""
    m, p = channel(NYS, NXS=3, NZS=2, INDEX_GRAD_PRE=0, DT=1e-3, Re=500.0, a_V=a_V, b_V=b_V, V_Microblow0=1e-3)
    sim, ctx = compare(m, p)
    assert abs(ctx.dpdx()[0] - sim.dpdx) <= (1e-8 if NYS < 8 else 1e-11)


def test_velocity_changes_between_steps():
    """The vorticity kept by the solve follows every change of the velocity: a
    disturbance added between steps, and an evaluation of another field."""
    def poke(it, sim, ctx):
        if it == 3:
            for k in range(3):
                sim.u[k] = sim.u[k] * 1.01
            ctx.update_velocity(np.stack(sim.u, axis=-1))
        if it == 4:
            ctx.nonlinear(np.stack([2.0 * u for u in sim.u], axis=-1))
        if it == 5:
            ctx.solve(1234.5, np.stack(sim.u, axis=-1), np.zeros((sim.m.nkz, 2, sim.m.nkx), complex),
                      np.zeros((sim.m.nkz, 2, sim.m.nkx, 3), complex))
    compare(*channel(15), nsteps=7, poke=poke)
