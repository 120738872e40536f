"""Register-form transforms with run-time factors (csrc/any_length.cu): every
class of split (largest factor up to 16, 20, 25), odd lengths, full and
truncated spectra, against the oracle's nonlinear term (all nine transforms
and the products).  The bound is the transform tolerance of the other tests:
1e-12 of the largest value, some 4 n log2(n) eps of a length-n transform."""
import numpy as np
import pytest

import cdns
from oracle_cases import band_spectrum, orc
from test_gpu_parity import ctx_for

pytestmark = pytest.mark.gpu

PI = float(np.pi)


def mesh(NXS, NYS, NZS, NX2, NY2, NZ2):
    m = orc.Mesh(max(2 * NXS, 4), max(NYS, 4), max(2 * NZS, 4), NXS, NYS, NZS, NX2, NY2, NZ2, 4.0 * PI, 2.0 * PI)
    return m, orc.Parm(Re=180.0, DT=5e-5)


def check_nonlinear(m, p):
    ctx = ctx_for(m, p)
    cst = orc.make_constants(m, p.Re)
    u = [band_spectrum(m, seed=31 + k) for k in range(3)]
    N, _, B = orc.nonlinear_term(m, cst, u)
    got, bc = ctx.nonlinear(np.stack(u, axis=-1))
    scale = max(np.abs(n).max() for n in N)
    for k in range(3):
        assert np.abs(got[..., k] - N[k]).max() <= 1e-12 * scale
    bscale = max(np.abs(B[0]).max(), np.abs(B[1]).max(), scale)
    for w in range(2):
        assert np.abs(bc[:, w] - B[w]).max() <= 1e-12 * bscale * (m.NYS + 1)
    return ctx


# 15, 45, 75, 147, 225: odd; 12 .. 256: factors to 16; 162, 200, 288: to 20; 147, 250, 252 (14 x 18), 384: to 25
X_LENGTHS = [12, 15, 30, 45, 75, 98, 126, 147, 162, 200, 225, 240, 250, 252, 256, 288, 384]


@pytest.mark.parametrize("n", X_LENGTHS)
def test_x_lengths(n):
    check_nonlinear(*mesh((n - 1) // 2, 6, 3, n, 8, 9))
    check_nonlinear(*mesh(n // 3, 5, 2, n, 8, 7))


@pytest.mark.parametrize("n", X_LENGTHS)
def test_z_lengths(n):
    check_nonlinear(*mesh(4, 6, (n - 1) // 2, 10, 8, n))
    check_nonlinear(*mesh(9, 5, n // 3, 21, 8, n))


@pytest.mark.parametrize("n", [9, 12, 15, 24, 30, 75, 90, 162, 384])
def test_no_streamwise_modes(n):
    """NXS = 0: one line of x (nkx = 1), more output lines per block than points at 9 and 12."""
    check_nonlinear(*mesh(0, 6, 3, n, 8, 9))
    check_nonlinear(*mesh(0, 5, 0, n, 12, 15))


@pytest.mark.parametrize("nx2,nz2", [(30, 20), (36, 90), (200, 18)])
def test_full_spectrum(nx2, nz2):
    """Nyquist modes kept (NX2 = 2 NXS, NZ2 = 2 NZS)."""
    check_nonlinear(*mesh(nx2 // 2, 6, nz2 // 2, nx2, 8, nz2))


@pytest.mark.parametrize("ny2,nys", [(12, 12), (12, 5), (30, 20), (50, 33), (90, 60), (126, 84), (162, 107),
                                     (200, 131), (250, 166), (252, 252), (288, 191), (384, 255)])
def test_y_lengths(ny2, nys, monkeypatch):
    monkeypatch.setenv("CDNS_Y_TRANSFORM", "fft")
    ctx = check_nonlinear(*mesh(7, nys, 3, 18, ny2, 9))
    assert ctx.tuning()["y_synthesis"] == "fft"
