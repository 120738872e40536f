"""cdns_transform_fine_backward_noalloc as the only call of a process: no
context has raised the shared-memory limits of the kernels it launches."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ALONE = """
import sys
sys.path[:0] = [{root!r} + "/channel-dns_b200", {root!r} + "/oracle", {root!r} + "/tests"]
import numpy as np, torch, cdns
from oracle_cases import band_spectrum, channel_case, orc
m, _ = channel_case(32)
mesh = cdns.Mesh(m.NX, m.NY, m.NZ, m.NXS, m.NYS, m.NZS, m.NX2, m.NY2, m.NZ2, m.XL, m.ZL)
U = band_spectrum(m, 3)
src = torch.from_numpy(U.view(np.float64).copy()).cuda()
out = torch.empty(m.fine_shape(), dtype=torch.float64, device="cuda")
cdns.fine_backward_noalloc(mesh, src.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream)
torch.cuda.synchronize()
ref = orc.fine_backward(m, U)
assert np.abs(out.cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()
"""


def test_noalloc_without_a_context():
    r = subprocess.run([sys.executable, "-c", ALONE.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
