"""
A gamma-law buffer of zero width, and one whose onset lies at the origin: its
rate is infinite (a division by zero, a power of zero in the reference), which
takes a zone denser than the target to the floors in one stage. The drop-in
stage against the oracle's.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import host as oh  # noqa: E402
from oracle import host_gam as og  # noqa: E402
from sailfish_b200 import _capi  # noqa: E402


@pytest.mark.parametrize("width", [0.0, 6.0])
@pytest.mark.parametrize("n", [24, 320])  # the row march, the tiles
def test_an_infinite_rate_takes_zones_to_the_floors(n, width):
    p = np.zeros((n + 4, n + 4, 4))
    p[..., 0], p[..., 3] = 2.0, 0.5
    cfg = og.GamConfig(-6.0, 6.0, -6.0, 6.0, n, n, alpha=0.1)
    m1, m2 = oh.Mass(0.6, 0.4, 0.1, 0.0, 0.5, 0.05, 1, 2.0, 0.1), oh.Mass(0.4, -0.6, 0.0, 0.1, -0.4, 0.05, 1, 2.0, 0.1)
    buf = (0.34, 7e-4, 1.0, 1000.0, 6.0, width, 1)  # density, pressure, mass, rate, radius, width, on
    u, want = np.zeros_like(p), np.zeros_like(p)
    k = og.GamKernels("oracle", 1.5)
    k.primitive_to_conserved(n, n, p, u, cfg.gamma_law_index)
    edges, dt = (-6.0, 6.0, -6.0, 6.0), 1e-3 * 24 / n
    k.advance_rk(cfg, *edges, u, p, want, buf, m1, m2, 0.0, dt)
    du, dp = torch.from_numpy(u).cuda(), torch.from_numpy(p).cuda()
    out = torch.zeros_like(dp)
    lib = _capi.lib()
    lib.cbdiso_b200_set_stream(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert lib.cbdgam_b200_set_plm_theta(1.5) == 0
    assert lib.cbdgam_2d_advance_rk(n, n, *edges, *(ctypes.c_void_p(t.data_ptr()) for t in (du, dp, out)),
                                    cfg.gamma_law_index, *buf, *m1.args(), *m2.args(), cfg.alpha, 0.0, dt,
                                    cfg.velocity_ceiling, cfg.cooling_coefficient, cfg.mach_ceiling,
                                    cfg.density_floor, cfg.pressure_floor, int(cfg.constant_softening)) == 0
    got, want = out.cpu().numpy()[2:-2, 2:-2], want[2:-2, 2:-2]
    beyond = np.hypot(*np.meshgrid(*[-6.0 + (np.arange(n) + 0.5) * 12.0 / n] * 2)) > 6.0 - width
    assert np.isfinite(want).all() and (want[beyond] == [1e-10, 0.0, 0.0, 1e-12]).all()
    for q in range(4):
        assert np.abs(got[..., q] - want[..., q]).max() <= 1e-13 * np.abs(want[..., q]).max()
