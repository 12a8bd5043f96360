"""
Zone-wise kernels on grids of more zones than one grid of threads, where each
thread steps through its rows and columns without a division: rows shorter
and longer than the step, one row, one column. Against the oracle.
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
from sailfish_b200.cbdgam_2d import Solver  # noqa: E402
from sailfish_b200.cbdiso_2d import _as_diagnostic  # noqa: E402
from sailfish_b200.mesh import PlanarCartesian2DMesh  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402


@pytest.mark.parametrize("shape", [(1, 1), (2, 5), (33, 31), (40, 32), (1, 1300001), (650001, 2), (2000, 701), (1001, 606),
                                   (2047, 2051)])
def test_isothermal_zone_kernels(shape):
    ni, nj = shape
    padded = (ni + 4, nj + 4, 3)
    rng = np.random.default_rng(5)
    p = rng.uniform(0.5, 2.0, padded)
    p[..., 1:] -= 1.25
    # softening of 0.5 keeps every force of order one, a sink wide enough to act in some zones only
    m = oh.Mass(0.7, 0.5, 0.25, 0.1, -0.2, 0.5, 2, 3.0, 0.4)
    args = (-4.0, 4.0, -3.0, 3.0)
    k = oh.Kernels("oracle", 1.5)
    u, ws, rate = np.zeros(padded), np.zeros(padded[:2]), np.zeros(padded)
    k.primitive_to_conserved(ni, nj, p, u)
    k.wavespeed(ni, nj, *args, 0.04, 100.0, 1, m, m, p, ws)
    k.point_mass_source_term(ni, nj, *args, m.args(1.0, 1.0), p, rate)

    lib = _capi.lib()
    lib.cbdiso_b200_set_stream(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    dp = torch.from_numpy(p).cuda()
    du, dws, drate = (torch.zeros(a.shape, dtype=torch.float64, device="cuda") for a in (u, ws, rate))
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (dp, du, dws, drate)]
    assert lib.cbdiso_2d_primitive_to_conserved(ni, nj, ptr[0], ptr[1]) == 0
    assert lib.cbdiso_2d_wavespeed(ni, nj, *args, 0.04, 100.0, 1, *m.args(), *m.args(), ptr[0], ptr[2]) == 0
    assert lib.cbdiso_2d_point_mass_source_term(ni, nj, *args, *m.args(1.0, 1.0), ptr[0], ptr[3]) == 0
    assert np.array_equal(du.cpu().numpy(), u)
    assert np.array_equal(dws.cpu().numpy(), ws)
    # pow and exp: an ulp of each of the few terms, against the largest rate
    assert np.abs(drate.cpu().numpy() - rate).max() <= 1e-14 * np.abs(rate).max()


@pytest.mark.parametrize("constant_softening", [True, False])
@pytest.mark.parametrize("shape", [(1, 1), (1, 700001), (350001, 2), (700, 701), (1153, 401)])
def test_gamma_law_reductions(shape, constant_softening):
    ni, nj = shape
    setup = CircumbinaryDisk(eos="gamma-law", domain_radius=6.0, mass_ratio=0.5, eccentricity=0.2,
                             constant_softening=constant_softening)
    mesh = PlanarCartesian2DMesh(-6.0, -6.0, 6.0, 6.0, ni, nj)
    x = -6.0 + (np.arange(ni)[:, None] + 0.5) * 12.0 / ni
    y = -6.0 + (np.arange(nj)[None, :] + 0.5) * 12.0 / nj
    state = setup.primitive_array(0.0, x, y) * np.random.default_rng(6).uniform(0.95, 1.05, shape + (4,))
    diags = [dict(quantity="mdot", which_mass="both", accretion=True),
             dict(quantity="torque", which_mass=1, gravity=True),
             dict(quantity="torque", which_mass="both", accretion=True, radial_cut=(0.2, 1.0))]
    onset = [0.0] * 4
    setup.primitive(0.0, [5.9, 0.0], onset)
    cfg = og.GamConfig(-6.0, 6.0, -6.0, 6.0, ni, nj, alpha=0.1, constant_softening=constant_softening,
                       buffer_is_enabled=True, buffer_surface_density=onset[0], buffer_surface_pressure=onset[3],
                       masses=oh.binary_masses(1.0, 1.0, 0.5, 0.2))
    ref = og.GamOracleSolver(cfg, state, 0.0)
    s = Solver(setup=setup, mesh=mesh, physics=setup.physics, solution=state)
    s._physics = s._physics._replace(diagnostics=[_as_diagnostic(d) for d in diags])
    # the wavespeed is a correctly rounded quotient and root, and a maximum has no order
    assert s.maximum_wavespeed() == ref.maximum_wavespeed()
    got, want = np.array(s.reductions()), np.array(ref.reductions(diags))
    scale = np.abs(np.array(ref.reductions(diags, absolute=True)))
    assert (np.abs(got - want) <= 1e-12 * scale).all()
