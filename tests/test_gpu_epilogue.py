"""
The stage's epilogue launch against the standalone reduction of the same
state: the wavespeed maximum bit for bit (the epilogue drops zones by an
estimate, the reduction evaluates every zone exactly), the sums to rounding.
Covers cached gravity factors (RK2), none (RK1, RK3), no cache, a state whose
zones all tie, edges of the tiles, and the generic diagnostics.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sailfish_b200.cbdiso_2d import Solver  # noqa: E402
from sailfish_b200.mesh import PlanarCartesian2DMesh  # noqa: E402
from sailfish_b200.setups import BinaryBondi, CircumbinaryDisk  # noqa: E402

RATES = [dict(quantity="mdot", which_mass=1, accretion=True), dict(quantity="fx", which_mass=2, accretion=True),
         dict(quantity="torque", which_mass="both", gravity=True), dict(quantity="power", which_mass=2, gravity=True)]
GENERIC = [dict(quantity="mdot", which_mass="both", accretion=True),
           dict(quantity="torque", which_mass=1, gravity=True, radial_cut=(0.5, 5.0)), dict(quantity="sigma_m1"),
           dict(quantity="mass")]


def _check(solver, steps=2):
    for _ in range(steps):
        solver.advance(solver.mesh.min_spacing() / solver.maximum_wavespeed() * 0.2)
    fused = solver._read_result().copy()
    state = solver.solution
    solver._reduce_now(True, solver._device_diags)
    alone = solver._read_result()
    assert fused[0] == alone[0]
    # Sums of n terms in two orders differ by at most 2 n eps times the sum of
    # magnitudes; the terms' magnitudes are bounded by the largest rate times n.
    n = state.shape[0] * state.shape[1]
    scale = np.abs(state).max() * (10.0 + 1.0 / 0.05 ** 2) * 16.0
    assert np.abs(fused[1:] - alone[1:]).max() <= 2 * n * 2.0 ** -53 * scale * n


@pytest.mark.parametrize("diagnostics", [RATES, GENERIC], ids=["rates", "generic"])
@pytest.mark.parametrize("rk,cache", [(1, True), (2, True), (2, False), (3, True)])
@pytest.mark.parametrize("shape", [(5, 130), (37, 64), (130, 257)])
def test_epilogue_equals_reduction(shape, rk, cache, diagnostics):
    setup = CircumbinaryDisk(domain_radius=6.0, mass_ratio=0.6, eccentricity=0.2)
    mesh = PlanarCartesian2DMesh(-6.0, -6.0, 6.0, 6.0, *shape)
    physics = dict(setup.physics, diagnostics=diagnostics)
    rng = np.random.default_rng(5)
    x = -6.0 + (np.arange(shape[0])[:, None] + 0.5) * 12.0 / shape[0]
    y = -6.0 + (np.arange(shape[1])[None, :] + 0.5) * 12.0 / shape[1]
    state = setup.primitive_array(0.0, x, y) * rng.uniform(0.9, 1.1, shape + (3,))
    _check(Solver(setup=setup, mesh=mesh, physics=physics, solution=state,
                  options=dict(rk_order=rk, plm_theta=1.5, face_cache=cache)))


@pytest.mark.parametrize("n", [3, 64, 200])
def test_every_zone_ties(n):
    """A uniform wind, globally isothermal: every zone has the maximum."""
    setup = BinaryBondi(bh_mass=1e-9, sink_rate=0.0)
    _check(Solver(setup=setup, mesh=setup.mesh(n), physics=dict(setup.physics, diagnostics=RATES),
                  options=dict(plm_theta=1.5)), steps=1)
