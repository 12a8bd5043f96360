"""
The default launch shape of small grids (segments of one to eight rows) gives
the states of an explicit shape bit for bit, and wavespeeds with them.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sailfish_b200.cbdiso_2d import Solver  # noqa: E402
from sailfish_b200.mesh import PlanarCartesian2DMesh  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402


@pytest.mark.parametrize("shape", [(1, 1), (1, 130), (2, 64), (33, 97), (64, 64), (130, 129), (257, 300), (400, 385)])
def test_default_shape_equals_an_explicit_one(shape):
    setup = CircumbinaryDisk(domain_radius=5.0, mass_ratio=0.4, eccentricity=0.3)
    mesh = PlanarCartesian2DMesh(-5.0, -5.0, 5.0, 5.0, *shape)
    x = -5.0 + (np.arange(shape[0])[:, None] + 0.5) * 10.0 / shape[0]
    y = -5.0 + (np.arange(shape[1])[None, :] + 0.5) * 10.0 / shape[1]
    state = setup.primitive_array(0.0, x, y) * np.random.default_rng(2).uniform(0.9, 1.1, shape + (3,))
    runs = []
    for tile in (None, (64, 16), (128, 5)):
        physics = dict(setup.physics, diagnostics=[dict(quantity="mdot", which_mass="both", accretion=True)])
        s = Solver(setup=setup, mesh=mesh, physics=physics, solution=state, options=dict(plm_theta=1.5, tile=tile))
        dts = []
        for _ in range(3):
            dts.append(mesh.min_spacing() / s.maximum_wavespeed() * 0.2)
            s.advance(dts[-1])
        runs.append((dts, s.solution))
    for dts, solution in runs[1:]:
        assert dts == runs[0][0]
        assert np.array_equal(solution, runs[0][1])
