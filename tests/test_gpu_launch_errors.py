"""
A launch that the CUDA runtime refuses on the host (a grid of more rows of
CTAs than a launch can have: an explicit tile shape on a very long mesh) fails
its own call only; the next call does not find the error again.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sailfish_b200 import _capi  # noqa: E402
from sailfish_b200.cbdiso_2d import Solver  # noqa: E402
from sailfish_b200.mesh import PlanarCartesian2DMesh  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402


@pytest.mark.parametrize("face_cache", [True, False])
def test_a_refused_launch_leaves_no_error_behind(face_cache):
    setup = CircumbinaryDisk(domain_radius=6.0, nu=1e-3)
    ni = 4 * 65535 + 1  # 4 rows per CTA: 65536 CTAs along an axis that holds 65535
    mesh = PlanarCartesian2DMesh(-6.0, -1e-5, 6.0, 1e-5, ni, 1)
    state = np.ones((ni, 1, 3))
    s = Solver(setup=setup, mesh=mesh, physics=setup.physics, solution=state,
               options=dict(plm_theta=1.5, tile=(64, 4), face_cache=face_cache))
    with pytest.raises(_capi.CbdError):
        s.advance(1e-9)
    # the guard fill of a new solver asks for the last error
    small = Solver(setup=setup, mesh=setup.mesh(16), physics=setup.physics, options=dict(plm_theta=1.5))
    small.advance(1e-4)
    assert np.isfinite(small.solution).all()
