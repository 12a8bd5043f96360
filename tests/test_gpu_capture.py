"""
Gamma-law steps captured in a CUDA graph, an odd number of them, replayed:
states and wavespeed maxima of the same steps taken one by one.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sailfish_b200.cbdgam_2d import Solver  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402


@pytest.mark.parametrize("n", [40, 300])
def test_gamma_steps_replay(n):
    # masses at rest (a captured step keeps its masses), a decelerating state
    setup = CircumbinaryDisk(eos="gamma-law", domain_radius=6.0)
    physics = dict(setup.physics)
    still = setup.point_masses(0.0)
    physics["point_mass_function"] = lambda t: still
    mesh = setup.mesh(n)

    def make():
        return Solver(setup=setup, mesh=mesh, physics=physics)

    a, b = make(), make()
    dt = 0.05 * mesh.min_spacing() / a.maximum_wavespeed()
    b.maximum_wavespeed()
    b.advance(dt)  # kernels loaded before the capture
    a.advance(dt)
    graph = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        b.advance(dt)
    torch.cuda.current_stream().wait_stream(side)
    for _ in range(3):
        a.advance(dt)
        graph.replay()
        assert b.maximum_wavespeed() == a.maximum_wavespeed()
    assert np.array_equal(a.solution, b.solution)
