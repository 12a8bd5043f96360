"""
Isothermal steps captured in a CUDA graph, mixed with steps taken one by one:
the states after every step, and the wavespeed and sums after steps that the
solver took itself, equal those of a solver without a graph. Every stage's
record travels with its launch, so a capture holds all that its steps need.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sailfish_b200.cbdiso_2d import Solver  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402


@pytest.mark.parametrize("order", ["c0e0e", "ec00e", "cec10e01e"])  # e: a step now, c: capture one, a digit: replay it
@pytest.mark.parametrize("rk,cache", [(1, False), (2, True), (2, False), (3, True)])
@pytest.mark.parametrize("n", [40, 300])
def test_mixed_steps(n, rk, cache, order):
    setup = CircumbinaryDisk(domain_radius=6.0, nu=1e-3)
    still = setup.point_masses(0.0)  # masses at rest: a captured step keeps its masses
    physics = dict(setup.physics, point_mass_function=lambda t: still,
                   diagnostics=[dict(quantity="mdot", which_mass=1, accretion=True),
                                dict(quantity="torque", which_mass="both", gravity=True)])
    mesh = setup.mesh(n)
    plain, mixed = (Solver(setup=setup, mesh=mesh, physics=physics,
                           options=dict(rk_order=rk, plm_theta=1.5, face_cache=cache)) for _ in range(2))
    dt = 0.1 * mesh.min_spacing() / plain.maximum_wavespeed()
    for _ in range(2):  # kernels loaded before any capture
        plain.advance(dt)
        mixed.advance(dt)
    graphs = []
    for op in order:
        if op == "c":
            # an even number: RK1 swaps its two buffers every step
            graphs.append(torch.cuda.CUDAGraph())
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.graph(graphs[-1], stream=side):
                for _ in range(6):
                    mixed.advance(dt)
            torch.cuda.current_stream().wait_stream(side)
            continue
        for _ in range(6):
            plain.advance(dt)
        if op == "e":
            for _ in range(6):
                mixed.advance(dt)
            assert mixed.maximum_wavespeed() == plain.maximum_wavespeed()
            assert mixed.reductions() == plain.reductions()
        else:
            graphs[int(op)].replay()
        assert np.array_equal(mixed.solution, plain.solution)
