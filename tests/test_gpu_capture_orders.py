"""
Captured gamma-law steps mixed with steps taken one by one: captures that are
replayed later, more than once, in another order or not at all. After every
step the wavespeed maximum is that of the state, as the standalone reduction
gives it, and the state that of the same steps without a graph. The state
decelerates, so that a maximum kept from an earlier step would show.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sailfish_b200.cbdgam_2d import Solver, initial_condition  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402


# "e": a step now; "c": capture a step (nothing runs); a digit: replay that capture
@pytest.mark.parametrize("face_cache", [True, False])
@pytest.mark.parametrize("order", ["ce", "ece", "c0e0e", "ce0e0", "ec0ee0", "cc010e1", "cec0e10e", "ccc201e0"])
@pytest.mark.parametrize("n", [40, 300])
def test_every_maximum_is_the_states_own(n, order, face_cache):
    # masses at rest: a captured step keeps its masses
    setup = CircumbinaryDisk(eos="gamma-law", domain_radius=6.0)
    physics = dict(setup.physics)
    still = setup.point_masses(0.0)
    physics["point_mass_function"] = lambda t: still
    mesh = setup.mesh(n)
    state = initial_condition(setup, mesh, 0.0)
    state[n // 3, n // 4, 3] *= 1e4  # one hot zone, cooling as it expands: the maximum falls at every step

    def make(solution=state):
        return Solver(setup=setup, mesh=mesh, physics=physics, solution=solution,
                      options=dict(face_cache=face_cache))

    plain, mixed = make(), make()
    dt = 0.02 * mesh.min_spacing() / plain.maximum_wavespeed()
    mixed.maximum_wavespeed()
    for s in (plain, mixed):
        s.advance(dt)  # kernels loaded before any capture
    graphs, last = [], plain.maximum_wavespeed()
    for op in order:
        if op == "c":
            graphs.append(torch.cuda.CUDAGraph())
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.graph(graphs[-1], stream=side):
                mixed.advance(dt)
            torch.cuda.current_stream().wait_stream(side)
        else:
            plain.advance(dt)
            if op == "e":
                mixed.advance(dt)
            else:
                graphs[int(op)].replay()
            assert np.array_equal(mixed.solution, plain.solution)
        alone = make(plain.solution).maximum_wavespeed()
        assert plain.maximum_wavespeed() == alone
        assert mixed.maximum_wavespeed() == alone
        assert op == "c" or alone < last
        last = alone
