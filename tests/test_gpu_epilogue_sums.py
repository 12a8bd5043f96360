"""
The sums that a step's epilogue leaves, against the oracle's on the same state,
within rounding: sinks whose reach crosses a tile's columns and rows, the
grid's corner and each other, with and without cached gravity factors.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import host as oh  # noqa: E402
from sailfish_b200.cbdiso_2d import Solver  # noqa: E402
from sailfish_b200.mesh import PlanarCartesian2DMesh  # noqa: E402
from sailfish_b200.physics import PointMass, SinkModel  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402

RATES = [dict(quantity="mdot", which_mass=1, accretion=True), dict(quantity="torque", which_mass=2, accretion=True),
         dict(quantity="torque", which_mass="both", gravity=True), dict(quantity="fx", which_mass=2, gravity=True)]
GENERIC = [dict(quantity="mdot", which_mass="both", accretion=True),
           dict(quantity="torque", which_mass=1, gravity=True, radial_cut=(0.5, 5.0)), dict(quantity="mass"),
           dict(quantity="torque", which_mass="both", accretion=True)]


def _scale(ref, d, x, y):
    if d["quantity"] != "torque":
        return abs(ref.reductions([d], absolute=True)[0]) / (ref.cfg.dx * ref.cfg.dy)
    which = (1, 2) if d["which_mass"] == "both" else (d["which_mass"],)
    rates = [ref.source_rates(w, gravity=not d.get("accretion"), accretion=d.get("accretion", False)) for w in which]
    return sum((np.abs(x * r[..., 2]) + np.abs(y * r[..., 1])).sum() for r in rates)


@pytest.mark.parametrize("diagnostics", [RATES, GENERIC], ids=["rates", "generic"])
@pytest.mark.parametrize("rk,cache", [(1, True), (2, True), (2, False), (3, True)])
@pytest.mark.parametrize("at", [((0.1, -0.02), (5.9, 5.9)), ((-5.95, 0.0), (-5.6, 0.3)), ((0.0, 0.0), (0.02, 0.01))])
@pytest.mark.parametrize("shape", [(37, 64), (130, 257)])
def test_sums_against_the_oracle(shape, at, rk, cache, diagnostics):
    ni, nj = shape
    setup = CircumbinaryDisk(domain_radius=6.0, nu=1e-3, buffer_is_enabled=False)
    mesh = PlanarCartesian2DMesh(-6.0, -6.0, 6.0, 6.0, ni, nj)
    # sinks of radius 0.15 and 0.25: they reach 0.6 and 1.0 far
    m = [(0.6, *at[0], 0.2, -0.1, 0.05, 1, 8.0, 0.15), (0.4, *at[1], -0.3, 0.15, 0.05, 1, 5.0, 0.25)]
    pair = tuple(PointMass(*v[:6], SinkModel(v[6]), *v[7:]) for v in m)
    x = -6.0 + (np.arange(ni)[:, None] + 0.5) * 12.0 / ni
    y = -6.0 + (np.arange(nj)[None, :] + 0.5) * 12.0 / nj
    state = setup.primitive_array(0.0, x, y) * np.random.default_rng(5).uniform(0.9, 1.1, shape + (3,))
    s = Solver(setup=setup, mesh=mesh, solution=state, options=dict(rk_order=rk, plm_theta=1.5, face_cache=cache),
               physics=dict(setup.physics, diagnostics=diagnostics, point_mass_function=lambda t: pair))
    cfg = oh.Config(-6.0, 6.0, -6.0, 6.0, ni, nj, nu=1e-3, masses=lambda t: tuple(oh.Mass(*v) for v in m))
    # Terms of a few roundings each, added up in another order: 2 n + 64 roundings of the sum of magnitudes at most,
    # a torque's terms being x f_y and y f_x (which cancel in a zone where the force points at the origin).
    bound = (2 * ni * nj + 64) * 2.0 ** -53
    for _ in range(2):
        s.advance(mesh.min_spacing() / s.maximum_wavespeed() * 0.2)
        ref = oh.OracleSolver(cfg, s.solution, 0.0, oh.Kernels("oracle", 1.5))
        got, want = np.array(s.reductions()), np.array(ref.reductions(diagnostics))
        scale = np.array([_scale(ref, d, x, y) for d in diagnostics]) * cfg.dx * cfg.dy
        assert scale.min() > 0.0
        assert (np.abs(got - want) <= bound * scale).all(), (got, want, scale)
