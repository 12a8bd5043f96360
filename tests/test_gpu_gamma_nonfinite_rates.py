"""
Source rates of a gamma-law state with single NaN or infinite values, near and
beyond a sink's reach: the drop-in source term and the reductions give a NaN
or an infinity where the oracle does, and its values elsewhere.
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
from sailfish_b200.cbdiso_2d import _as_diagnostic  # noqa: E402
from sailfish_b200.cbdgam_2d import Solver  # noqa: E402
from sailfish_b200.physics import PointMass, SinkModel  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402

N = 24
GAMMA = 5.0 / 3.0
MODELS = {0: "INACTIVE", 1: "ACCELERATION_FREE", 2: "TORQUE_FREE", 3: "FORCE_FREE"}


def _state():
    rng = np.random.default_rng(2)
    p = rng.uniform(0.5, 1.5, (N, N, 4))
    p[..., 1:3] -= 1.0
    return p


def _same(got, want):
    """Non-finite where the oracle is, its values (to an ulp of each power) where it is finite."""
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    ok = np.isfinite(want)
    assert np.abs(got[ok] - want[ok]).max(initial=0.0) <= 1e-14 * np.abs(want[ok]).max(initial=0.0)


@pytest.mark.parametrize("constant_softening", [True, False])
@pytest.mark.parametrize("model", [0, 1, 2, 3])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("field", [0, 1, 2, 3])
def test_drop_in_source_term(field, value, model, constant_softening):
    p = np.zeros((N + 4, N + 4, 4))
    p[2:-2, 2:-2] = _state()
    # a sink of radius 0.4 at (0.7, 0.5): zones in its reach and far from it
    for i, j in ((2 + N // 2 + 2, 2 + N // 2 + 2), (3, 4), (2 + N - 1, 2 + N - 1)):
        p[i, j, field] = value
    m1 = oh.Mass(0.7, 0.5, 0.25, 0.1, -0.2, 0.05, model, 3.0, 0.4)
    m2 = oh.Mass(0.3, -0.6, -0.3, -0.1, 0.3, 0.05, model, 2.0, 0.2)
    want = np.zeros_like(p)
    k = og.GamKernels("oracle", 1.5)
    args = (m1.args(1.0, 1.0), m2.args(1.0, 1.0), 1)
    k.point_mass_source_term(N, N, -4.0, 4.0, -4.0, 4.0, *args, p, want, constant_softening, GAMMA)
    lib = _capi.lib()
    lib.cbdiso_b200_set_stream(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    dp, dr = torch.from_numpy(p).cuda(), torch.zeros(p.shape, dtype=torch.float64, device="cuda")
    assert lib.cbdgam_2d_point_mass_source_term(N, N, -4.0, 4.0, -4.0, 4.0, *args[0], *args[1], 1,
                                                ctypes.c_void_p(dp.data_ptr()), ctypes.c_void_p(dr.data_ptr()),
                                                int(constant_softening), GAMMA) == 0
    _same(dr.cpu().numpy(), want)


@pytest.mark.parametrize("constant_softening", [True, False])
@pytest.mark.parametrize("model", [1, 2, 3])
@pytest.mark.parametrize("where", [(3, 4), (14, 14)])
@pytest.mark.parametrize("field,value", [(0, np.nan), (1, np.nan), (2, np.nan), (3, np.inf), (0, np.inf)])
def test_reductions(field, value, where, model, constant_softening):
    state = _state()
    state[where][field] = value
    m = [(0.7, 0.5, 0.25, 0.1, -0.2, 3.0, 0.4), (0.3, -0.6, -0.3, -0.1, 0.3, 2.0, 0.2)]  # mass, x, y, vx, vy, rate, radius
    pair = tuple(PointMass(a[0], a[1], a[2], a[3], a[4], 0.05, SinkModel[MODELS[model]], a[5], a[6]) for a in m)
    setup = CircumbinaryDisk(eos="gamma-law", domain_radius=4.0, constant_softening=constant_softening)
    diags = [dict(quantity="mdot", which_mass="both", accretion=True), dict(quantity="mdot", which_mass=2, accretion=True),
             dict(quantity="torque", which_mass=1, accretion=True), dict(quantity="torque", which_mass="both", gravity=True)]
    s = Solver(setup=setup, mesh=setup.mesh(N), solution=state,
               physics=dict(setup.physics, diagnostics=diags, point_mass_function=lambda t: pair))
    cfg = og.GamConfig(-4.0, 4.0, -4.0, 4.0, N, N, constant_softening=constant_softening,
                       masses=lambda t: tuple(oh.Mass(a[0], a[1], a[2], a[3], a[4], 0.05, model, a[5], a[6]) for a in m))
    ref = og.GamOracleSolver(cfg, state, 0.0)
    got, want = np.array(s.reductions()), np.array(ref.reductions(diags))
    assert np.array_equal(np.isfinite(got), np.isfinite(want)), (got, want)
    ok = np.isfinite(want)
    scale = np.abs(np.array(og.GamOracleSolver(cfg, _state(), 0.0).reductions(diags, absolute=True)))
    assert (np.abs(got[ok] - want[ok]) <= 1e-12 * scale[ok]).all()
