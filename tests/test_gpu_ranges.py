"""
Arguments outside the range of the straight-line quotients, roots and powers:
infinite, huge, tiny, denormal and zero pressures, densities and sound speeds,
heating instead of cooling. The wavespeeds against IEEE arithmetic, bit for
bit; the powers against the C library's; a cooled step against the oracle.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import host_gam as og  # noqa: E402
from sailfish_b200 import _capi  # noqa: E402
from sailfish_b200.cbdgam_2d import Solver  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402

GAMMA = 5.0 / 3.0
PRESSURES = [np.inf, 1e308, 1e300, 1e200, 1.0, 1e-12, 1e-290, 3e-302, 3e-305, 2.5e-308, 4e-315, 5e-324, 0.0]
DENSITIES = [1.0, 1e-10, 1e10, 3e-290, 1e300, 4e-310]


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _wavespeed(p):
    with np.errstate(all="ignore"):
        cs = np.sqrt(p[..., 3] / p[..., 0] * GAMMA)
        return np.maximum(np.maximum(np.abs(p[..., 1] - cs), np.abs(p[..., 1] + cs)),
                          np.maximum(np.abs(p[..., 2] - cs), np.abs(p[..., 2] + cs)))


def _states():
    p = np.zeros((len(DENSITIES), 2 * len(PRESSURES), 4))
    p[..., 0] = np.array(DENSITIES)[:, None]
    p[..., 3] = np.array(PRESSURES + PRESSURES)
    p[:, len(PRESSURES):, 1:3] = 0.3, -0.7  # half of them at rest, where the sound speed is the maximum
    return p


def _padded(p):
    return np.ascontiguousarray(np.pad(p, ((2, 2), (2, 2), (0, 0)), mode="edge"))


def test_gamma_law_wavespeed_array():
    p = _states()
    dp = torch.from_numpy(_padded(p)).cuda()
    ws = torch.zeros(dp.shape[:2], dtype=torch.float64, device="cuda")
    lib = _capi.lib()
    lib.cbdiso_b200_set_stream(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert lib.cbdgam_2d_wavespeed(*p.shape[:2], _ptr(dp), _ptr(ws), GAMMA) == 0
    assert np.array_equal(ws.cpu().numpy()[2:-2, 2:-2], _wavespeed(p), equal_nan=True)


def _grid(ni, nj):
    return _capi.GamGrid(ni=ni, nj=nj, xl=-1.0, xr=1.0, yl=-1.0, yr=1.0, plm_theta=1.5, gamma_law_index=GAMMA,
                         alpha=0.1, mach_ceiling=1e5, velocity_ceiling=1e16, constant_softening=1)


def test_gamma_law_reduced_maximum():
    lib, stream = _capi.lib(), torch.cuda.current_stream().cuda_stream
    g = _grid(1, 1)
    masses = (_capi.Mass * 2)()
    scratch = torch.zeros(int(lib.cbdgam_b200_scratch_bytes(ctypes.byref(g))) // 8, dtype=torch.float64, device="cuda")
    for p in _states().reshape(-1, 1, 1, 4):
        dp, out = torch.from_numpy(_padded(p)).cuda(), torch.zeros(9, dtype=torch.float64, device="cuda")
        assert lib.cbdgam_b200_reduce(ctypes.byref(g), masses, None, 0, _ptr(dp), _ptr(scratch), _ptr(out), stream) == 0
        assert np.array_equal(out[:1].cpu().numpy(), _wavespeed(p).ravel(), equal_nan=True), p


@pytest.mark.parametrize("shape", [(3, 5), (200, 300)])  # the row march and the tiles
@pytest.mark.parametrize("pressure", [1e150, 1e-12, 3e-290, 3e-302, 3e-305, 4e-315])
def test_gamma_law_stage_maximum(shape, pressure):
    """A uniform gas at rest, floors of zero: the maximum that the stage leaves is the written state's."""
    lib, stream = _capi.lib(), torch.cuda.current_stream().cuda_stream
    g = _grid(*shape)
    state = np.zeros(shape + (4,))
    state[..., 0], state[..., 3] = 1.0, pressure
    a = torch.from_numpy(_padded(state)).cuda()
    b, ws = torch.zeros_like(a), torch.zeros(1, dtype=torch.float64, device="cuda")
    st = _capi.GamStage(a=0.0, dt=1e-3)
    assert lib.cbdgam_b200_advance_stage(ctypes.byref(g), ctypes.byref(st), _ptr(a), None, _ptr(b), _ptr(ws), stream) == 0
    out = b.cpu().numpy()[2:-2, 2:-2]
    assert np.array_equal(out[..., 0], state[..., 0])
    assert ws.item() == _wavespeed(out).max()


@pytest.mark.parametrize("cs2", [np.inf, 1e300, 1e-302, 1e-305, 4e-315, 0.0])
def test_isothermal_wavespeed_array(cs2):
    p = np.zeros((5, 7, 3))
    p[..., 0] = 1.0
    p[3:, :, 1:] = 0.3, -0.7
    dp = torch.from_numpy(_padded(p)).cuda()
    ws = torch.zeros(dp.shape[:2], dtype=torch.float64, device="cuda")
    m = [0.0] * 8 + [0]
    lib = _capi.lib()
    lib.cbdiso_b200_set_stream(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert lib.cbdiso_2d_wavespeed(5, 7, -1.0, 1.0, -1.0, 1.0, cs2, 100.0, 1, *m, *m, _ptr(dp), _ptr(ws)) == 0
    cs = np.sqrt(cs2)
    want = np.maximum(np.abs(p[..., 1:] - cs), np.abs(p[..., 1:] + cs)).max(axis=-1)
    assert np.array_equal(ws.cpu().numpy()[2:-2, 2:-2], want)


@pytest.mark.parametrize("mach2", [1e-150, 100.0, 1e150, 1e297, 1e305])
def test_locally_isothermal_wavespeed_array(mach2):
    from oracle import host as oh

    p = _padded(np.ones((5, 7, 3)) * [1.0, 0.0, 0.0])
    dp = torch.from_numpy(p).cuda()
    ws = torch.zeros(dp.shape[:2], dtype=torch.float64, device="cuda")
    m = [oh.Mass(0.5, x, 0.1, 0.0, 0.0, 0.05, 1, 1.0, 0.1) for x in (0.5, -0.5)]
    want = np.zeros(p.shape[:2])
    oh.Kernels("oracle", 1.5).wavespeed(5, 7, -1.0, 1.0, -1.0, 1.0, 0.0, mach2, 2, *m, p, want)
    lib = _capi.lib()
    lib.cbdiso_b200_set_stream(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert lib.cbdiso_2d_wavespeed(5, 7, -1.0, 1.0, -1.0, 1.0, 0.0, mach2, 2, *m[0].args(), *m[1].args(), _ptr(dp),
                                   _ptr(ws)) == 0
    assert np.array_equal(ws.cpu().numpy(), want)


def test_powers_outside_their_safe_range():
    x = np.array([1e-120, 1e-200, 1e120, 1e200, 0.0, np.inf, -0.5, -0.999, -1.0, -0.25])
    dx, out = torch.from_numpy(x).cuda(), torch.zeros(8 * x.size, dtype=torch.float64, device="cuda")
    assert _capi.lib().cbdgam_b200_eval_powers(x.size, _ptr(dx), _ptr(out), torch.cuda.current_stream().cuda_stream) == 0
    got = out.cpu().numpy().reshape(-1, 8)
    with np.errstate(all="ignore"):
        want = np.stack([np.power(x, 3.0), np.power(x, -2.0), np.power(1.0 + x, -1.0 / 3.0)], axis=1)
    # CUDA's and the C library's pow, an ulp or two each
    np.testing.assert_allclose(got[:, [0, 1, 5]], want, rtol=1e-15, atol=0)


@pytest.mark.parametrize("cooling", [1e307, 1e100, 1.0, -0.02])
def test_cooled_step_against_the_oracle(cooling):
    """Cooling arguments that overflow, leave the powers' range, lie in it, and below one (heating)."""
    n = 40
    setup = CircumbinaryDisk(eos="gamma-law", domain_radius=6.0, cooling_coefficient=cooling, buffer_is_enabled=False)
    mesh = setup.mesh(n)
    state = np.ones((n, n, 4)) * np.random.default_rng(3).uniform(0.9, 1.1, (n, n, 4))
    state[..., 1:3] -= 1.0
    physics = dict(setup.physics, buffer_is_enabled=False, point_mass_function=lambda t: (_still(), _still()))
    ref = og.GamOracleSolver(og.GamConfig(-6.0, 6.0, -6.0, 6.0, n, n, alpha=0.1, cooling_coefficient=cooling), state, 0.0)
    s = Solver(setup=setup, mesh=mesh, physics=physics, solution=state)
    dt = 1e-3
    s.advance(dt)
    ref.advance(dt)
    got, want = s.solution, ref.solution
    assert np.isfinite(want).all()
    for q in range(4):
        assert np.abs(got[..., q] - want[..., q]).max() <= 1e-13 * np.abs(want[..., q]).max()


def _still():
    from sailfish_b200.physics import PointMass

    return PointMass()


@pytest.mark.parametrize("shape", [(3, 65), (64, 97), (97, 129), (230, 290), (1000, 1000)])
def test_no_floor_takes_the_same_values(shape):
    """Without a pressure floor the stages test every temperature's range: the same bits on an ordinary state."""
    from sailfish_b200.mesh import PlanarCartesian2DMesh

    setup = CircumbinaryDisk(eos="gamma-law", domain_radius=6.0, mass_ratio=0.5, eccentricity=0.2)
    mesh = PlanarCartesian2DMesh(-6.0, -6.0, 6.0, 6.0, *shape)
    out = []
    for floor in (1e-12, 0.0):
        s = Solver(setup=setup, mesh=mesh, physics=setup.physics, options=dict(pressure_floor=floor))
        dt = mesh.min_spacing() / s.maximum_wavespeed() * 0.02
        for _ in range(3):
            s.advance(dt)
        out.append((s.solution, s.maximum_wavespeed()))
    assert out[0][0][..., 3].min() > 1e-12
    assert np.array_equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
