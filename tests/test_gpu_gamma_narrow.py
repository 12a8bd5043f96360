"""
Which of the gamma-law stage's kernels a large grid takes: never strips that
leave more than a twelfth of their columns idle beside the other kernel's
tiles, whatever the grid's shape (the rule, on the host), and the states of
long narrow grids of more than 1280^2 zones against the oracle.
"""

import ctypes

import numpy as np
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

from oracle import host as oh  # noqa: E402
from oracle import host_gam as og  # noqa: E402
from sailfish_b200 import _capi  # noqa: E402
from sailfish_b200.mesh import PlanarCartesian2DMesh  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402


def columns(ni, nj):
    g = _capi.GamGrid(ni=ni, nj=nj, xl=-1.0, xr=1.0, yl=-1.0, yr=1.0, gamma_law_index=5.0 / 3.0)
    return _capi.lib().cbdgam_b200_stage_columns(ctypes.byref(g))


@pytest.mark.parametrize("zones", [960 * 960, 1280 * 1280, 2048 * 2048])
def test_strips_do_not_idle(zones):
    for nj in list(range(1, 700)) + list(range(1000, 1300, 7)) + [2047, 2048, 2049, 4100, 8000]:
        ni = zones // nj + 1
        c = columns(ni, nj)
        tiles = -(-nj // 32) * 32
        if c != 32 and -(-nj // 128) * ni > 888:  # beyond one wave of one-row strips
            assert c == 128 and -(-nj // c) * c <= 1.08 * tiles, (ni, nj)
        if nj % 128 == 0:
            assert c == 128, (ni, nj)


def test_small_and_square_grids():
    assert [columns(n, n) for n in (1, 64, 97, 200, 256, 512, 900, 1000, 1153, 1280, 1281, 2048, 4096)] == [
        64, 64, 128, 128, 32, 32, 32, 128, 32, 128, 128, 128, 128]
    assert columns(0, 4) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(13000, 130), (12800, 128), (28000, 60), (8000, 260)])
def test_two_steps_against_the_oracle(shape):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from sailfish_b200.cbdgam_2d import Solver

    ni, nj = shape
    setup = CircumbinaryDisk(eos="gamma-law", domain_radius=6.0, mass_ratio=0.5, eccentricity=0.2)
    mesh = PlanarCartesian2DMesh(-6.0, -6.0, 6.0, 6.0, ni, nj)
    x = -6.0 + (np.arange(ni)[:, None] + 0.5) * 12.0 / ni
    y = -6.0 + (np.arange(nj)[None, :] + 0.5) * 12.0 / nj
    state = setup.primitive_array(0.0, x, y) * np.random.default_rng(8).uniform(0.95, 1.05, shape + (4,))
    onset = [0.0] * 4
    setup.primitive(0.0, [5.9, 0.0], onset)
    cfg = og.GamConfig(-6.0, 6.0, -6.0, 6.0, ni, nj, alpha=0.1, buffer_is_enabled=True,
                       buffer_surface_density=onset[0], buffer_surface_pressure=onset[3],
                       masses=oh.binary_masses(1.0, 1.0, 0.5, 0.2))
    ref = og.GamOracleSolver(cfg, state, 0.0)
    s = Solver(setup=setup, mesh=mesh, physics=setup.physics, solution=state)
    for _ in range(2):
        dt = mesh.min_spacing() / s.maximum_wavespeed() * 0.05
        s.advance(dt)
        ref.advance(dt)
    got, want = s.solution, ref.solution
    # one ulp of a zone's powers where glibc misrounds, over four stages: below
    # 1e-13 of a field's maximum
    for q in range(4):
        assert np.abs(got[..., q] - want[..., q]).max() <= 1e-13 * np.abs(want[..., q]).max()
    assert np.mean(got != want) < 0.02
