"""
The fused stage adjoint's segments (one row and up, by the grid's size) against
the separate passes on grids at the edges of strips and segments: lambda_rd and
lambda_n bit for bit, the chained parameter sums to rounding.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sailfish_b200 import _capi  # noqa: E402
from sailfish_b200.adjoint import mass_jacobians  # noqa: E402
from sailfish_b200.cbdiso_2d import Solver  # noqa: E402
from sailfish_b200.mesh import PlanarCartesian2DMesh  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402


@pytest.mark.parametrize("shape", [(1, 1), (2, 120), (7, 121), (130, 64), (149, 363), (300, 241)])
def test_march_equals_passes(shape):
    lib = _capi.lib()
    setup = CircumbinaryDisk(domain_radius=4.0, mass_ratio=0.5, eccentricity=0.1)
    mesh = PlanarCartesian2DMesh(-4.0, -4.0, 4.0, 4.0, *shape)
    rng = np.random.default_rng(3)
    x = -4.0 + (np.arange(shape[0])[:, None] + 0.5) * 8.0 / shape[0]
    y = -4.0 + (np.arange(shape[1])[None, :] + 0.5) * 8.0 / shape[1]
    state = setup.primitive_array(0.0, x, y) * rng.uniform(0.9, 1.1, shape + (3,))
    s = Solver(setup=setup, mesh=mesh, physics=setup.physics, solution=state, options=dict(plm_theta=1.5))
    g = ctypes.byref(s._grid)
    st, ep = _capi.Stage(), s._epilogue(0.01, True, [])
    from sailfish_b200.cbdiso_2d import _mass_struct

    for k, m in enumerate(s._point_masses(0.0)):
        _mass_struct(m, st.mass[k])
    st.a, st.dt, st.buffer_central_mass = 0.5, 0.01 * mesh.min_spacing(), 1.0
    rec = (ctypes.c_char * int(lib.cbdiso_b200_stage_record_bytes()))()
    assert lib.cbdiso_b200_stage_record(g, ctypes.byref(st), ctypes.byref(ep), rec) == 0
    dev = torch.frombuffer(bytearray(rec), dtype=torch.uint8).cuda()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    P = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    p = s._buf[0]
    pn, out = p.clone(), torch.empty_like(p)
    assert lib.cbdiso_b200_advance_stage(g, ctypes.byref(st), P(dev), P(p), P(pn), P(out), None, None, None,
                                         stream) == 0
    lam = torch.zeros_like(p)
    lam[2:-2, 2:-2] = torch.from_numpy(rng.normal(size=shape + (3,))).cuda()
    jac = torch.from_numpy(mass_jacobians(np.array([0.0]), 0.5, 0.1).reshape(20)).cuda()
    got = []
    for variant in (1, 0):
        lib.cbdiso_b200_set_adjoint_variant(variant)
        try:
            rd, ln = torch.zeros_like(p), torch.zeros_like(p)
            ws = torch.zeros(int(lib.cbdiso_b200_adjoint_workspace_bytes(g)) // 8 + 8, dtype=torch.float64, device="cuda")
            rows = int(lib.cbdiso_b200_adjoint_chain_blocks(g))
            acc, par = (torch.zeros(n, dtype=torch.float64, device="cuda") for n in (4 * rows, 4))
            assert lib.cbdiso_b200_stage_adjoint_chained(g, P(dev), P(p), P(pn), P(out), P(lam), P(rd), P(ln), P(jac),
                                                         P(acc), P(ws), stream) == 0
            assert lib.cbdiso_b200_adjoint_chain_finish(P(acc), rows, P(par), stream) == 0
            got.append((rd.cpu().numpy(), ln.cpu().numpy(), par.cpu().numpy(), acc.abs().sum().item()))
        finally:
            lib.cbdiso_b200_set_adjoint_variant(1)
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1])
    # two orders of the same terms: n eps times their magnitudes, which the
    # blocks' partial sums bound from below by their own and cancellation
    # inside a block by a factor of its terms at most
    n = shape[0] * shape[1] * 20
    assert np.abs(got[0][2] - got[1][2]).max() <= n * 2.0 ** -53 * (got[0][3] + got[1][3]) * 128
