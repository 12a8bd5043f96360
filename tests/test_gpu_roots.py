"""
The quotient and roots that the kernels compute without the CUDA operators'
slow paths, against the IEEE operations: every result is the rounded one, so
the comparison is for equal bits.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from sailfish_b200 import _capi  # noqa: E402


def _eval(a, b):
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    out = torch.empty(3 * a.size, dtype=torch.float64, device="cuda")
    st = _capi.lib().cbdiso_b200_eval_roots(a.size, ctypes.c_void_p(da.data_ptr()), ctypes.c_void_p(db.data_ptr()),
                                            ctypes.c_void_p(out.data_ptr()),
                                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    return out.cpu().numpy().reshape(-1, 3)


def _signed(rng, mantissa, exponents):
    sign = np.where(rng.random(mantissa.size) < 0.5, -1.0, 1.0)
    return sign * np.ldexp(mantissa, exponents)


@pytest.mark.parametrize("span", [3, 60, 480])
def test_quotient_and_roots_are_ieee(span):
    rng = np.random.default_rng(span)
    n = 2_000_000
    a = _signed(rng, rng.uniform(1.0, 2.0, n), rng.integers(-span, span + 1, n))
    b = _signed(rng, rng.uniform(1.0, 2.0, n), rng.integers(-span, span + 1, n))
    # mantissas next to a power of two, exact squares
    b[0::16] = np.nextafter(np.abs(np.ldexp(1.0, rng.integers(-span, span + 1, b[0::16].size))), np.inf)
    b[1::16] = np.nextafter(np.abs(np.ldexp(1.0, rng.integers(-span, span + 1, b[1::16].size))), 0.0)
    b[2::16] = np.ldexp(1.0, rng.integers(-span, span + 1, b[2::16].size))
    b[3::16] = rng.integers(1, 1 << 26, b[3::16].size).astype(float) ** 2
    out = _eval(a, b)
    root = np.sqrt(np.abs(b))
    assert np.array_equal(out[:, 0], a / b)
    assert np.array_equal(out[:, 1], root)
    assert np.array_equal(out[:, 2], a / root)


def test_zero_and_nonfinite_operands():
    a = np.array([1.0, 0.0, 1.0, np.nan, 1.0])
    b = np.array([0.0, 0.0, np.inf, 1.0, np.nan])
    out = _eval(a, b)
    # a division by zero or infinity does not pass as a finite value
    assert np.isnan(out[:, 0]).all()
    assert out[0, 1] == 0.0 and out[1, 1] == 0.0
    assert not np.isfinite(out[2, 1]) and np.isnan(out[4, 1])


def test_scale_height_geometry_is_correctly_rounded():
    from fractions import Fraction

    rng = np.random.default_rng(11)
    x = np.concatenate([rng.uniform(0.0, 20.0, 4000), np.ldexp(rng.uniform(1.0, 2.0, 2000), rng.integers(-12, 12, 2000)),
                        [0.0]])
    dx = torch.from_numpy(x).cuda()
    out = torch.empty(8 * x.size, dtype=torch.float64, device="cuda")
    assert _capi.lib().cbdgam_b200_eval_powers(x.size, ctypes.c_void_p(dx.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    got = out.cpu().numpy().reshape(-1, 8)[:, 7]
    root = np.sqrt(x * x + 1e-12)
    want = [float(1 / Fraction(float(r)) ** 3) for r in root]  # Fraction to float rounds to nearest
    assert list(got) == want
