"""The refined reciprocals of the kernels against 64-bit mantissas (numpy's long
double) over mantissas and exponents.

Bars: 1 / sqrt(x): half an ulp for the last addition, half for the rounding of
x y inside e, less than a fifth for the terms left out of the series after an
estimate good to 2^-19: 2 ulp.  1 / z: two roundings in |z|^2, one in its
reciprocal (whose Newton step leaves the square of the estimate's error), one in
the product: 4 units of 2^-53 (2^-24 in float32) in each part."""
import ctypes

import numpy as np
import pytest

from capytaine_b200 import _lib

pytestmark = pytest.mark.gpu

wide = np.longdouble
if np.finfo(wide).nmant < 63:
    pytest.skip("needs a long double of 64 bits of mantissa", allow_module_level=True)


def _run(kind, values):
    import torch
    t = torch.as_tensor(values, device="cuda")
    out = torch.empty_like(t)
    _lib.check(_lib.load().bem_reciprocals(kind, t.shape[0], ctypes.c_void_p(t.data_ptr()),
                                           ctypes.c_void_p(out.data_ptr()), _lib.stream_ptr()))
    return out.cpu().numpy()


@pytest.mark.parametrize("low,high", [(-1022, -900), (-60, 60), (-2, 2), (900, 1022)])
def test_reciprocal_square_root(low, high):
    rng = np.random.default_rng(1)
    x = np.ldexp(rng.uniform(1.0, 2.0, 1 << 18), rng.integers(low, high + 1, 1 << 18))
    x[:4] = np.ldexp([1.0, 1.0, np.nextafter(2.0, 1.0), np.nextafter(1.0, 2.0)], [low, high, low, high])
    got = _run(0, x)
    want = 1 / np.sqrt(x.astype(wide))
    assert np.max(np.abs(got.astype(wide) - want) / np.spacing(want.astype(np.float64))) <= 2


# moduli where the squares are in range, where they are not, and across the edge
@pytest.mark.parametrize("kind,u,exponents", [(1, 2.0 ** -53, (-1020, -500)), (1, 2.0 ** -53, (-500, -440)),
                                              (1, 2.0 ** -53, (-100, 100)), (1, 2.0 ** -53, (440, 1020)),
                                              (2, 2.0 ** -24, (-124, -48)), (2, 2.0 ** -24, (-52, -48)),
                                              (2, 2.0 ** -24, (-40, 40)), (2, 2.0 ** -24, (48, 124))])
def test_complex_reciprocal(kind, u, exponents):
    rng = np.random.default_rng(2)
    n = 1 << 18
    z = np.ldexp(rng.uniform(0.5, 1.0, (n, 2)) * rng.choice([-1, 1], (n, 2)), rng.integers(*exponents, (n, 1)))
    z[::3, 0] *= 2.0 ** -rng.integers(0, 4, z[::3].shape[0])  # parts of different sizes
    z[1::3, 1] *= 2.0 ** -rng.integers(0, 4, z[1::3].shape[0])
    if kind == 2:
        z = z.astype(np.float32).astype(np.float64)
    got = _run(kind, z)
    big = np.ldexp(wide(1), -np.max(np.frexp(z)[1], axis=1))  # squares inside the long double's range
    x, y = z[:, 0].astype(wide) * big, z[:, 1].astype(wide) * big
    d = x * x + y * y
    want = np.stack([x / d * big, -y / d * big], axis=1)
    normal = np.abs(want) >= (np.finfo(np.float64).tiny if kind == 1 else np.finfo(np.float32).tiny)
    assert np.mean(normal) > 0.9
    error = np.abs(got.astype(wide) - want) / np.abs(want)
    assert np.max(error[normal]) <= 4 * u
