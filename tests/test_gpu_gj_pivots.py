"""The panel Gauss-Jordan inverse of the mixed LU's diagonal blocks with its
pivots in every kind of place: identity, reversed, random and cyclic row orders
of a dominant 128-row block (rows of every panel and of all four row slots of a
lane), several matrices per launch, and a zero column reported as LAPACK's info.
The inverse is checked against numpy's at 1e-4 of its largest entry: float32
elimination of 128 rows with multipliers of order one (128 x 6e-8 times a growth
of a few, times the blocks' condition of less than 10)."""
import ctypes

import numpy as np
import pytest

from capytaine_b200 import _lib

pytestmark = pytest.mark.gpu


def _vp(t):
    return ctypes.c_void_p(t.data_ptr() if hasattr(t, "data_ptr") else int(t))


def _solve_block(mats):
    """The 128 x 128 blocks' inverses, through solves with the identity's columns."""
    import torch
    lib = _lib.load()
    n, batch = 128, len(mats)
    K = torch.stack([torch.as_tensor(np.ascontiguousarray(m.T)) for m in mats]).cuda()
    work = torch.empty(int(lib.bem_clu_workspace_bytes(n, batch)) + 1024, dtype=torch.uint8, device="cuda")
    wptr = (work.data_ptr() + 1023) // 1024 * 1024
    piv = torch.empty((batch, n), dtype=torch.int32, device="cuda")
    info = torch.zeros(batch, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    s = _lib.stream_ptr()
    _lib.check(lib.bem_clu_factor(_vp(K), n, n * n, n, n, batch, _vp(piv), _vp(info), _vp(wptr), _vp(err), s))
    X = torch.eye(n, dtype=torch.complex128, device="cuda").repeat(batch, 1, 1).contiguous()
    _lib.check(lib.bem_clu_solve(_vp(wptr), n, batch, _vp(piv), _vp(X), n, n * n, n, _vp(err), s))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    return X.transpose(1, 2).cpu().numpy(), info.cpu().numpy()


def test_inverse_for_every_pivot_order():
    rng = np.random.default_rng(11)
    n = 128
    orders = [np.arange(n), np.arange(n)[::-1], (np.arange(n) + 1) % n, (np.arange(n) + 64) % n,
              (np.arange(n) ^ 1), (np.arange(n) ^ 65), rng.permutation(n), rng.permutation(n)]
    mats = []
    for o in orders:
        m = 0.5 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
        m[np.arange(n), np.arange(n)] += 3.0 * np.exp(1j * rng.uniform(0, 6, n))
        mats.append(m[o])
    X, info = _solve_block(mats)
    assert info.tolist() == [0] * len(mats)
    for m, x in zip(mats, X):
        ref = np.linalg.inv(m)
        assert np.abs(x - ref).max() < 1e-4 * np.abs(ref).max()


@pytest.mark.parametrize("column", [0, 7, 8, 77, 127])
def test_zero_column_is_reported(column):
    m = np.eye(128, dtype=complex) * 2.0
    m[:, column] = 0.0
    _, info = _solve_block([np.eye(128, dtype=complex), m])
    assert info.tolist() == [0, column + 1]


@pytest.mark.parametrize("scale", [1e-36, 1e-30, 1e-19, 2.0 ** -50, 2.0 ** 50, 1e19, 1e30, 1e36])
def test_inverse_at_every_scale(scale):
    # squares of these pivots leave the range of float32, their reciprocals do not
    rng = np.random.default_rng(13)
    n = 128
    m = 0.5 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
    m[np.arange(n), np.arange(n)] += np.exp(1j * rng.uniform(0, 6, n))
    m[:, ::3] *= 3.0  # columns on both sides of a range's edge
    X, info = _solve_block([m * scale])
    assert info.tolist() == [0]
    ref = np.linalg.inv(m * scale)
    assert np.abs(X[0] - ref).max() < 1e-4 * np.abs(ref).max()


@pytest.mark.parametrize("pivot", [1e-40, 1e-42j, np.inf])
def test_pivot_without_a_finite_reciprocal_is_reported(pivot):
    m = np.eye(128, dtype=complex)
    m[41, 41] = pivot
    _, info = _solve_block([m])
    assert info.tolist() == [42]
