"""The float64 LU at the sizes where its blocks, panels and tiles change shape:
factors and triangle inverses against numpy, pivots inside the 64-row blocks.

Bars: the factors are compared through P A = L U, whose backward error is a few
eps times n |L| |U| / |A| (below 1e-12 for these matrices of moderate growth);
the triangles' inverses through L11 inv(L11) = 1, a few eps times 64 times the
blocks' condition (below 1e3 here)."""
import ctypes

import numpy as np
import pytest

from capytaine_b200 import _lib

pytestmark = pytest.mark.gpu


def _vp(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("n,batch", [(64, 1), (128, 5), (192, 2), (448, 3), (832, 1)])
def test_factors_reproduce_the_matrix(n, batch):
    import torch
    rng = np.random.default_rng(n)
    lib = _lib.load()
    mats = []
    for b in range(batch):
        m = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        for k in range(0, n, 64):  # the pivots of each block in a random order of its rows
            m[k + rng.permutation(64), k + np.arange(64)] += 3 * np.sqrt(n)
        mats.append(m)
    A = torch.as_tensor(np.array([m.T for m in mats]), device="cuda").contiguous()
    piv = torch.empty((batch, n), dtype=torch.int32, device="cuda")
    info = torch.zeros(batch, dtype=torch.int32, device="cuda")
    work = torch.empty(int(lib.bem_zlu_workspace_bytes(n, batch)), dtype=torch.uint8, device="cuda")
    _lib.check(lib.bem_zlu_factor(_vp(A), n, n, n * n, batch, _vp(piv), _vp(info), _vp(work), _lib.stream_ptr()))
    F, p = A.cpu().numpy(), piv.cpu().numpy()
    inv = work.cpu().numpy()[:batch * (n // 64) * 2 * 4096 * 16].view(np.complex128).reshape(batch, n // 64, 2, 64, 64)
    assert info.cpu().numpy().tolist() == [0] * batch
    for b in range(batch):
        lu = F[b].T
        L, U = np.tril(lu, -1) + np.eye(n), np.triu(lu)
        rows = np.concatenate([k + p[b, k:k + 64] for k in range(0, n, 64)])
        assert sorted(rows) == list(range(n))
        assert np.abs(L @ U - mats[b][rows]).max() < 1e-12 * np.abs(mats[b]).max()
        for i in range(n // 64):
            s = slice(64 * i, 64 * i + 64)
            for tri, x in ((L[s, s], inv[b, i, 0].T), (U[s, s], inv[b, i, 1].T)):
                assert np.abs(tri @ x - np.eye(64)).max() < 1e-11


@pytest.mark.parametrize("scale", [1e-300, 1e-200, 1e-158, 1e-139, 1e139, 1e158, 1e200, 1e290])
def test_factors_at_every_scale(scale):
    # squares of these pivots leave the range of float64, their reciprocals do not
    import torch
    lib = _lib.load()
    rng = np.random.default_rng(17)
    n = 192
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3 * np.sqrt(n) * np.eye(n)
    A *= scale
    B = rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))
    At = torch.as_tensor(np.ascontiguousarray(A.T), device="cuda")
    Bt = torch.as_tensor(np.ascontiguousarray(B.T), device="cuda")
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    work = torch.empty(int(lib.bem_zlu_workspace_bytes(n, 1)), dtype=torch.uint8, device="cuda")
    s = _lib.stream_ptr()
    _lib.check(lib.bem_zlu_factor(_vp(At), n, n, n * n, 1, _vp(piv), _vp(info), _vp(work), s))
    _lib.check(lib.bem_zlu_solve(_vp(At), n, n, n * n, 1, _vp(piv), _vp(work), _vp(Bt), n, n * 2, 2, _vp(err), s))
    assert int(info.item()) == 0 and int(err.item()) == 0
    X = Bt.cpu().numpy().T * scale  # X of the unscaled matrix
    want = np.linalg.solve(A / scale, B)
    assert np.abs(X - want).max() < 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("nrhs", [1, 4, 5, 8, 9, 15, 16, 17])
def test_solves_at_the_edges_of_the_column_groups(nrhs):
    # 13 block rows: long chains in both sweeps; the last block row is mostly padding
    import torch
    lib = _lib.load()
    rng = np.random.default_rng(nrhs)
    n, npad, batch = 773, 832, 3
    mats = [rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3 * np.sqrt(n) * np.eye(n)
            for _ in range(batch)]
    B = rng.standard_normal((batch, n, nrhs)) + 1j * rng.standard_normal((batch, n, nrhs))
    A = torch.zeros((batch, npad, npad), dtype=torch.complex128, device="cuda")
    A[:, :n, :n] = torch.as_tensor(np.array([m.T for m in mats]))
    s = _lib.stream_ptr()
    _lib.check(lib.bem_zpad_identity(_vp(A), npad, npad * npad, batch, n, npad, s))
    piv = torch.empty((batch, npad), dtype=torch.int32, device="cuda")
    info = torch.zeros(batch, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    work = torch.empty(int(lib.bem_zlu_workspace_bytes(npad, batch)), dtype=torch.uint8, device="cuda")
    _lib.check(lib.bem_zlu_factor(_vp(A), npad, npad, npad * npad, batch, _vp(piv), _vp(info), _vp(work), s))

    def solve(columns):
        nc = columns.shape[2]
        X = torch.zeros((batch, nc, npad), dtype=torch.complex128, device="cuda")
        X[:, :, :n] = torch.as_tensor(np.ascontiguousarray(columns.transpose(0, 2, 1)))
        _lib.check(lib.bem_zlu_solve(_vp(A), npad, npad, npad * npad, batch, _vp(piv), _vp(work), _vp(X), npad,
                                     npad * nc, nc, _vp(err), s))
        assert int(err.item()) == 0 and float(X[:, :, n:].abs().sum()) == 0.0
        return X[:, :, :n].cpu().numpy().transpose(0, 2, 1)
    X = solve(B)
    assert info.cpu().numpy().tolist() == [0] * batch
    for b in range(batch):
        want = np.linalg.solve(mats[b], B[b])
        # backward error below 1e-12 (see above), condition below 10
        assert np.abs(X[b] - want).max() < 1e-11 * np.abs(want).max()
    one = solve(B[:, :, -1:])
    assert np.abs(X[:, :, -1:] - one).max() < 1e-13 * np.abs(one).max()


@pytest.mark.parametrize("weak", [1.0, 1e-2, 1e-4, 1e-6])
@pytest.mark.parametrize("n", [128, 320])
def test_factors_of_blocks_with_ill_conditioned_triangles(n, weak):
    # a first block close to rank one: its triangles are ill-conditioned.  The entries
    # of L U of an elimination are off by at most n u (|L| |U|) (Higham, Accuracy and
    # Stability of Numerical Algorithms, theorem 9.3), and by sqrt(n) of that in place
    # of n as the roundings' signs are random; products of the panels with the
    # triangles' whole inverses add up to ten times as much.
    import torch
    lib = _lib.load()
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A[:64, :64] = weak * A[:64, :64] + np.outer(rng.standard_normal(64), rng.standard_normal(64))
    At = torch.as_tensor(np.ascontiguousarray(A.T), device="cuda")
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    work = torch.empty(int(lib.bem_zlu_workspace_bytes(n, 1)), dtype=torch.uint8, device="cuda")
    _lib.check(lib.bem_zlu_factor(_vp(At), n, n, n * n, 1, _vp(piv), _vp(info), _vp(work), _lib.stream_ptr()))
    lu, p = At.cpu().numpy().T, piv.cpu().numpy()
    rows = np.concatenate([k + p[k:k + 64] for k in range(0, n, 64)])
    L, U = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    error = np.abs((L.astype(np.clongdouble) @ U - A[rows]).astype(complex))
    ratio = (error / (np.abs(L) @ np.abs(U))).max() / (n * 2.0 ** -53)
    assert ratio <= 1 / np.sqrt(n)


@pytest.mark.parametrize("n", [64, 192, 448])
def test_updates_round_to_a_dominant_matrix_once(n):
    # products far smaller than the diagonal: what is left of the error is the
    # rounding of each update of a diagonal entry, one per eight columns in its own
    # block and one per block before it, half a unit of 2^-53 each
    import torch
    lib = _lib.load()
    rng = np.random.default_rng(n)
    A = 0.02 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n) + np.eye(n) * (0.6 + 0.7j)
    At = torch.as_tensor(np.ascontiguousarray(A.T), device="cuda")
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    work = torch.empty(int(lib.bem_zlu_workspace_bytes(n, 1)), dtype=torch.uint8, device="cuda")
    _lib.check(lib.bem_zlu_factor(_vp(At), n, n, n * n, 1, _vp(piv), _vp(info), _vp(work), _lib.stream_ptr()))
    lu, p = At.cpu().numpy().T, piv.cpu().numpy()
    assert np.array_equal(p, np.tile(np.arange(64), n // 64))
    L, U = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    diagonal = np.diag(L.astype(np.clongdouble) @ U - A)
    error = np.maximum(np.abs(diagonal.real), np.abs(diagonal.imag)).max()
    assert error <= (8 + n // 64) * 2.0 ** -54
