"""Products and solves of device matrices held in any form against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forms(torch, A):
    a = torch.as_tensor(A, device="cuda")
    column_major = a.T.contiguous().T
    return {"column-major": (column_major, A), "row-major": (a.contiguous(), A),
            "conjugated": (column_major.conj(), A.conj()), "conjugate transpose": (a.contiguous().mH, A.conj().T),
            "negated": (torch._neg_view(column_major), -A),
            "complex64": (column_major.to(torch.complex64), A.astype(np.complex64))}


@pytest.mark.parametrize("form", ["column-major", "row-major", "conjugated", "conjugate transpose", "negated",
                                  "complex64"])
@pytest.mark.parametrize("n,m", [(70, 70), (1, 9), (9, 1), (1, 1), (130, 33)])
def test_products_and_solves(n, m, form):
    import torch
    from capytaine_b200.engine import B200Engine, DeviceMatrix
    rng = np.random.default_rng(n + m)
    A = rng.standard_normal((n, m)) + 1j * rng.standard_normal((n, m))
    if n == m:
        A += 4 * n * np.eye(n)
    t, ref = _forms(torch, A)[form]
    M = DeviceMatrix(t, B200Engine())
    # float64 sums of m (products) or the refined residual times the condition number, a
    # few here; complex64 results are rounded to 2^-24 on return
    tol = 2e-7 if form == "complex64" else 1e-12
    ref = ref.astype(np.complex128)
    for nrhs in (0, 1, 3):
        x = rng.standard_normal((ref.shape[1], nrhs)) + 1j * rng.standard_normal((ref.shape[1], nrhs))
        want = ref @ x
        got = M @ x
        assert got.shape == want.shape and np.all(np.abs(got - want) <= tol * (np.abs(ref) @ np.abs(x)))
        if n == m:
            solutions = [M.solve(want)]
            if nrhs and form != "complex64":
                solutions.append(M.gmres(want, atol=0.0, rtol=1e-13))
            for got in solutions:
                assert got.shape == x.shape
                assert np.all(np.abs(got - x) <= 10 * tol * max(1.0, np.abs(x).max(initial=0)))


def test_solves_keep_to_the_matrix_that_was_factored():
    import torch
    from capytaine_b200.engine import B200Engine, DeviceMatrix
    rng = np.random.default_rng(5)
    n = 100
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4 * n * np.eye(n)
    b = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    M = DeviceMatrix(torch.as_tensor(A.T.copy(), device="cuda").T, B200Engine())
    first = M.solve(b)
    M.t.mul_(3.0)
    assert np.array_equal(M.solve(b), first)
    assert np.allclose(M @ first, 3 * b, rtol=0, atol=1e-11)  # products are of the matrix as it is
