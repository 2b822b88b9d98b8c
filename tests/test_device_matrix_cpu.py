"""The column-major copy or view that the kernels read of a device matrix holds
the values of the tensor, whatever torch defers (conjugation, sign)."""
import pytest
import torch

from capytaine_b200.engine import _column_major

SHAPES = [(5, 5), (1, 4), (4, 1), (1, 1), (3, 0)]
FORMS = {
    "column-major": lambda a: a.T.contiguous().T,
    "row-major": lambda a: a.contiguous(),
    "conjugated": lambda a: a.T.contiguous().T.conj(),
    "conjugate transpose": lambda a: a.mH.contiguous().mH,
    "negated": lambda a: torch._neg_view(a.T.contiguous().T),
    "strided": lambda a: torch.stack([a, 2 * a], dim=-1)[..., 0],
    "broadcast": lambda a: a[:, :1].expand(a.shape),
}


@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("shape", SHAPES)
def test_column_major_holds_the_values(shape, form, dtype):
    a = torch.randn(shape, dtype=dtype, generator=torch.Generator().manual_seed(3))
    t = FORMS[form](a)
    want = t.resolve_conj().resolve_neg().to(torch.complex128).T.contiguous()
    got = _column_major(t)
    assert got.dtype == torch.complex128 and got.shape == want.shape and not got.is_conj() and not got.is_neg()
    # the memory itself, as a kernel sees it
    assert got.numel() == 0 or got.stride(1) == 1 or got.shape[1] == 1
    flat = torch.as_strided(torch.view_as_real(got.detach()), (got.numel(), 2), (2, 1))
    assert torch.equal(flat.reshape(*want.shape, 2), torch.view_as_real(want))


def test_column_major_of_the_engine_s_matrices_is_a_view():
    t = torch.randn((6, 4), dtype=torch.complex128).T.contiguous().T
    assert _column_major(t).data_ptr() == t.data_ptr()
