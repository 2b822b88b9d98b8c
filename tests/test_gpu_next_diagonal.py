"""The mixed LU's two ways to the next diagonal block (its own float32 kernel, or
a tensor-core tile behind the panel product): one block and two, odd and even
numbers of blocks, batches on both sides of the rule and one that changes over
within a factorisation, and matrices of different active sizes.  The factors
solve to a residual of 5e-4: operands of 11 bits (2^-11) in updates that stay
below the matrix itself (dominant diagonal)."""
import ctypes

import pytest

from capytaine_b200 import _lib

pytestmark = pytest.mark.gpu


def _vp(t):
    return ctypes.c_void_p(t.data_ptr() if hasattr(t, "data_ptr") else int(t))


def _factor_and_check(n, batch, active=None):
    import torch
    lib = _lib.load()
    gen = torch.Generator(device="cuda").manual_seed(7)
    K = torch.randn(batch, n, n, dtype=torch.complex128, device="cuda", generator=gen)
    K.diagonal(dim1=1, dim2=2).add_(3 * n ** 0.5)
    for b, a in enumerate(active or []):  # identity beyond the active size
        K[b, a:, :] = 0
        K[b, :, a:] = 0
        K[b].diagonal()[a:] = 1
    work = torch.empty(int(lib.bem_clu_workspace_bytes(n, batch)) + 1024, dtype=torch.uint8, device="cuda")
    wptr = (work.data_ptr() + 1023) // 1024 * 1024
    piv = torch.empty((batch, n), dtype=torch.int32, device="cuda")
    info = torch.zeros(batch, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    s = _lib.stream_ptr()
    if active is None:
        _lib.check(lib.bem_clu_factor(_vp(K), n, n * n, n, n, batch, _vp(piv), _vp(info), _vp(wptr), _vp(err), s))
    else:
        act = (ctypes.c_int32 * batch)(*active)
        _lib.check(lib.bem_clu_factor_grouped(_vp(K), n, n * n, n, n, batch, act, _vp(piv), _vp(info), _vp(wptr),
                                              _vp(err), s))
    B = torch.randn(batch, 3, n, dtype=torch.complex128, device="cuda", generator=gen)
    X = B.clone()
    _lib.check(lib.bem_clu_solve(_vp(wptr), n, batch, _vp(piv), _vp(X), n, 3 * n, 3, _vp(err), s))
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and info.abs().max().item() == 0
    R = torch.bmm(X, K) - B  # K is column-major: row vectors times its transpose
    rel = R.norm(dim=2) / B.norm(dim=2)
    assert rel.max().item() < 5e-4


@pytest.mark.parametrize("n,batch", [(128, 2), (256, 3), (384, 1), (640, 24), (640, 25), (1408, 24), (1920, 1)])
def test_factors_solve(n, batch):
    _factor_and_check(n, batch)


@pytest.mark.parametrize("batch", [4, 26])
def test_active_sizes(batch):
    _factor_and_check(768, batch, [128 * (1 + i % 6) for i in range(batch)])
