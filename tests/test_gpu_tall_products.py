"""The tall product at the edges of its rows, depth chunks and column tiles, and in
a workspace sized for more matrices than the call has.  Bar: 1e-13 of the largest
entry (sums of up to 2500 products of order-one terms in float64)."""
import ctypes

import numpy as np
import pytest

from capytaine_b200 import _lib

pytestmark = pytest.mark.gpu


def _vp(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("M,K,nrhs,batch,sized", [(1, 1, 1, 1, 1), (127, 31, 8, 1, 3), (128, 64, 9, 2, 2),
                                                  (129, 65, 16, 3, 40), (735, 735, 1, 1, 8), (64, 2500, 7, 5, 5),
                                                  (1300, 33, 2, 60, 60)])
def test_tall_product(M, K, nrhs, batch, sized):
    import torch
    rng = np.random.default_rng(M + K)
    lib = _lib.load()
    a, x, y = (rng.standard_normal(s) + 1j * rng.standard_normal(s)
               for s in ((batch, K, M), (batch, nrhs, K), (batch, nrhs, M)))  # column-major matrices
    A, X, Y = (torch.as_tensor(v, device="cuda") for v in (a, x, y))
    nbytes = int(lib.bem_zgemm_ts_workspace_bytes(M, K, nrhs, sized))
    work = torch.full((nbytes + 64,), 7, dtype=torch.uint8, device="cuda")
    _lib.check(lib.bem_zgemm_ts(M, K, nrhs, -1.0, 0.5, _vp(A), M, M * K, _vp(X), K, K * nrhs, 1.0, 0.0, _vp(Y), M,
                                M * nrhs, batch, _vp(work), _lib.stream_ptr()))
    ref = y + (-1 + 0.5j) * np.einsum("bkm,bck->bcm", a, x)
    assert np.abs(Y.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()
    assert (work[nbytes:] == 7).all()  # nothing past the workspace
