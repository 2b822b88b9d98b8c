"""The float32 block substitutions where their launch changes shape: right-hand
sides at the ends of the 8- and 16-column kernels and over several launches,
one block (no dependency) to many, and batches on both sides of the rule that
puts three CTAs on an SM.  Against numpy at the bar of the float32 factors with
TF32 updates (5e-3, as test_float32_lu_solve); the same columns solved one at a
time must agree with the block of columns to float32 rounding (1e-5)."""
import numpy as np
import pytest

from capytaine_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch,nrhs", [(100, 1, 8), (256, 3, 9), (300, 1, 16), (384, 2, 17), (130, 40, 5),
                                          (900, 1, 33)])
def test_block_substitutions(n, batch, nrhs):
    import torch
    from test_gpu_mixed import _setup, _vp
    lib, npad, mats, rhs, K, B, work, wptr, piv, info, err = _setup(n, batch, nrhs, n + nrhs)
    one = B[:, nrhs - 1:].clone().contiguous()
    s = _lib.stream_ptr()
    _lib.check(lib.bem_clu_solve(_vp(wptr), npad, batch, _vp(piv), _vp(B), npad, npad * nrhs, nrhs, _vp(err), s))
    _lib.check(lib.bem_clu_solve(_vp(wptr), npad, batch, _vp(piv), _vp(one), npad, npad, 1, _vp(err), s))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    for b in range(batch):
        x = B[b, :, :n].T.cpu().numpy()
        ref = np.linalg.solve(mats[b], rhs[b])
        assert np.abs(x - ref).max() / np.abs(ref).max() < 5e-3
        last = one[b, 0, :n].cpu().numpy()
        assert np.abs(x[:, -1] - last).max() / np.abs(last).max() < 1e-5
        assert B[b, :, n:].abs().max().item() == 0.0 if npad > n else True
