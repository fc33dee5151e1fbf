"""The backward SiLU epilogue where its output does not take 16-byte stores (row strides off 4,
column tiles past the edge) and on ragged rows, against FP64, with nothing written past the end."""
import numpy as np
import pytest

import mlp_oracle as mo
from indicatrix_b200 import surrogate
from test_gpu_surrogate import _dev, _stream, _tol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (130, 27, 64), (33, 42, 40), (129, 257, 70), (257, 36, 96),
                                   (100, 30, 256), (1000, 100, 27)])
def test_backward_silu_scalar_epilogue(m, n, k):
    import torch

    rng = np.random.default_rng(m + n + k)
    dzn = rng.standard_normal((m, k)).astype(np.float32)
    w = (rng.standard_normal((k, n)) / 16.0).astype(np.float32)
    zp = rng.standard_normal((m, n)).astype(np.float32) * 3.0
    a, b, z = _dev(dzn, torch.bfloat16), _dev(w, torch.bfloat16), torch.from_numpy(zp).cuda()
    dz = torch.full((m * n + 8,), 5.0, device="cuda")
    dzb = torch.full((m * n + 8,), 5.0, dtype=torch.bfloat16, device="cuda")
    assert surrogate._lib().ix_mlp_backward_silu(m, n, k, a.data_ptr(), b.data_ptr(), z.data_ptr(), dz.data_ptr(),
                                                 dzb.data_ptr(), _stream()) == 0
    assert bool((dz[m * n:] == 5.0).all()) and bool((dzb[m * n:] == 5.0).all())
    sg = mo.silu_grad(zp.astype(np.float64))
    want = (mo.bf16(dzn) @ mo.bf16(w)) * sg
    ab = np.abs(mo.bf16(dzn)) @ np.abs(mo.bf16(w))
    got = dz[:m * n].reshape(m, n).cpu().numpy()
    # The accumulation's error scaled by |silu'|, and the fast logistic's in silu' itself.
    assert np.all(np.abs(got - want) <= _tol(k) * ab * np.abs(sg) + 2e-6 * ab)
    assert np.array_equal(dzb[:m * n].reshape(m, n).float().cpu().numpy(), mo.bf16(got).astype(np.float32))
    assert surrogate._lib().ix_mlp_status(1) == 0
