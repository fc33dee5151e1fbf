"""The bias gradient's column sums: row counts around a CTA pass and a cluster pass, ragged
columns, against f64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 31, 32, 33, 64, 65, 255, 256, 257, 4096, 5001])
@pytest.mark.parametrize("n", [1, 27, 32, 33, 256])
def test_bias_grad_matches_fp64(m, n):
    import torch

    from indicatrix_b200.surrogate import _lib

    g = torch.Generator(device="cuda").manual_seed(m * 1000 + n)
    dz = torch.randn(m, n, device="cuda", generator=g)
    db = torch.full((n + 1,), 7.0, device="cuda")
    assert _lib().ix_mlp_bias_grad(m, n, dz.data_ptr(), db.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    want = dz.double().sum(0)
    # At most m / 256 + 1 serial terms, a 5-level tree and 8 more: that many roundings of at
    # most the sum of magnitudes.
    tol = (m / 256 + 14) * np.finfo(np.float32).eps * dz.double().abs().sum(0)
    assert bool(((db[:n].double() - want).abs() <= tol).all()) and float(db[n]) == 7.0
