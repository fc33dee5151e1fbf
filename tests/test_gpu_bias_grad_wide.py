"""The bias gradient's two launch shapes: a wide matrix's sums are the bits of its columns summed
32 at a time (clusters of CTAs), and few rows sum as f64 does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sums(dz):
    import torch

    from indicatrix_b200.surrogate import _lib

    m, n = dz.shape
    db = torch.full((n + 1,), 7.0, device="cuda")
    assert _lib().ix_mlp_bias_grad(m, n, dz.data_ptr(), db.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert float(db[n]) == 7.0
    return db[:n]


@pytest.mark.parametrize("m", [129, 131, 160, 255, 256, 257, 511, 1000, 2001])
@pytest.mark.parametrize("n", [2400, 16421])
def test_wide_sums_equal_the_clusters(m, n):
    import torch

    g = torch.Generator(device="cuda").manual_seed(m + n)
    dz = torch.randn(m, n, device="cuda", generator=g)
    got = _sums(dz)
    for c in (0, 32, 1024, n // 2, n - 33, n - 5):
        assert torch.equal(got[c:c + 32], _sums(dz[:, c:c + 32].contiguous()))


@pytest.mark.parametrize("m", [1, 3, 4, 5, 31, 32, 33, 64, 65, 96, 97, 127, 128])
@pytest.mark.parametrize("n", [1, 31, 33, 256, 5000])
def test_few_rows_match_fp64(m, n):
    import torch

    dz = torch.randn(m, n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(m * 7 + n))
    # One term a partial sum, a 5-level tree and at most 4 more: that many roundings.
    tol = 10 * np.finfo(np.float32).eps * dz.double().abs().sum(0)
    assert bool(((_sums(dz).double() - dz.double().sum(0)).abs() <= tol).all())
