"""Calls of the bias gradient that are refused, and what a refused call leaves behind: nothing
that a later call could report as its own error."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1 << 31])
def test_bias_grad_refuses_column_counts_without_a_launch(n):
    import torch

    from indicatrix_b200.surrogate import _lib

    lib, s = _lib(), torch.cuda.current_stream().cuda_stream
    dz, db = torch.ones(4, device="cuda"), torch.full((4,), 7.0, device="cuda")
    xb = torch.empty(4, dtype=torch.bfloat16, device="cuda")
    assert lib.ix_mlp_bias_grad(1, n, dz.data_ptr(), db.data_ptr(), s) == 1
    assert lib.ix_mlp_to_bf16(4, dz.data_ptr(), xb.data_ptr(), s) == 0
    assert bool((db == 7.0).all()) and bool((xb == 1.0).all())
