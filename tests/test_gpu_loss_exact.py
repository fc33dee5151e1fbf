"""The loss on differences whose every partial sum is exact in f32, so that a missing block, warp
or element shows whatever the order: sizes of one block, of two, and past the grid's 2368."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 1), (256, 1), (512, 1), (32, 32), (1 << 15, 32), (1 << 21, 1)])
def test_loss_and_gradient_of_small_integers_are_exact(m, n):
    import torch

    from indicatrix_b200.surrogate import _lib

    g = torch.Generator(device="cuda").manual_seed(m + n)
    # d in -2 .. 2 and m n = 2^p <= 2^21: every term is a multiple of 2^-21, every sum below 8.
    y = torch.randint(-1, 2, (m, n), device="cuda", generator=g).float()
    t = torch.randint(-1, 2, (m, n), device="cuda", generator=g).float()
    y[-1, -1], t[-1, -1] = 1.0, -1.0  # the last element counts
    dy, dyb = torch.empty_like(y), torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    loss = torch.full((1,), 2.0, device="cuda")
    assert _lib().ix_mlp_mse_grad(m, n, y.data_ptr(), t.data_ptr(), dy.data_ptr(), dyb.data_ptr(), loss.data_ptr(),
                                  torch.cuda.current_stream().cuda_stream) == 0
    d = y.double() - t.double()
    assert float(loss) == 2.0 + float((d * d).sum()) / (m * n)
    assert torch.equal(dy.double(), 2.0 * d / (m * n)) and torch.equal(dyb.double(), dy.double())
