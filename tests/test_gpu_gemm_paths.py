"""The GEMM's staging and epilogue forms on the same numbers: transposed views that can be
turned in registers and those that cannot (ragged edges, unaligned rows), outputs that take
16-byte stores and those that do not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(128, 32, 64), (256, 256, 512), (256, 256, 65), (136, 40, 128), (130, 33, 64),
                                   (27, 256, 4096), (1, 1, 1)])
@pytest.mark.parametrize("ta,tb", [(1, 0), (1, 1), (0, 0)])
@pytest.mark.parametrize("pad", [0, 1, 8])
def test_transposed_operands_match_fp64(m, n, k, ta, tb, pad):
    import torch

    from indicatrix_b200.surrogate import _lib

    g = torch.Generator(device="cuda").manual_seed(m + 7 * n + 13 * k)
    # Operands inside wider rows: `pad` extra columns shift every row's alignment.
    ra, ca = (k, m) if ta else (m, k)
    rb, cb = (n, k) if tb else (k, n)
    a = torch.randn(ra, ca + pad, device="cuda", generator=g).bfloat16()
    b = torch.randn(rb, cb + pad, device="cuda", generator=g).bfloat16()
    c = torch.full((m, n + pad), 5.0, device="cuda")
    assert _lib().ix_mlp_gemm_bf16(ta, tb, m, n, k, a.data_ptr(), ca + pad, b.data_ptr(), cb + pad, c.data_ptr(),
                                   n + pad, torch.cuda.current_stream().cuda_stream) == 0
    A, B = a[:, :ca].double(), b[:, :cb].double()
    A, B = (A.T if ta else A), (B.T if tb else B)
    # FP32 accumulation of exact products: k roundings of at most the sum of magnitudes.
    tol = (k + 8) * np.finfo(np.float32).eps * (A.abs() @ B.abs()) + 1e-30
    assert bool(((c[:, :n].double() - A @ B).abs() <= tol).all())
    assert bool((c[:, n:] == 5.0).all())
