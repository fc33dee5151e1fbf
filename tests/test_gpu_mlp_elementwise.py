"""Adam over many tensors in one launch and the outputs' way out of their standardisation:
tensor counts around a launch's 16, sizes around a block, against f64 and numpy."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stream():
    import torch

    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("n", [1, 2, 16, 17])
def test_adam_multi_matches_fp64(n):
    import torch

    from indicatrix_b200.surrogate import AdamTensor, _lib

    g = torch.Generator(device="cuda").manual_seed(n)
    lr, b1, b2, eps, step = 1e-3, 0.9, 0.999, 1e-8, 3
    sizes = [(1, 255, 256, 257, 70001)[i % 5] for i in range(n)]
    state = [[torch.randn(k + 1, device="cuda", generator=g) for _ in range(4)] for k in sizes]  # w, g, m, v
    for s in state:
        s[3].abs_()
    before = [[a.double() for a in s] for s in state]
    wb = [torch.zeros(k + 1, dtype=torch.bfloat16, device="cuda") if i % 2 == 0 else None for i, k in enumerate(sizes)]
    rows = (AdamTensor * n)()
    for i, (k, (w, gr, m, v)) in enumerate(zip(sizes, state)):
        rows[i] = (k, w.data_ptr(), wb[i].data_ptr() if wb[i] is not None else None, gr.data_ptr(), m.data_ptr(),
                   v.data_ptr())
    assert _lib().ix_mlp_adam_multi(n, rows, lr, b1, b2, eps, step, _stream()) == 0
    for k, s, old, h in zip(sizes, state, before, wb):
        w, gr, m, v = (a[:k] for a in old)
        m2, v2 = b1 * m + (1 - b1) * gr, b2 * v + (1 - b2) * gr * gr
        u = lr * (m2 / (1 - b1 ** step)) / ((v2 / (1 - b2 ** step)).sqrt() + eps)
        # The 32-bit betas put 1 - beta2 off by 2^-24 / 1e-3 of itself at most, and with
        # it the bias correction; the rest are a dozen roundings.
        rel = 2.0 ** -24 / (1 - b2) * 2 + 12 * 2.0 ** -24
        scale = b1 * m.abs() + (1 - b1) * gr.abs()
        assert bool(((s[2][:k].double() - m2).abs() <= rel * scale).all())
        assert bool(((s[3][:k].double() - v2).abs() <= rel * v2).all())
        ub = lr * scale / (1 - b1 ** step) / ((v2 / (1 - b2 ** step)).sqrt() + eps)
        assert bool(((s[0][:k].double() - (w - u)).abs() <= 2 * rel * ub + 2.0 ** -23 * w.abs()).all())
        assert all(float(a[k]) == float(o[k]) for a, o in zip(s, old))  # nothing past the end
        if h is not None:
            assert bool((h[:k] == s[0][:k].bfloat16()).all()) and float(h[k]) == 0.0


def test_adam_multi_refuses_null_tensors():
    from indicatrix_b200.surrogate import AdamTensor, _lib

    rows = (AdamTensor * 1)()
    rows[0].count = 4
    assert _lib().ix_mlp_adam_multi(1, rows, 1e-3, 0.9, 0.999, 1e-8, 1, _stream()) == 1
    assert _lib().ix_mlp_adam_multi(1, C.cast(None, C.POINTER(AdamTensor)), 1e-3, 0.9, 0.999, 1e-8, 1, _stream()) == 1


@pytest.mark.parametrize("m", [1, 9, 255, 256, 4097])
def test_members_metrics_equal_numpy(m):
    from indicatrix_b200.surrogate import SurrogateEnsemble, normalize, sample_designs

    ens = SurrogateEnsemble(3, seed=5)
    rng = np.random.default_rng(m)
    for net in ens.nets:
        net.t_std = rng.uniform(0.1, 9.0, 27).astype(np.float32)
        net.t_mean = rng.standard_normal(27).astype(np.float32)
    x = normalize(sample_designs(m, m))
    xb = ens.nets[0].to_device_bf16(x)
    want = np.stack([net.forward_device(xb)[0].cpu().numpy() * net.t_std + net.t_mean for net in ens.nets])
    got = ens.predict_members(x)
    assert got.dtype == want.dtype and np.array_equal(got, want)
    assert np.array_equal(ens.nets[1].predict(x), want[1])
    ens.nets[2].t_mean = 0.5  # a plain number still broadcasts
    assert np.array_equal(ens.predict_members(x)[2], ens.nets[2].forward_device(xb)[0].cpu().numpy() *
                          ens.nets[2].t_std + 0.5)


@pytest.mark.parametrize("m,n", [(1, 1), (255, 1), (256, 1), (257, 1), (4096, 27), (30000, 27)])
def test_mse_loss_and_gradient_match_fp64(m, n):
    import torch

    from indicatrix_b200.surrogate import _lib

    g = torch.Generator(device="cuda").manual_seed(m + n)
    y, t = (torch.randn(m, n, device="cuda", generator=g) for _ in range(2))
    dy, dyb = torch.empty_like(y), torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    loss = torch.full((1,), 2.0, device="cuda")
    assert _lib().ix_mlp_mse_grad(m, n, y.data_ptr(), t.data_ptr(), dy.data_ptr(), dyb.data_ptr(), loss.data_ptr(),
                                  _stream()) == 0
    d = y.double() - t.double()
    eps = float(np.finfo(np.float32).eps)
    want = 2.0 + float((d * d).mean())
    # At most min(blocks, 2368) atomics, each half an ulp of a sum below 8, and 8 roundings a term.
    blocks = min((m * n + 255) // 256, 148 * 16)
    assert abs(float(loss) - want) <= (4 * blocks + 8 * (1 + m * n // (256 * blocks))) * eps + 8 * eps * want
    assert bool(((dy.double() - 2 * d / (m * n)).abs() <= 4 * eps * (y.abs() + t.abs()).double() * 2 / (m * n)).all())
    assert bool((dyb == dy.bfloat16()).all())
