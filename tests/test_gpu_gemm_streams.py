"""Weight gradients (products split over K, whose partial sums need memory of their own) from
several streams and threads at once, and under graph capture: the bits of the calls made one
after another."""
import threading

import numpy as np
import pytest

from indicatrix_b200 import surrogate

pytestmark = pytest.mark.gpu


def _case(seed, rows):
    rng = np.random.default_rng(seed)
    net = surrogate.SurrogateMLP(seed=seed)
    x = surrogate.normalize(surrogate.sample_designs(rows, seed))
    return net, net.to_device_bf16(x), net.torch.from_numpy(rng.standard_normal((rows, 27)).astype(np.float32)).cuda()


def _flat(grads):
    return [g for pair in grads for g in pair]


@pytest.mark.parametrize("rows", [(4096, 4096), (4096, 1500), (513, 3000)])
def test_gradients_of_two_networks_on_two_streams(rows):
    import torch

    cases = [_case(i + 1, r) for i, r in enumerate(rows)]
    want = [_flat(net._gradients_device(xb, tt)[1]) for net, xb, tt in cases]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in cases]
    got = [[], []]
    for _ in range(12):
        for i, (net, xb, tt) in enumerate(cases):
            with torch.cuda.stream(streams[i]):
                got[i].append(_flat(net._gradients_device(xb, tt)[1]))
    torch.cuda.synchronize()
    for w, runs in zip(want, got):
        for run in runs:
            assert all(torch.equal(a, b) for a, b in zip(w, run))


def test_gradients_from_two_threads():
    import torch

    cases = [_case(3, 4096), _case(4, 700)]
    want = [_flat(net._gradients_device(xb, tt)[1]) for net, xb, tt in cases]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        net, xb, tt = cases[i]
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(20):
                run = _flat(net._gradients_device(xb, tt)[1])
                s.synchronize()
                if not all(torch.equal(a, b) for a, b in zip(want[i], run)):
                    bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_a_captured_weight_gradient_replays_on_new_operands():
    import torch

    lib = surrogate._lib()
    n, k, m = 256, 256, 4096
    g = torch.Generator(device="cuda").manual_seed(9)
    dz = torch.randn(m, n, device="cuda", generator=g).bfloat16()
    h = torch.randn(m, k, device="cuda", generator=g).bfloat16()
    dw, eager = torch.zeros(n, k, device="cuda"), torch.empty(n, k, device="cuda")

    def call(out):
        assert lib.ix_mlp_gemm_bf16(1, 0, n, k, m, dz.data_ptr(), n, h.data_ptr(), k, out.data_ptr(), k,
                                    torch.cuda.current_stream().cuda_stream) == 0

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(dw)
    for seed in (1, 2, 3):
        dz.copy_(torch.randn(m, n, device="cuda", generator=g.manual_seed(seed)))
        graph.replay()
        call(eager)
        assert torch.equal(dw, eager)
    assert lib.ix_mlp_status(1) == 0


@pytest.mark.parametrize("m,n,k", [(256, 256, 4096), (27, 256, 4096), (128, 32, 8192), (128, 128, 16384),
                                   (9344, 32, 1024), (256, 12, 513), (64, 64, 64)])
def test_a_workspace_gives_the_same_bits(m, n, k):
    """The caller's workspace: the pool's sums, and nothing past IX_MLP_GEMM_WORKSPACE floats."""
    import torch

    lib, s = surrogate._lib(), torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(k, m, device="cuda", generator=g).bfloat16()
    b = torch.randn(k, n, device="cuda", generator=g).bfloat16()
    want, got = torch.empty(m, n, device="cuda"), torch.empty(m, n, device="cuda")
    ws = torch.full((surrogate.GEMM_WORKSPACE + 4096,), 7.0, device="cuda")
    assert lib.ix_mlp_gemm_bf16(1, 0, m, n, k, a.data_ptr(), m, b.data_ptr(), n, want.data_ptr(), n, s) == 0
    assert lib.ix_mlp_gemm_bf16_ws(1, 0, m, n, k, a.data_ptr(), m, b.data_ptr(), n, got.data_ptr(), n, ws.data_ptr(),
                                   s) == 0
    assert torch.equal(got, want) and bool((ws[surrogate.GEMM_WORKSPACE:] == 7.0).all())
