"""Device entries of one backend called on several streams with nothing waiting between: the
buffers they share are handed on in order, so every call gives what it gives alone."""
import ctypes as C

import numpy as np
import pytest

from indicatrix_b200 import display, materials, workloads
from indicatrix_b200.backend import BatchPlan, FrameScene, camera_new

pytestmark = pytest.mark.gpu


def _view(yaw, w, h):
    base = workloads.round_brilliant_frame(8, 8)
    return FrameScene(camera_new(yaw, 0.45, 2.4, 42.0), w, h, base.planes,
                      materials.isotropic(materials.cauchy(1.76, 0.0, 0.0)), 32, base.environment)


@pytest.mark.parametrize("w,h", [(96, 64), (161, 91), (640, 360)])
@pytest.mark.parametrize("same_view", [True, False])
def test_displayed_frames_on_two_streams(backend, w, h, same_view):
    import torch

    g = torch.Generator(device="cuda").manual_seed(w)
    frames = [_view(0.6, w, h), _view(0.6 if same_view else 1.9, w, h)]
    scenes = [f.to_abi() for f in frames]
    sums = [torch.rand(h, w, 3, device="cuda", generator=g) * 16.0 for _ in frames]

    def show(i, out, stream):
        assert display.display_frame_device(backend, scenes[i], 16, sums[i].data_ptr(), out.data_ptr(), True,
                                            stream_ptr=stream.cuda_stream if stream else None)

    def buffer():
        return torch.zeros(h, w, 4, dtype=torch.uint8, device="cuda")

    want = [buffer(), buffer()]
    for i in range(2):
        torch.cuda.synchronize()
        show(i, want[i], None)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [[buffer() for _ in range(16)] for _ in range(2)]
    torch.cuda.synchronize()
    for k in range(16):
        for i in range(2):
            show(i, outs[i][k], streams[i])
    # The host form on the backend's own stream, behind the last of them.
    host = display.display_frame(backend, frames[0], 16, sums[0].cpu().numpy(), True)
    torch.cuda.synchronize()
    for i in range(2):
        assert all(torch.equal(want[i], o) for o in outs[i])
    assert np.array_equal(np.asarray(host).reshape(h, w, 4), want[0].cpu().numpy())


def test_more_streams_than_colour_buffers(backend):
    import torch

    w, h = 200, 120
    g = torch.Generator(device="cuda").manual_seed(3)
    views = [_view(0.6, w, h).to_abi(), _view(2.2, w, h).to_abi()]
    sums = [torch.rand(h, w, 3, device="cuda", generator=g) * 16.0 for _ in range(7)]

    def show(i, view, out, stream):
        assert display.display_frame_device(backend, views[view], 16, sums[i].data_ptr(), out.data_ptr(), False,
                                            stream_ptr=stream.cuda_stream if stream else None)

    want = torch.zeros(2, 7, h, w, 4, dtype=torch.uint8, device="cuda")
    for view in range(2):
        for i in range(7):
            torch.cuda.synchronize()
            show(i, view, want[view, i], None)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(6)] + [None]
    got = torch.zeros(12, 7, h, w, 4, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for k in range(12):  # the view changes while frames of the other are in flight
        for i in range(7):
            show(i, k // 3 % 2, got[k, i], streams[(i + k) % 7])
    torch.cuda.synchronize()
    for k in range(12):
        assert torch.equal(got[k], want[k // 3 % 2])


def test_traced_frames_on_two_streams(backend):
    import torch

    frames = [workloads.round_brilliant_frame(72, 50),
              workloads.tilted_scene(workloads.random_stones(2, seed=5)[1], 20.0, 64, 48)]
    scenes, keep = [], []
    for fs in frames:
        sc = fs.to_abi()
        planes = torch.from_numpy(np.ascontiguousarray(fs.planes, np.float32)).cuda()
        sc.planes = C.cast(C.c_void_p(planes.data_ptr()), C.POINTER(C.c_float))
        scenes.append(sc)
        keep.append(planes)
    spp = [24, 9]

    def trace(i, out, stream):
        assert backend.accumulate_device(scenes[i], 5, spp[i], out.data_ptr(), False,
                                         stream_ptr=stream.cuda_stream if stream else None) == 0

    def buffer(i):
        return torch.zeros(frames[i].height, frames[i].width, 3, dtype=torch.float64, device="cuda")

    want = [buffer(0), buffer(1)]
    for i in range(2):
        torch.cuda.synchronize()
        trace(i, want[i], None)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [[buffer(i) for _ in range(12)] for i in range(2)]
    torch.cuda.synchronize()
    for k in range(12):
        for i in range(2):
            trace(i, outs[i][k], streams[i])
    host = np.zeros((frames[0].height, frames[0].width, 3))
    assert backend.try_accumulate(frames[0], 5, spp[0], host)
    torch.cuda.synchronize()
    for i in range(2):
        assert all(torch.equal(want[i], o) for o in outs[i])
    assert np.array_equal(host, want[0].cpu().numpy())


def test_a_plan_runs_on_any_stream(backend):
    import torch

    jobs = [(workloads.tilted_scene(s, t, 40, 32), 3, 32) for s in workloads.random_stones(4, seed=2) for t in (0.0, 20.0)]
    plan = BatchPlan(backend, jobs)
    plan.run()
    want = plan.download()
    streams = [torch.cuda.Stream(), torch.cuda.Stream(), None]
    for k in range(9):
        s = streams[k % 3]
        plan.run(s.cuda_stream if s else None)
        if k % 2:
            plan.run(streams[(k + 1) % 2].cuda_stream)
        assert np.array_equal(plan.download(), want)
    plan.close()


def test_a_captured_frame_replays(backend):
    import torch

    w, h = 160, 90
    fs = _view(0.6, w, h)
    sc = fs.to_abi()
    sums = torch.rand(h, w, 3, device="cuda") * 16.0
    out, want = (torch.zeros(h, w, 4, dtype=torch.uint8, device="cuda") for _ in range(2))
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    # In flight on one stream while another captures: the capture holds the call alone.
    assert display.display_frame_device(backend, sc, 16, sums.data_ptr(), want.data_ptr(), True,
                                        stream_ptr=side.cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert display.display_frame_device(backend, sc, 16, sums.data_ptr(), out.data_ptr(), True,
                                            stream_ptr=torch.cuda.current_stream().cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert display.display_frame_device(backend, sc, 16, sums.data_ptr(), want.data_ptr(), True)
    torch.cuda.synchronize()
    assert torch.equal(out, want)
