"""The work that a program has this library do, as measurable cases.

A case is a dict of plain values; ``kind`` names the entry point it goes through:

* ``frame``     ``GpuBackend.try_accumulate``: samples of one frame added into the caller's
                sums, a progressive renderer's step (the next sample range each pass);
* ``batch``     ``BatchPlan.run`` + ``download``: random stones x tilts in one launch;
* ``designs``   ``surrogate.evaluate_designs``: traced metrics of a set of cut designs;
* ``metrics``   the analytic optical metrics: one pose, many poses, or the axis sweeps;
* ``train``     ``SurrogateMLP.train_step``: forward, backward and Adam on one batch;
* ``predict``   ``SurrogateEnsemble.predict_members``: a population scored by 4 networks;
* ``display``   ``display.display_frame_device``: average, denoise and tone-map a frame.

Sizes are those of the library's own benchmark, tests and defaults, or smaller and ragged
ones of the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from indicatrix_b200 import backend as ixb
from indicatrix_b200 import abi, display, geometry, materials, surrogate, workloads

# Counted floating-point operations per traced path of each stone (add, sub, mul, div and
# sqrt 1, FMA 2): the oracle's operation-counting build on the benchmark's scenes.
FLOPS_PER_PATH = {"round": 1.05e4, "random": 6.3e3, "uniaxial": 4.0e4, "sun": 8.5e3}
MEAN_SPP = 120  # of the random stones: drawn from {32, 64, 128, 256}
LR = 1e-3


def listed():
    return [
        # An interactive editor's first image after each change: latency counts.
        {"name": "preview_160x120_1spp", "kind": "frame", "stone": "round", "width": 160, "height": 120, "spp": 1,
         "dtype": "float32"},
        # The benchmark's frame: a round brilliant face up.
        {"name": "frame_256_64spp", "kind": "frame", "stone": "round", "width": 256, "height": 256, "spp": 64,
         "dtype": "float32"},
        # One progressive step of a full-screen render of a coloured stone.
        {"name": "frame_1080p_8spp", "kind": "frame", "stone": "random", "width": 1920, "height": 1080, "spp": 8,
         "dtype": "float64"},
        # A birefringent, pleochroic crystal: the step cut of the stress workload.
        {"name": "uniaxial_251x193_64spp", "kind": "frame", "stone": "uniaxial", "width": 251, "height": 193,
         "spp": 64, "dtype": "float64"},
        # A carved, partly frosted stone under the sun: the extended transport.
        {"name": "sun_192_48spp", "kind": "frame", "stone": "sun", "width": 192, "height": 192, "spp": 48,
         "dtype": "float32"},
        # A catalogue page: stones of every size and material, each at the 9 tilts.
        {"name": "batch_16x9_64", "kind": "batch", "stones": 16, "tilts": 9, "width": 64, "height": 64},
        # One generation's finalists of a design search, traced.
        {"name": "designs_64", "kind": "designs", "designs": 64, "size": 32, "spp": 32},
        # The metric readout beside the editor's view.
        {"name": "metrics_pose", "kind": "metrics", "mode": "pose", "poses": 1},
        # The tilt-performance chart: 181 tilts on each of four axes.
        {"name": "metrics_axes", "kind": "metrics", "mode": "axes", "poses": 724},
        # One optimiser step of the surrogate at its training batch.
        {"name": "train_4096", "kind": "train", "batch": 4096},
        # One generation's population scored by the ensemble.
        {"name": "predict_4096", "kind": "predict", "batch": 4096},
        # A displayed frame of a still view (its guides are kept by the backend).
        {"name": "display_1080p", "kind": "display", "width": 1920, "height": 1080, "spp": 16, "signature": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "batch", "designs", "metrics", "train", "predict", "display"])
    if kind == "frame":
        stone = rng.choice(["round", "random", "uniaxial", "sun"])
        most = 1 << (21 if stone in ("uniaxial", "sun") else 24)  # paths
        w, h = _log_int(rng, 48, 1600), _log_int(rng, 32, 1200)
        spp = min(_log_int(rng, 1, 96), max(1, most // (w * h)))
        return {"kind": kind, "stone": stone, "width": w, "height": h, "spp": spp,
                "dtype": rng.choice(["float32", "float64"])}
    if kind == "batch":
        return {"kind": kind, "stones": rng.randint(1, 16), "tilts": rng.randint(1, 9), "width": _log_int(rng, 24, 64),
                "height": _log_int(rng, 24, 64)}
    if kind == "designs":
        return {"kind": kind, "designs": _log_int(rng, 1, 64), "size": rng.randint(16, 32), "spp": 2 * rng.randint(4, 16)}
    if kind == "metrics":
        mode = rng.choice(["pose", "poses", "profile", "axes"])
        poses = {"pose": 1, "poses": _log_int(rng, 2, 700), "profile": abi.PROFILE_ANGLES}.get(mode)
        return {"kind": kind, "mode": mode, "poses": poses or abi.AXIS_TILTS * rng.randint(1, 4)}
    if kind in ("train", "predict"):
        return {"kind": kind, "batch": _log_int(rng, 1 if kind == "predict" else 64, 4096)}
    return {"kind": kind, "width": _log_int(rng, 160, 1920), "height": _log_int(rng, 90, 1080),
            "spp": _log_int(rng, 1, 200), "signature": rng.random() < 0.7}


_backend = None


def _the_backend():
    """The process's one backend, as a program keeps it."""
    global _backend
    if _backend is None:
        _backend = ixb.GpuBackend.acquire()
        if not _backend.available:
            raise RuntimeError("no CUDA backend")
    return _backend


def _frame_scene(case, rng):
    w, h, stone = case["width"], case["height"], case["stone"]
    if stone == "random":
        spec = workloads.random_stones(2, seed=int(rng.integers(1 << 30)))[1]  # the second of a pair absorbs
        return workloads.tilted_scene(spec, float(rng.uniform(0.0, 40.0)), w, h)
    make = {"round": workloads.round_brilliant_frame, "uniaxial": workloads.anisotropic_stress_frame,
            "sun": workloads.carved_sun_frame}[stone]
    fs = make(w, h)
    if stone == "sun":
        fs.camera = ixb.camera_new(float(rng.uniform(0.0, 6.28)), float(rng.uniform(0.5, 1.4)),
                                   workloads.FACE_UP_DISTANCE, workloads.DEFAULT_FOV_DEG)
    else:  # near face up
        fs.camera = ixb.camera_new(float(rng.uniform(0.0, 6.28)), float(workloads.FACE_UP_PITCH - rng.uniform(0.0, 0.2)),
                                   workloads.FACE_UP_DISTANCE, workloads.DEFAULT_FOV_DEG)
    return fs


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    b, kind = _the_backend(), case["kind"]
    if kind == "frame":
        return {"case": case, "backend": b, "scene": _frame_scene(case, rng), "offset": int(rng.integers(1 << 16)),
                "accum": np.zeros((case["height"], case["width"], 3), case["dtype"])}
    if kind == "batch":
        stones = workloads.random_stones(case["stones"], seed=int(rng.integers(1 << 30)))
        jobs = [(workloads.tilted_scene(s, t, case["width"], case["height"]), 0, s.spp)
                for s in stones for t in workloads.TILTS_DEG[:case["tilts"]]]
        return {"case": case, "plan": ixb.BatchPlan(b, jobs)}
    if kind == "designs":
        return {"case": case, "backend": b, "designs": surrogate.sample_designs(case["designs"], seed),
                "spec": surrogate.RenderSpec(case["size"], case["size"], case["spp"])}
    if kind == "metrics":
        spec = workloads.random_stones(1, seed=int(rng.integers(1 << 30)))[0]
        poses = [(0, float(rng.uniform(0.0, 6.28)), float(rng.uniform(0.3, 1.57))) for _ in range(case["poses"])]
        return {"case": case, "backend": b, "planes": spec.planes, "material": spec.material, "poses": poses,
                "lighting": ixb.MetricsLighting(light_yaw=0.85, light_pitch=float(rng.uniform(0.6, 1.2)))}
    if kind == "train":
        x, t = _batch(case, seed)
        return {"case": case, "net": surrogate.SurrogateMLP(seed=seed), "x": x, "t": t}
    if kind == "predict":
        return {"case": case, "ensemble": surrogate.SurrogateEnsemble(4, seed=seed), "x": _batch(case, seed)[0]}
    w, h = case["width"], case["height"]
    mat = materials.isotropic(materials.cauchy(1.76, 0.0, 0.0))
    base = workloads.round_brilliant_frame(8, 8)
    fs = ixb.FrameScene(ixb.camera_new(0.60, 0.45, 2.4, 42.0), w, h, base.planes, mat, 32, base.environment)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    # Sums of spp samples whose mean is uniform noise on a 1/32768 grid in [0, 2).
    color = torch.randint(0, 65536, (h, w, 3), device="cuda", generator=g).float() / 32768.0
    return {"case": case, "backend": b, "frame": fs, "scene": fs.to_abi(), "accum": color * float(case["spp"]),
            "rgba": torch.empty((h, w, 4), dtype=torch.uint8, device="cuda"), "stream": torch.cuda.Stream()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "frame":
        spp = case["spp"]
        if not state["backend"].try_accumulate(state["scene"], state["offset"], spp, state["accum"]):
            raise RuntimeError("declined: %s" % state["backend"].last_lost_reason())
        state["offset"] = (state["offset"] + spp) % (1 << 22)
        return state["accum"]
    if kind == "batch":
        state["plan"].run()
        return state["plan"].download()
    if kind == "designs":
        return surrogate.evaluate_designs(state["backend"], state["designs"], state["spec"])
    if kind == "metrics":
        return _metrics(state, case["mode"], case["poses"])
    if kind == "train":
        loss = state["net"].train_step(state["x"], state["t"], LR)
        return {"loss": loss, "w": [layer.w for layer in state["net"].layers],
                "b": [layer.b for layer in state["net"].layers]}
    if kind == "predict":
        return state["ensemble"].predict_members(state["x"])
    if not display.display_frame_device(state["backend"], state["scene"], case["spp"], state["accum"].data_ptr(),
                                        state["rgba"].data_ptr(), case["signature"],
                                        stream_ptr=state["stream"].cuda_stream):
        raise RuntimeError("declined: %s" % state["backend"].last_lost_reason())
    return state["rgba"]


def _metrics(state, mode, n):
    b, planes, mat, light = state["backend"], state["planes"], state["material"], state["lighting"]
    if mode == "pose":
        _, yaw, pitch = state["poses"][0]
        return b.evaluate_gem_optical_metrics(planes, mat, yaw, pitch, light)
    if mode == "poses":
        return b.evaluate_metrics_batch([(planes, mat.dispersion)], state["poses"], light)
    if mode == "profile":
        return b.evaluate_angular_profile(planes, mat, light)
    curves = b.evaluate_axis_profiles(planes, mat, abi.PROFILE_AZIMUTHS_DEG[:n // abi.AXIS_TILTS], light)
    return [[c.brilliance, c.extinction, c.windowing] for c in curves]


def work(case):
    kind = case["kind"]
    planes = 121 * 16
    if kind == "frame":
        px = case["width"] * case["height"]
        return {"bytes": planes + 2 * px * 3 * (4 if case["dtype"] == "float32" else 8),
                "flops": px * case["spp"] * FLOPS_PER_PATH[case["stone"]]}
    if kind == "batch":
        px = case["stones"] * case["tilts"] * case["width"] * case["height"]
        return {"bytes": case["stones"] * planes + px * 24, "flops": px * MEAN_SPP * FLOPS_PER_PATH["random"]}
    if kind == "designs":
        paths = case["designs"] * 9 * case["size"] ** 2 * case["spp"]
        return {"bytes": case["designs"] * (48 + 27 * 4), "flops": paths * FLOPS_PER_PATH["random"]}
    if kind == "metrics":
        # 18 x 18 fan cells; per cell 5 aperture rays of 3 wavelengths and 5 yaw-jittered
        # rays, about 6 facets each, 14 operations a plane (the sweeps trace one
        # wavelength of the aperture rays alone).
        rays = 324 * (20 if case["mode"] in ("pose", "poses") else 5)
        return {"bytes": planes + 20 * case["poses"], "flops": case["poses"] * rays * 6 * 80 * 14}
    if kind in ("train", "predict"):
        dims = surrogate.DIMS
        weights = sum(a * b for a, b in zip(dims[:-1], dims[1:]))
        n = case["batch"]
        if kind == "train":
            return {"bytes": 4 * n * (dims[0] + dims[-1]) + weights * 4 * 6, "flops": 6 * n * weights}
        return {"bytes": 4 * n * (dims[0] + 4 * dims[-1]) + 4 * weights * 2, "flops": 4 * 2 * n * weights}
    px = case["width"] * case["height"]
    # Sums, normal, depth, facet and signature in, RGBA8 out; 5 passes of 25 taps.
    return {"bytes": px * (12 + 12 + 4 + 4 + (4 if case["signature"] else 0) + 4), "flops": px * 5 * 25 * 30}


def _batch(case, seed):
    x = surrogate.normalize(surrogate.sample_designs(case["batch"], seed))
    t = np.random.default_rng(seed + 1).standard_normal((case["batch"], surrogate.N_OUTPUTS)).astype(np.float32)
    return x, t


def _weights(seed):
    """The starting weights SurrogateMLP(seed) documents: normal / sqrt(fan_in), zero biases."""
    g = np.random.default_rng(seed)
    dims = surrogate.DIMS
    return [(g.standard_normal((o, i)) / math.sqrt(i)).astype(np.float32).astype(np.float64)
            for i, o in zip(dims[:-1], dims[1:])]


def exact(case, seed):
    """In 64 bits: the networks' outputs, and the loss and updated weights of one Adam step.
    The traced results are Monte-Carlo sums of branching paths and the display's are
    bytes: they have no value in 64 bits to be compared with."""
    if case["kind"] == "predict":
        x = _batch(case, seed)[0].astype(np.float64)
        out = []
        for i in range(4):
            h, ws = x, _weights(seed + 1000 * i)
            for w in ws[:-1]:
                z = h @ w.T
                h = z / (1.0 + np.exp(-z))
            out.append(h @ ws[-1].T)
        return np.stack(out)
    if case["kind"] == "train":
        x, t = (torch.from_numpy(a).double() for a in _batch(case, seed))
        ws = [torch.from_numpy(w).requires_grad_() for w in _weights(seed)]
        bs = [torch.zeros(w.shape[0], dtype=torch.float64, requires_grad=True) for w in ws]
        h = x
        for i, (w, b) in enumerate(zip(ws, bs)):
            z = h @ w.T + b
            h = z if i == len(ws) - 1 else z * torch.sigmoid(z)
        loss = ((h - t) ** 2).mean()
        loss.backward()
        # Adam's first step: both moments are corrected to the gradient itself.  A bias
        # starts at zero and takes +-LR by its gradient's sign, which 16-bit activations
        # leave open where the gradient nearly cancels: no 64-bit value to be near to.
        step = lambda p: (p - LR * p.grad / (p.grad.abs() + 1e-8)).detach()  # noqa: E731
        return {"loss": loss.detach().item(), "w": [step(w) for w in ws], "b": [None] * len(bs)}
    return None
