"""General backprojection: centre-position sweeps of parallel geometries on the staged column kernel
and the column walk that reuses rows, against the FP64 oracle (src/ufo-general-backproject-task.c's
transform chain) at the edges: partly filled columns of 16, detector heights that are no multiple of
four (rows of the transposed projections), descending and coarse steps, centres far from the middle,
tilted axes, FP16 samples, and magnifications on both sides of one row per voxel.

Tolerance: FP32 coordinates and sums, 2e-5 relative L2 (half: FP16 samples on both sides)."""
import math

import numpy as np
import pytest
import torch

import oracle
import ufob

pytestmark = pytest.mark.gpu


def _proj(n, H, W, seed):
    p = np.random.default_rng(seed).standard_normal((n, H, W)).astype(np.float32)
    k = np.ones(5, np.float32) / 5  # smooth, so that the interpolation is well conditioned
    p = np.apply_along_axis(lambda r: np.convolve(r, k, "same"), 2, p)
    return np.ascontiguousarray(np.apply_along_axis(lambda r: np.convolve(r, k, "same"), 1, p).astype(np.float32))


def _run(proj, props, staging="auto", compute="float"):
    n = proj.shape[0]
    t = ufob.GeneralBackprojectTask(num_projections=n)
    t.set_property("staging", staging)
    t.set_property("compute-type", compute)
    for k, v in props.items():
        t.set_property(k, v)
    out = t.process(torch.from_numpy(proj).cuda())
    torch.cuda.synchronize()
    ufob.device_status()
    return out.cpu().numpy()


def _oracle(proj, props):
    kw = {k.replace("-", "_") if k in ("x-region", "y-region") else k: v for k, v in props.items()}
    return oracle.general_backproject(proj, proj.shape[0], **kw)


BASE = {"x-region": (-20.0, 21.0, 1.0), "y-region": (-17.0, 20.0, 1.0), "center-position-x": 33.25,
        "center-position-z": 21.5}
SWEEPS = [
    (45, 66, {"parameter": "center-position-x", "z": 2.0, "region": (31.0, 35.0, 0.25)}),         # 16 slices
    (42, 67, {"parameter": "center-position-x", "z": -3.5, "region": (20.0, 46.0, 1.53)}),        # 17, W odd
    (41, 64, {"parameter": "center-position-x", "z": 0.0, "region": (34.0, 29.0, -0.5)}),         # descending
    (44, 64, {"parameter": "center-position-x", "z": 1.0, "region": (30.0, 57.0, 3.0)}),          # 9, three bins
    (43, 64, {"parameter": "center-position-x", "z": 4.0, "region": (-9.0, 90.0, 2.5), "axis-angle-x": 0.4}),
    (44, 64, {"parameter": "center-position-z", "z": 1.0, "region": (18.0, 25.0, 0.3), "axis-angle-x": 0.6}),
    (44, 64, {"parameter": "center-position-z", "z": 1.0, "region": (10.0, 30.0, 1.1), "detector-angle-y": 0.05}),
]


@pytest.mark.parametrize("H,W,props", SWEEPS)
def test_centre_sweeps(cuda, H, W, props):
    proj = _proj(40, H, W, H + W)
    props = {**BASE, **props}
    got, ref = _run(proj, props), _oracle(proj, props)
    assert got.shape == ref.shape
    for z in range(ref.shape[0]):
        assert np.linalg.norm(got[z] - ref[z]) < 2e-5 * np.linalg.norm(ref) / math.sqrt(ref.shape[0]), z


def test_centre_sweep_half(cuda):
    proj = _proj(30, 42, 64, 8)
    props = {**BASE, "parameter": "center-position-x", "z": 1.0, "region": (31.0, 36.0, 0.25)}
    ref = _oracle(proj.astype(np.float16).astype(np.float32), props)
    assert oracle.rel_l2(_run(proj, props, compute="half"), ref) < 2e-5


# v per voxel: 0.5 .. 1.6 rows (cone on both sides of the axis, coarse and descending z, roll-free tilt)
WALKS = [
    {"axis-angle-x": math.pi / 6, "region": (-18.0, 18.0, 1.0)},
    {"axis-angle-x": math.pi / 6, "region": (-18.0, 18.0, 1.15)},   # 0.996 rows
    {"axis-angle-x": 2.2, "region": (-9.0, 9.0, 1.0)},              # v falls along z
    {"region": (-10.0, 10.0, 1.0)},                                 # one row exactly
    {"region": (-10.0, 10.0, 0.5)},
    {"source-position-y": -90.0, "detector-position-y": 25.0, "region": (-15.0, 15.0, 1.0)},
    {"source-position-y": -400.0, "detector-position-y": 10.0, "region": (-15.0, 15.0, 0.9)},
]


@pytest.mark.parametrize("props", WALKS)
def test_column_walks(cuda, props):
    proj = _proj(36, 45, 64, len(props))
    props = {**BASE, **props}
    ref = _oracle(proj, props)
    got = _run(proj, props)
    assert oracle.rel_l2(got, ref) < 2e-5
    assert oracle.rel_l2(got, _run(proj, props, staging="texture")) < 2e-5


# steps too coarse to stage: the texture gathers do it, and no copy of the projections is made for it
def test_unstaged_sweep_takes_no_memory(cuda):
    proj = torch.randn(64, 512, 1024, device="cuda")
    t = ufob.GeneralBackprojectTask(num_projections=64)
    for k, v in {**BASE, "center-position-x": 512.0, "center-position-z": 256.0, "parameter": "center-position-x",
                 "z": 3.0, "region": (200.0, 800.0, 30.0)}.items():
        t.set_property(k, v)
    out = torch.empty(20, 37, 41, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    t.process(proj, out=out)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < proj.numel()  # a quarter of the copy
    t.set_property("staging", "texture")
    assert torch.equal(out, t.process(proj))
    ufob.device_status()
