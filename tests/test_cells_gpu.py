"""FP32 stacks from slice cells: the same bits as the row kernel (tile 2, 32 x 32 pixels of four
slices, whose arithmetic and order it keeps) at edges of its 32 x 64 x 8 tiles, odd widths and
regions, angle counts around its stages and sum blocks, quadrants and exact 0 and 90 degree angles,
and the FP64 oracle on a few slices."""
import math

import numpy as np
import pytest
import torch

import oracle
import ufob

pytestmark = pytest.mark.gpu


def _both(sino, **props):
    t = torch.from_numpy(sino).cuda()
    a = ufob.BackprojectTask(**props).process(t)
    b = ufob.BackprojectTask(tile=2, **props).process(t)
    torch.cuda.synchronize()
    ufob.device_status()
    return a.cpu().numpy(), b.cpu().numpy()


# (slices, angles, width, properties): both sides of the rule that picks the kernel
CASES = [
    (64, 40, 250, {}),
    (5, 33, 1100, {}),
    (37, 1, 353, {}),
    (37, 7, 353, dict(axis_pos=150.25)),
    (33, 8, 385, dict(angle_offset=math.pi / 2)),
    (40, 17, 417, dict(angle_step=math.pi / 2)),  # exact 0, 90, 180, 270 degrees
    (40, 24, 416, dict(axis_pos=207.5, angle_step=math.pi / 4, angle_offset=5.5)),
    (70, 31, 256, dict(roi_x=3, roi_y=17, roi_width=243, roi_height=191)),
    (32, 64, 320, dict(roi_x=250, roi_y=100, roi_width=320, roi_height=500)),  # partly beyond the detector
]


@pytest.mark.parametrize("nz,P,W,props", CASES)
def test_same_bits_as_rows(cuda, nz, P, W, props):
    sino = np.random.default_rng(nz * P + W).standard_normal((nz, P, W)).astype(np.float32)
    got, rows = _both(sino, **props)
    np.testing.assert_array_equal(got, rows)
    if not props.get("roi_width"):
        for z in (0, nz - 1):
            ref = oracle.backproject(sino[z], **props)
            assert oracle.rel_l2(got[z], ref) < 2e-5


def test_nonfinite_and_groups(cuda):
    """Two groups of 32 slices; infinities and NaNs reach the same pixels as in the row kernel."""
    sino = np.random.default_rng(5).standard_normal((41, 30, 300)).astype(np.float32)
    sino[3, 4, 100], sino[40, 29, 0], sino[35, 7, 299] = math.inf, math.nan, -math.inf
    got, rows = _both(sino)
    np.testing.assert_array_equal(got, rows)


def test_unaligned_rows(cuda):
    """A pitch and a base the row kernel has to restage."""
    nz, P, W = 32, 20, 321
    buf = torch.randn(nz, P, W + 2, device="cuda")
    out = [torch.empty(nz, W, W, device="cuda") for _ in range(2)]
    for o, tile in zip(out, (-1, 2)):
        bp = ufob.BackprojectTask(tile=tile)
        ufob.check(ufob.lib().ufob_backproject_run(bp._h, buf.data_ptr() + 4, ufob.F32, ufob.ROWS, W, P, nz, W + 2,
                                                   (W + 2) * P, o.data_ptr(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1])


# One handle driven on several streams by one thread: the cells of a call must not be packed while another
# call's kernel still reads the buffer (the table is built, and the buffer grown, by the first call).
@pytest.mark.parametrize("make", [lambda: ufob.BackprojectTask(axis_pos=190.0),
                                  lambda: ufob.StackedBackprojectTask(precision_mode="single", axis_pos=190.0)])
def test_two_streams(cuda, make):
    nz, P, W = 70, 120, 384
    task = make()
    stacks = [torch.randn(nz, P, W, device="cuda") for _ in range(2)]
    want = [task.process(x).clone() for x in stacks]
    outs = [torch.empty_like(w) for w in want]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(5):
        for o in outs:
            o.zero_()
        torch.cuda.synchronize()
        for x, o, st in zip(stacks, outs, streams):
            task.process(x, out=o, stream=st)
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert torch.equal(o, w)
    ufob.device_status()


# The buffer stays within 2 GiB: eight slices of 8192 x 9000 are 2.36 GB as cells, so they run from rows.
def test_large_sinograms_take_no_cells(cuda):
    nz, P, W = 5, 9000, 8192
    sino = torch.zeros(nz, P, W, device="cuda")
    sino[:, :, ::7] = torch.rand(nz, P, (W + 6) // 7, device="cuda")
    roi = dict(roi_x=3500, roi_y=3600, roi_width=1024, roi_height=1024)  # 512 tiles of 32 x 64
    task = ufob.BackprojectTask(**roi)
    out = torch.empty(nz, 1024, 1024, device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    task.process(sino, out=out)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 64 << 20
    want = ufob.BackprojectTask(tile=2, **roi).process(sino)
    assert torch.equal(out, want)


# ---- launches that have to be the cell kernel: a packing and a backprojection per 32 slices

def _launches(f):
    n = ufob.launch_count()
    out = f()
    return out, ufob.launch_count() - n


def _cells(task, run):
    run(task)  # builds the angle table
    out, n = _launches(lambda: run(task))
    assert n == 2 * ((out.shape[0] + 31) // 32), "not the cell kernel"
    return out


# odd widths and heights, odd regions inside and across the detector's edge, two to four groups with a
# remainder of few slices, angle counts around stages and sum blocks, steep and exact angles
CELL_CASES = [
    (96, 40, 250, {}),
    (5, 33, 1100, {}),
    (37, 7, 353, dict(axis_pos=150.25)),
    (32, 8, 385, dict(angle_offset=math.pi / 2)),
    (61, 17, 417, dict(angle_step=math.pi / 2)),
    (64, 24, 416, dict(axis_pos=207.5, angle_step=math.pi / 4, angle_offset=5.5)),
    (101, 31, 400, dict(roi_x=3, roi_y=17, roi_width=383, roi_height=371)),
    (32, 64, 320, dict(roi_x=250, roi_y=100, roi_width=320, roi_height=500)),
]


@pytest.mark.parametrize("nz,P,W,props", CELL_CASES)
def test_cells_give_the_rows_bits(cuda, nz, P, W, props):
    t = torch.randn(nz, P, W, device="cuda")
    got = _cells(ufob.BackprojectTask(**props), lambda task: task.process(t))
    assert torch.equal(got, ufob.BackprojectTask(tile=2, **props).process(t))
    ufob.device_status()
    z = nz - 1
    ref = oracle.backproject(t[z].cpu().numpy(), **props)
    # rows of noise: 32-bit detector coordinates (2^-14 of a bin at 1100) times the step to the next bin
    assert oracle.rel_l2(got[z].cpu().numpy(), ref) < 1e-4


def test_cells_nonfinite(cuda):
    t = torch.randn(61, 30, 417, device="cuda")
    t[3, 4, 100], t[60, 29, 0], t[35, 7, 416] = math.inf, math.nan, -math.inf
    got = _cells(ufob.BackprojectTask(), lambda task: task.process(t)).cpu().numpy()
    np.testing.assert_array_equal(got, ufob.BackprojectTask(tile=2).process(t).cpu().numpy())


def test_cells_from_unaligned_rows(cuda):
    """An odd pitch and base: the packing reads them in place, the row kernel restages."""
    nz, P, W = 56, 20, 321
    buf = torch.randn(nz, P, W + 2, device="cuda")
    out = [torch.empty(nz, W, W, device="cuda") for _ in range(2)]

    def run(task, o):
        ufob.check(ufob.lib().ufob_backproject_run(task._h, buf.data_ptr() + 4, ufob.F32, ufob.ROWS, W, P, nz, W + 2,
                                                   (W + 2) * P, o.data_ptr(), torch.cuda.current_stream().cuda_stream))
        return o

    _cells(ufob.BackprojectTask(), lambda task: run(task, out[0]))
    run(ufob.BackprojectTask(tile=2), out[1])
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1])


# launches whose last waves are nearly empty stay with the row kernel, the others take the cells
@pytest.mark.parametrize("nz,W,cells", [(64, 288, False), (64, 320, False), (40, 416, False), (24, 480, True),
                                        (32, 512, True), (12, 1001, True)])
def test_filled_waves(cuda, nz, W, cells):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes chosen for 148 SMs")
    t = torch.randn(nz, 3, W, device="cuda")
    task = ufob.BackprojectTask()
    task.process(t)
    got, n = _launches(lambda: task.process(t))
    assert n == (2 * ((nz + 31) // 32) if cells else 1)
    assert torch.equal(got, ufob.BackprojectTask(tile=2).process(t))
