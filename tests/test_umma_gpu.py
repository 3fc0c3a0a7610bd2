"""FP16 stacks on the tensor cores (the FBP's default FP16 form and stacked-backproject's half mode):
edges of the 11 x 20 pixel tiles, of the slice shares of a CTA, of the angle stages, and rows with
non-finite values.

Tolerance: filtered sinograms round to 11 bits (2^-12 relative) and weights to 2^-12; on random
data, where neighbouring bins are independent, both add up to a few 1e-4 relative L2."""
import math

import numpy as np
import pytest
import torch

import oracle
import ufob

pytestmark = pytest.mark.gpu

TOL = 1e-3


def _raw(nz, P, W, seed):
    return np.random.default_rng(seed).standard_normal((nz, P, W)).astype(np.float32)


def _ref(raw, N, **bp):
    nz, P, W = raw.shape
    filt = oracle.fft_filter_ifft(raw.reshape(-1, W), size_x=N, crop_width=W).reshape(nz, P, W)
    return np.stack([oracle.backproject(filt[z].astype(np.float32), **bp) for z in range(nz)])


def _fbp(raw, N, **bp):
    f = ufob.FBP(filter_props={"size_x": N, "crop_width": raw.shape[-1]}, bp_props=bp, storage=ufob.F16)
    out = f.process(torch.from_numpy(raw).cuda()).cpu().numpy()
    ufob.device_status()
    return out


# tiles: one pixel short of, at and past the 11-wide and 20-high tile; odd and tiny widths
@pytest.mark.parametrize("W", [5, 10, 11, 12, 19, 20, 21, 45, 121])
def test_tile_edges(cuda, W):
    raw, N = _raw(17, 37, W, W), 1 << (W - 1).bit_length()
    assert oracle.rel_l2(_fbp(raw, N), _ref(raw, N)) < TOL


# slices: partly filled octets and 16-slice products, each share size and two shares
@pytest.mark.parametrize("nz", [17, 23, 33, 64, 70, 96, 113, 128, 131, 200, 257])
def test_slice_shares(cuda, nz):
    raw = _raw(nz, 40, 60, nz)
    got, ref = _fbp(raw, 64), _ref(raw, 64)
    for z in (0, 7, nz // 2, nz - 1):
        assert oracle.rel_l2(got[z], ref[z]) < TOL, z


# angles: fewer than a stage, partly filled stages and groups of 32, for each stage length
@pytest.mark.parametrize("nz", [20, 50, 120])
@pytest.mark.parametrize("P", [1, 2, 3, 7, 9, 31, 33, 70])
def test_angle_counts(cuda, nz, P):
    raw = _raw(nz, P, 48, P)
    assert oracle.rel_l2(_fbp(raw, 64), _ref(raw, 64)) < TOL


# blocks of 64 angles whose sums are added to the totals: block ends, for either split of the totals
# between registers and shared memory (up to 32, 64, 96 and 128 slices)
@pytest.mark.parametrize("nz", [17, 33, 65, 128])
@pytest.mark.parametrize("P", [63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 161, 200, 320])
def test_angle_blocks(cuda, nz, P):
    raw = _raw(nz, P, 40, P)
    got, ref = _fbp(raw, 64), _ref(raw, 64)
    for z in range(nz):
        assert oracle.rel_l2(got[z], ref[z]) < TOL, z


# Large sums of one sign, as of rows that were not filtered: the tensor cores cut each addition off at the
# accumulator's last bit, on average half of 2^-23 of the sum so far.  In a block of 64 angles that is at
# most 64 / 4 * 2^-23 = 1.9e-6 of its sum; the weights' rounding (2^-12 at most, 2^-12 / sqrt(3) in the mean)
# of neighbouring bins 0.4 apart adds 0.4 * 1.4e-4 / sqrt(1500) = 1.5e-6 and FP32 totals less.  (One sum over
# all 1500 angles: 3.8e-5.)  The reference takes the rows as stored, rounded to 16 bits.
@pytest.mark.parametrize("nz", [20, 50, 120])
def test_sums_of_one_sign(cuda, nz):
    P, W = 1500, 96
    raw = np.random.default_rng(nz).uniform(1.0, 2.0, (nz, P, W)).astype(np.float16).astype(np.float32)
    t = ufob.StackedBackprojectTask(precision_mode="half", axis_pos=W / 2)
    got = t.process(torch.from_numpy(raw).cuda()).cpu().numpy()
    ufob.device_status()
    for z in (0, nz - 1):
        ref = oracle.stacked_backproject(raw[z:z + 1], "single", axis_pos=W / 2)[0]
        assert oracle.rel_l2(got[z], ref) < 5e-6, z


# the issuing lanes read window starts that the other lanes of their warps write, anew for every 32
# angles: passes over seven such groups agree to the bit, for each stage length
@pytest.mark.parametrize("nz", [20, 50, 120])
def test_passes_repeat(cuda, nz):
    raw = _raw(nz, 200, 150, nz)
    f = ufob.FBP(filter_props={"size_x": 256, "crop_width": 150}, storage=ufob.F16)
    dev = torch.from_numpy(raw).cuda()
    first = f.process(dev).clone()
    for _ in range(4):
        assert torch.equal(f.process(dev), first)
    ufob.device_status()
    assert oracle.rel_l2(first[nz - 1:].cpu().numpy(), _ref(raw[nz - 1:], 256)) < TOL


def test_roi_axis_offset(cuda):
    raw = _raw(18, 60, 100, 4)
    bp = dict(axis_pos=43.3, angle_step=math.pi / 50, angle_offset=0.7, roi_x=70, roi_y=5, roi_width=61,
              roi_height=90)  # part of the region sees no detector
    assert oracle.rel_l2(_fbp(raw, 128, **bp), _ref(raw, 128, **bp)) < TOL


@pytest.mark.parametrize("nz", [17, 45])
def test_stacked_half(cuda, nz):
    raw = _raw(nz, 50, 77, nz)
    t = ufob.StackedBackprojectTask(precision_mode="half", axis_pos=36.5)
    got = t.process(torch.from_numpy(raw).cuda()).cpu().numpy()
    ref = np.stack([oracle.stacked_backproject(raw[z:z + 1], "single", axis_pos=36.5)[0] for z in range(nz)])
    assert oracle.rel_l2(got, ref) < TOL


# one infinite bin, FP16 overflow and a NaN row: only the pixels that interpolate them may change.
# stacked-backproject takes the rows as they are, so the affected pixels are known exactly.
@pytest.mark.parametrize("bad", [math.inf, -math.inf, math.nan, 1.0e6])
def test_nonfinite_bins_stay_local(cuda, bad):
    nz, P, W, axis = 20, 33, 90, 44.6
    raw = _raw(nz, P, W, 9)
    dirty = raw.copy()
    hits = [(3, 5, 41), (3, 32, 0), (17, 11, W - 1)]
    for z, p, j in hits:
        dirty[z, p, j] = bad
    t = ufob.StackedBackprojectTask(precision_mode="half", axis_pos=axis)
    clean = t.process(torch.from_numpy(raw).cuda()).cpu().numpy()
    got = t.process(torch.from_numpy(dirty).cuda()).cpu().numpy()
    ufob.device_status()
    x = np.arange(W) + 0.5 - np.float32(axis)
    touched = np.zeros((nz, W, W), bool)
    near = np.zeros((nz, W, W), bool)
    for z, p, j in hits:
        a = p * math.pi / P
        h = x[None, :] * math.cos(a) - x[:, None] * math.sin(a) + np.float32(axis) - 0.5
        touched[z] |= np.abs(h - j) < 0.999
        near[z] |= np.abs(h - j) < 1.001
    assert not np.isfinite(got[touched]).any()
    assert np.isfinite(got[~near]).all()
    assert oracle.rel_l2(got[~near], clean[~near]) < TOL


# bad bins in several octets, stages and windows, for each stage length: every finite pixel has the bits
# of the same stack with zeros in their place, and the other slices those of the clean stack
@pytest.mark.parametrize("nz", [20, 50, 90, 120, 250])
def test_nonfinite_bins_leave_the_rest(cuda, nz):
    P, W = 70, 120
    raw = _raw(nz, P, W, nz)
    rng = np.random.default_rng(nz)
    zeroed, dirty = raw.copy(), raw.copy()
    bad_slices = sorted({0, 7, 9, nz // 2, nz - 1})
    for z in bad_slices:
        for _ in range(12):
            p, j = rng.integers(P), rng.integers(W)
            dirty[z, p, j] = rng.choice([math.nan, math.inf, -math.inf, 1.0e6, -1.0e6])
            zeroed[z, p, j] = 0.0
    dirty[9, :, 31], zeroed[9, :, 31] = math.nan, 0.0  # a dead detector pixel
    t = ufob.StackedBackprojectTask(precision_mode="half", axis_pos=57.3)
    clean, want, got = (t.process(torch.from_numpy(x).cuda()).cpu().numpy() for x in (raw, zeroed, dirty))
    ufob.device_status()
    finite = np.isfinite(got)
    assert not finite.all() and finite.any()
    np.testing.assert_array_equal(got[finite], want[finite])
    good = [z for z in range(nz) if z not in bad_slices]
    np.testing.assert_array_equal(got[good], clean[good])


# a dead slice (the FFT fills its rows with NaN, and those of the slice it is transformed with) costs its
# octet one look-up per pixel: the pass stays near the clean one (sampling all slices at the angles
# concerned took 40 times as long)
def test_dead_slice_is_cheap(cuda):
    nz, P, W = 64, 600, 512
    f = ufob.FBP(storage=ufob.F16)
    clean = torch.randn(nz, P, W, device="cuda")
    dead = clean.clone()
    dead[17, :, 200] = math.nan

    def ms(x, out):
        f.process(x, out=out)
        a, b = torch.cuda.Event(True), torch.cuda.Event(True)
        a.record()
        for _ in range(5):
            f.process(x, out=out)
        b.record()
        torch.cuda.synchronize()
        return a.elapsed_time(b)

    outs = [torch.empty(nz, W, W, device="cuda") for _ in range(2)]
    t_clean, t_dead = ms(clean, outs[0]), ms(dead, outs[1])
    ufob.device_status()
    assert t_dead < 5 * t_clean, (t_dead, t_clean)
    good = [z for z in range(nz) if z not in (16, 17)]
    assert torch.equal(outs[0][good], outs[1][good])
    assert torch.isnan(outs[1][17, W // 4:3 * W // 4, W // 4:3 * W // 4]).all()


# the host pipeline makes large images in bands of rows, and shares a remainder of few slices among the
# other chunks: the same bits as one call of all slices, whatever the chunks (70 slices in chunks of 32
# were once 32 + 32 on the tensor cores and 6 on the slice-quad kernel)
@pytest.mark.parametrize("nz,chunk", [(20, 32), (70, 32), (64, 64), (33, 32), (49, 32), (18, 17), (52, 17)])
def test_host_bands(cuda, nz, chunk):
    P, W = 20, 1030
    raw = torch.randn(nz, P, W)
    f = ufob.FBP(filter_props={"size_x": 2048, "crop_width": W}, storage=ufob.F16)
    got = f.process_host(raw.pin_memory(), out=torch.empty(nz, W, W).pin_memory(), slices_per_chunk=chunk)
    want = f.process(raw.cuda()).cpu()
    ufob.device_status()
    assert torch.equal(got, want)
    ref = _ref(raw[nz - 1:].numpy(), 2048)  # a slice of the last chunk
    assert oracle.rel_l2(got[nz - 1:].numpy(), ref) < TOL


ROI = dict(roi_x=900, roi_y=1100, roi_width=64, roi_height=48)


# 260 slices of 1500 x 2048 are more than one group: the four left over take the kernel of the call
def test_remainder_of_groups(cuda):
    sino = torch.randn(260, 1500, 2048, device="cuda")
    f = ufob.FBP(bp_props=ROI, storage=ufob.F16)
    whole, tail = f.process(sino), f.process(sino[200:].contiguous())
    ufob.device_status()
    assert torch.equal(whole[200:], tail)


# slices so large that fewer than 17 of them would fit a group at four bytes a value
def test_large_slices(cuda):
    nz, P, W = 20, 4500, 5000
    raw = torch.randn(nz, P, W).pin_memory()
    f = ufob.FBP(filter_props={"size_x": 8192, "crop_width": W}, bp_props=ROI, storage=ufob.F16)
    host = f.process_host(raw, out=torch.empty(nz, 48, 64).pin_memory())
    assert torch.equal(f.process(raw.cuda()).cpu(), host)
    ufob.device_status()
    assert oracle.rel_l2(host[7:8].numpy(), _ref(raw[7:8].numpy(), 8192, **ROI)) < TOL


# every FFT size of the register-radix filter (its teams meet as half warps at 256, on named barriers, or
# one team fills a CTA at 4096, which stores octets another way) and the shared-memory filter on both sides
SIZES = [(60, 64), (250, 256), (500, 512), (1000, 1024), (2000, 2048), (4000, 4096), (5000, 8192)]


# One angle of 0 degrees puts pixel x of any row on bin x with weight 1, so the image is the octet's halves
# times pi: the FP16 rounding of the rows form up to one step of a value whose FP32 round-off differs (the FFT
# pairs other rows), for small values one step of the row's largest.
@pytest.mark.parametrize("W,N", SIZES)
@pytest.mark.parametrize("nz", [17, 23])
def test_octet_cells(cuda, W, N, nz):
    raw = _raw(nz, 1, W, N)
    got = _fbp(raw, N, roi_x=0, roi_y=1, roi_width=W, roi_height=2) / np.float32(math.pi)
    ref = oracle.fft_filter_ifft(raw.reshape(-1, W), size_x=N, crop_width=W)
    f = ufob.FilterTask(size_x=N, crop_width=W)
    for z in range(nz):
        rows = f.process(torch.from_numpy(raw[z]).cuda(), dtype=ufob.F16).float().cpu().numpy()[0]
        scale = float(np.abs(rows).max())
        for y in range(2):
            assert oracle.rel_l2(got[z, y], ref[z]) < 2e-3
            assert np.all(np.abs(got[z, y] - rows) <= 2.0 ** -10 * np.abs(rows) + 2.0 ** -11 * scale)


# raw projections through the preprocessing fused into the filter
@pytest.mark.parametrize("W,N", SIZES)
def test_octets_from_projections(cuda, W, N):
    nz, P = 19, 6
    rng = np.random.default_rng(W)
    dark = rng.uniform(90, 110, (nz, W)).astype(np.float32)
    flat = (dark + rng.uniform(800, 1200, (nz, W))).astype(np.float32)
    data = (dark + rng.uniform(50, 1000, (P, nz, W))).astype(np.float32)
    roi = dict(roi_x=W // 3, roi_y=W // 4, roi_width=40, roi_height=23)
    f = ufob.FBP(filter_props={"size_x": N, "crop_width": W}, bp_props=roi, storage=ufob.F16)
    dev = [torch.from_numpy(a).cuda() for a in (data, dark, flat)]
    got = f.process_projections(dev[0], ffc=ufob.FlatFieldCorrectTask(absorption_correct=1), dark=dev[1],
                                flat=dev[2]).cpu().numpy()
    ufob.device_status()
    sinos = oracle.transpose_projections(oracle.flat_field_correct(data, dark, flat, absorption_correct=True))
    ref = _ref(np.ascontiguousarray(sinos, dtype=np.float32), N, **roi)
    for z in range(nz):
        assert oracle.rel_l2(got[z], ref[z]) < TOL, z
