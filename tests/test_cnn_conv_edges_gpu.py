"""Convolution kernels at the edges of their tiling, against the FP64 oracle: channel counts whose
K = 9 * Cin does not fill a chunk of 64 or crosses taps inside one, output columns split over CTAs
unevenly, weight gradients with several taps per CTA and a last, smaller share of them, channels past
one CTA's columns, pixel counts around a chunk and a CTA's range, and an unaligned gradient buffer."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
import ufob
from test_cnn_gpu import _as64, _bf16, _fwd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ci,co,h,w", [(48, 48, 7, 9), (16, 144, 5, 11), (64, 192, 8, 8), (192, 96, 4, 4),
                                       (32, 240, 16, 8), (16, 16, 1, 1), (32, 16, 1, 130)])
def test_forward_edges(cuda, ci, co, h, w):
    rng = np.random.default_rng(ci * co + h)
    x, wt = rng.standard_normal((2, h, w, ci)), rng.standard_normal((co, 9, ci)) / np.sqrt(9 * ci)
    xb, wb = _bf16(x), _bf16(wt)
    # FP32 sums of at most 9 * 256 exact products: sqrt(2304) * 2^-24 = 3e-6 relative
    assert oracle.rel_l2(_fwd(xb, wb).cpu().numpy(), oracle.conv3x3_nhwc(_as64(xb), _as64(wb))) < 1e-5


@pytest.mark.parametrize("ci,co,n,h,w", [(48, 48, 2, 7, 9), (144, 16, 1, 8, 8), (16, 144, 3, 5, 5), (32, 32, 1, 1, 1),
                                         (16, 32, 2, 33, 31), (256, 256, 1, 6, 7), (64, 80, 5, 16, 16)])
@pytest.mark.parametrize("shift", [0, 1])
def test_weight_gradient_edges(cuda, ci, co, n, h, w, shift):
    rng = np.random.default_rng(ci + 3 * co + h)
    xb, dzb = _bf16(rng.standard_normal((n, h, w, ci))), _bf16(rng.standard_normal((n, h, w, co)))
    fn = ufob.lib().ufob_conv3x3_wgrad
    fn.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int] * 5 + [ctypes.c_void_p]
    fn.restype = ctypes.c_int
    buf = torch.zeros(co * 9 * ci + 1, dtype=torch.float32, device="cuda")
    dw = buf[shift:shift + co * 9 * ci]
    ufob.check(fn(xb.data_ptr(), dzb.data_ptr(), dw.data_ptr(), n, h, w, ci, co, None))
    torch.cuda.synchronize()
    ufob.device_status()
    ref = oracle.conv3x3_wgrad_nhwc(_as64(xb), _as64(dzb))
    assert oracle.rel_l2(dw.cpu().numpy().reshape(co, 9, ci), ref) < 1e-5
