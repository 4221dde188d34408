"""The reference-form a-trous tiles at every step up to the largest, on an image large enough
for the block size of many tiles per SM, with a few special fwidth_z (pixels that run the
per-pixel form beside others of their block), against the oracle, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import violet_gb300 as vg
from oracle import pyoracle as po
from tests.test_gpu_atrous_tile import inputs

pytestmark = pytest.mark.gpu

W, H = 1280, 640  # 1,600 tiles of 64x8


@pytest.fixture(scope="module")
def planes():
    n = W * H
    depth, gbuf, color, var = inputs(W, H, 0)
    at = np.random.default_rng(5).integers(0, n, n // 500)
    gbuf[2 * n + at] = np.where(np.arange(at.size) % 2, 0x7C00, 0xC000)  # infinite, -2
    return depth, gbuf, color, var


@pytest.mark.parametrize("step", [1, 4, 7, 12, 13, 16])
def test_atrous_steps(planes, step):
    import torch

    n = W * H
    oc, ov = np.zeros(2 * n, np.uint32), np.zeros(2 * n, np.uint16)
    po.lib().vlto_denoise_atrous(W, H, *[po.ptr(a) for a in planes], po.ptr(oc), po.ptr(ov), step)
    dev = [torch.from_numpy(a.view(np.uint8).copy()).cuda() for a in planes]
    gc, gv = torch.zeros(8 * n, dtype=torch.uint8, device="cuda"), torch.zeros(4 * n, dtype=torch.uint8, device="cuda")
    assert vg.lib().vlt_denoise_atrous(W, H, *[C.c_void_p(t.data_ptr()) for t in dev], C.c_void_p(gc.data_ptr()),
                                       C.c_void_p(gv.data_ptr()), step, None) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(gc.cpu().numpy().view(np.uint32), oc)
    np.testing.assert_array_equal(gv.cpu().numpy().view(np.uint16), ov)
