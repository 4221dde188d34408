"""The reference-form a-trous tiles over special values with ordinary geometry, against the
oracle, bit for bit: infinite, NaN and negative variances and infinite and NaN colours, a few
of an image's, one in every 64x8 tile, and all of them; and finite negative variances alone,
whose sums are finite."""
import ctypes as C

import numpy as np
import pytest

import violet_gb300 as vg
from oracle import pyoracle as po
from tests.test_gpu_atrous_tile import inputs

pytestmark = pytest.mark.gpu


def spoil(color, var, w, h, kind):
    """Special values into copies of the (h, w, 2) planes."""
    color, var = color.reshape(h, w, 2).copy(), var.view(np.float16).reshape(h, w, 2).copy()
    rng = np.random.default_rng(w + h)
    if kind == "few":
        for k, v in enumerate((np.inf, np.nan, -np.inf, -3.0)):
            var[(7 * k + 3) % h, (53 * k + 11) % w, k & 1] = v
        color[h // 2, w // 3, 0] = 31 << 6
        color[h // 3, w // 2, 1] = (31 << 17) | (5 << 11)
    elif kind == "tile":
        var[3::8, 17::64, 0] = np.inf
        var[5::8, 40::64, 1] = np.nan
        color[6::8, 2::64, 1] = 31 << 22
    elif kind == "all":
        var[...] = np.where(rng.random(var.shape) < 0.5, np.inf, -1.0)
        var[rng.random(var.shape) < 0.2] = np.nan
        color[rng.random(color.shape) < 0.05] = (31 << 6) | 1
    else:
        var[rng.random(var.shape) < 0.3] *= np.float16(-1.0)
    return color.reshape(-1), var.reshape(-1).view(np.uint16)


@pytest.mark.parametrize("kind", ["few", "tile", "all", "negative"])
@pytest.mark.parametrize("step", [1, 3, 16])
@pytest.mark.parametrize("w,h", [(1, 1), (65, 9), (200, 70), (1000, 75)])
def test_atrous_values(w, h, step, kind):
    import torch

    n = w * h
    depth, gbuf, color, var = inputs(w, h, 0)
    color, var = spoil(color, var, w, h, kind)
    oc, ov = np.zeros(2 * n, np.uint32), np.zeros(2 * n, np.uint16)
    po.lib().vlto_denoise_atrous(w, h, po.ptr(depth), po.ptr(gbuf), po.ptr(color), po.ptr(var), po.ptr(oc),
                                 po.ptr(ov), step)
    dev = [torch.from_numpy(a.view(np.uint8).copy()).cuda() for a in (depth, gbuf, color, var)]
    gc, gv = torch.zeros(8 * n, dtype=torch.uint8, device="cuda"), torch.zeros(4 * n, dtype=torch.uint8, device="cuda")
    assert vg.lib().vlt_denoise_atrous(w, h, *[C.c_void_p(t.data_ptr()) for t in dev], C.c_void_p(gc.data_ptr()),
                                       C.c_void_p(gv.data_ptr()), step, None) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(gc.cpu().numpy().view(np.uint32), oc)
    np.testing.assert_array_equal(gv.cpu().numpy().view(np.uint16), ov)
