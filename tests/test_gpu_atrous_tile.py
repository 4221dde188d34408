"""The reference-form a-trous pass over staged tiles (steps up to 16) and per pixel (larger
steps) against the oracle, bit for bit: at the edges of the 64x8 tiles and of the image,
and with inputs on which a block leaves the short path (infinite and NaN colours,
infinite, NaN and negative variances, negative and infinite fwidth_z, tiny depths)."""
import ctypes as C

import numpy as np
import pytest

import violet_gb300 as vg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (63, 7), (64, 8), (65, 9), (129, 33), (200, 70), (1000, 75)]


def inputs(w, h, special):
    n = w * h
    host = vg.Scene(17, w, h, disocclusion_frac=0.05).generate_host(2)
    rng = np.random.default_rng(w * 1000 + h)
    # R11G11B10 words with every exponent code below 31, zeros among them
    def words():
        r = rng.integers(0, 31 << 6, n, dtype=np.uint32)
        g = rng.integers(0, 31 << 6, n, dtype=np.uint32)
        b = rng.integers(0, 31 << 5, n, dtype=np.uint32)
        # mostly mid-range exponents, so that weights are not all 0
        mid = rng.random(n) < 0.9
        r = np.where(mid, (14 << 6) + (r & 0xFF), r)
        g = np.where(mid, (14 << 6) + (g & 0xFF), g)
        b = np.where(mid, (14 << 5) + (b & 0x7F), b)
        return (r | (g << 11) | (b << 22)).astype(np.uint32)

    color = np.stack([words(), words()], -1).reshape(-1).copy()
    var = rng.lognormal(0, 3, 2 * n).clip(0, 60000).astype(np.float16)
    var[rng.random(2 * n) < 0.05] = 0
    var[rng.random(2 * n) < 0.01] = np.float16(-0.0)
    depth, gbuf = host["depth"], host["gbuffer"]
    if special:
        k = max(1, n // 97)
        at = lambda: rng.integers(0, n, k)  # noqa: E731
        color[2 * at()] = 31 << 6                      # infinite red
        color[2 * at() + 1] = (31 << 17) | (5 << 11)   # NaN green
        var[2 * at()] = np.inf
        var[2 * at() + 1] = np.nan
        var[2 * at()] = -1.5
        depth[at()] = 1e-30
        depth[at()] = 3e38
        gbuf[2 * n + at()] = 0x0000C000                # fwidth_z -2
        gbuf[2 * n + at()] = 0x00007C00                # fwidth_z infinite
    return depth, gbuf, color, var.view(np.uint16)


@pytest.mark.parametrize("special", [0, 1])
@pytest.mark.parametrize("step", [1, 2, 3, 8, 16, 17])
@pytest.mark.parametrize("w,h", SIZES)
def test_atrous_tile(w, h, step, special):
    import torch

    n = w * h
    depth, gbuf, color, var = inputs(w, h, special)
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
