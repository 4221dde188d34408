"""The fast-history clamp (reference form) against the oracle, bit for bit, around the edges
of its staged tiles and of the image, with infinite and NaN codes among the colours."""
import ctypes as C

import numpy as np
import pytest

import violet_gb300 as vg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("special", [0, 1])
@pytest.mark.parametrize("w,h", [(1, 1), (31, 3), (32, 4), (33, 5), (65, 9), (200, 41)])
def test_fast_clamp(w, h, special):
    import torch

    n = w * h
    rng = np.random.default_rng(n + special)

    def words():
        c = (rng.integers(0, 18 << 6, 2 * n) | (rng.integers(0, 18 << 6, 2 * n) << 11)
             | (rng.integers(0, 18 << 5, 2 * n) << 22)).astype(np.uint32)
        c[rng.random(2 * n) < 0.2] = 0
        if special:
            c[rng.random(2 * n) < 0.05] = 31 << 6
            c[rng.random(2 * n) < 0.05] = (31 << 27) | (3 << 22)
        return c

    fast, color = words(), words()
    want = color.copy()
    po.lib().vlto_denoise_fast_history_clamp(w, h, po.ptr(fast), po.ptr(want))
    f, c = (torch.from_numpy(a.view(np.uint8).copy()).cuda() for a in (fast, color))
    assert vg.lib().vlt_denoise_fast_history_clamp(w, h, C.c_void_p(f.data_ptr()), C.c_void_p(c.data_ptr()), None) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(c.cpu().numpy().view(np.uint32), want)
