"""The disocclusion fix and the spatial fallback (reference form) against the oracle, bit
for bit, with tiles of no, few (weights evaluated by the block) and many short-history
pixels (each walks its taps), at sizes around the 32x4 tiles. The float forms run the same
scheme and are compared over whole frames elsewhere."""
import ctypes as C

import numpy as np
import pytest

import violet_gb300 as vg
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.0, 0.01, 0.06, 0.3, 1.0])
@pytest.mark.parametrize("w,h", [(1, 1), (31, 3), (32, 4), (33, 5), (100, 37), (257, 66)])
def test_short_history_filters(w, h, share):
    import torch

    n = w * h
    host = vg.Scene(23, w, h, disocclusion_frac=0.05).generate_host(1)
    rng = np.random.default_rng(n + int(100 * share))
    # lengths by 2x2 quad (a pixel is short when its quad's longest history is below 4), 0 for some
    quad = np.where(rng.random(((h + 1) // 2, (w + 1) // 2)) < share, rng.integers(1, 4, ((h + 1) // 2, (w + 1) // 2)), 9)
    length = quad.repeat(2, 0).repeat(2, 1)[:h, :w].astype(np.uint8)
    length[rng.random((h, w)) < 0.1] = 0
    length = np.ascontiguousarray(length.reshape(-1))
    color = (rng.integers(10, 18, 2 * n).astype(np.uint32) * 0x08020040 + rng.integers(0, 64, 2 * n).astype(np.uint32))
    mom = rng.lognormal(0, 2, 2 * n).clip(0, 6e4).astype(np.float16).view(np.uint16)
    depth, gbuf = host["depth"], host["gbuffer"]
    dev = [torch.from_numpy(a.view(np.uint8).copy()).cuda() for a in (depth, gbuf, length, color, mom)]
    for name in ("vlt_denoise_disocclusion_fix", "vlt_denoise_spatial_fallback"):
        oc, om = np.zeros(2 * n, np.uint32), np.zeros(2 * n, np.uint16)
        getattr(po.lib(), name.replace("vlt_", "vlto_"))(w, h, *[po.ptr(a) for a in (depth, gbuf, length, color, mom)],
                                                         po.ptr(oc), po.ptr(om))
        gc = torch.zeros(8 * n, dtype=torch.uint8, device="cuda")
        gm = torch.zeros(4 * n, dtype=torch.uint8, device="cuda")
        assert getattr(vg.lib(), name)(w, h, *[C.c_void_p(t.data_ptr()) for t in dev], C.c_void_p(gc.data_ptr()),
                                       C.c_void_p(gm.data_ptr()), None) == 0
        torch.cuda.synchronize()
        np.testing.assert_array_equal(gc.cpu().numpy().view(np.uint32), oc)
        np.testing.assert_array_equal(gm.cpu().numpy().view(np.uint16), om)
