"""The query selection at the edges of the miss scatter's words, warps and blocks (128 queries
per warp, 512 per block), on an empty grid, where every query is a miss, and on a filled one,
against the sequential loop. The scratch memory holds ones before the call: no bit of a
query beyond the last may be read as a miss."""
import ctypes as C

import numpy as np
import pytest

import violet_gb300 as vg
from oracle import pyoracle as po
from tests.test_gpu_hg_select import _check, _synth

pytestmark = pytest.mark.gpu

V = C.c_void_p


@pytest.mark.parametrize("filled", [0, 12])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 511, 512, 513, 1000, 4097])
def test_select_at_scatter_edges(n, filled):
    import torch

    lb, lib = 8, vg.lib()
    storage, queries = _synth(n + filled, lb, n, lambda rng, nb: np.full(nb, filled), 20, empty_frac=0.0)
    cnt = np.array([n], np.uint32)
    st_o, sel_o = storage.copy(), np.zeros(16 << lb, np.uint32)
    po.lib().vlto_hg_query_select(lb, n, po.ptr(queries), po.ptr(cnt), po.ptr(st_o), po.ptr(sel_o), 77)

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).cuda()

    q_g, c_g, st_g, sel_g = dev(queries), dev(cnt), dev(storage), dev(np.zeros(16 << lb, np.uint32))
    scratch = torch.full((lib.vlt_hg_select_scratch_bytes(lb, n),), 255, dtype=torch.uint8, device="cuda")
    assert lib.vlt_hg_query_select(lb, n, V(q_g.data_ptr()), V(c_g.data_ptr()), V(st_g.data_ptr()),
                                   V(sel_g.data_ptr()), 77, V(scratch.data_ptr()), None) == 0
    torch.cuda.synchronize()
    _check(st_g.cpu().numpy().view(np.uint32).reshape(-1, 4), sel_g.cpu().numpy().view(np.uint32), st_o, sel_o,
           "%d queries, %d cells per bucket" % (n, filled))
