"""The per-pass query compaction (its list order is unspecified) against the oracle, as
sets, at the edges of its 2,048-cell chunks, with an aligned and an unaligned selection
buffer and from an empty to a full selection."""
import ctypes as C

import numpy as np
import pytest

import violet_gb300 as vg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 4])
@pytest.mark.parametrize("share", [0.0, 0.002, 0.3, 1.0])
@pytest.mark.parametrize("log2_buckets", [4, 7, 8, 12])
def test_compact(log2_buckets, share, offset):
    import torch

    cells = 16 << log2_buckets
    rng = np.random.default_rng(cells + int(1000 * share))
    sel = np.where(rng.random(cells) < share, rng.integers(1, 1 << 31, cells) | 0x80000000, 0).astype(np.uint32)
    max_q = 1000
    qmask = (1 << int(max_q - 1).bit_length()) - 1
    buf = torch.zeros(4 * cells + 16, dtype=torch.uint8, device="cuda")
    buf[offset:offset + 4 * cells] = torch.from_numpy(sel.view(np.uint8)).cuda()
    idx, addr = (torch.zeros(cells, dtype=torch.int32, device="cuda") for _ in range(2))
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert vg.lib().vlt_hg_query_compact(log2_buckets, max_q, C.c_void_p(buf.data_ptr() + offset),
                                         C.c_void_p(idx.data_ptr()), C.c_void_p(addr.data_ptr()),
                                         C.c_void_p(count.data_ptr()), None) == 0
    torch.cuda.synchronize()
    want = np.nonzero(sel)[0]
    n = int(count.item())
    assert n == want.size
    a, i = addr[:n].cpu().numpy(), idx[:n].cpu().numpy().view(np.uint32)
    order = np.argsort(a)
    np.testing.assert_array_equal(a[order], want)
    got_bits = i[order] ^ sel[want]
    # the index is the low bits of the selection word, the same mask for every entry
    mask = np.bitwise_or.reduce(i) if n else 0
    assert (i[order] & ~np.uint32(0x7FFFFFFF)).max(initial=0) == 0
    assert n < 100 or mask in (qmask, 2 * qmask + 1)
    assert ((got_bits & np.uint32(mask)) == 0).all()
