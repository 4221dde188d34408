"""Batched passes whose blocks stage a tile or permute their rows, in every shape of the
autotuner against the same views alone: the reference form's fast-history clamp over several
tiles, and the float forms' five a-trous iterations on images that hold whole footprints of
step 16, so that batched blocks take the path without edge tests."""
import pytest

import violet_gb300 as vg
from tests import test_gpu_batch as tb

pytestmark = pytest.mark.gpu


def fast_reference():
    p = vg.params_reference()
    p.fast_history_clamp = 1
    return p


def test_batch_tile_shapes(monkeypatch):
    specs = [
        (200, 75, "ref", fast_reference(), 1, 0),
        (67, 33, "ref", fast_reference(), 2, 1),
        (300, 260, "f32", tb.small_plain1(), 3, 0),
        (333, 257, "f16", tb.small_plain1(), 4, 0),
    ]
    monkeypatch.setattr(tb, "view_specs", lambda: specs)
    _, table = tb.run_pair(12, graphs=True, autotune=True)  # ten shapes, then the first two again
    assert any("fast_clamp" in name for name in table) and "dn_atrous" in table
