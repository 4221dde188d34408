"""The small-float codec of the R11G11B10 words: the branch-free encode on the host
against rounding in binary64, and the GPU's decode on every code."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import violet_gb300 as vg

HERE = os.path.dirname(os.path.abspath(__file__))


def test_encode_rounds_to_nearest_even(tmp_path):
    exe = str(tmp_path / "ufloat_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "native", "ufloat_check.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _values(mantissa_bits):
    c = np.arange(32 << mantissa_bits, dtype=np.int64)
    e, m = c >> mantissa_bits, c & ((1 << mantissa_bits) - 1)
    one = 1 << mantissa_bits
    v = np.where(e == 0, m * 2.0 ** (-14 - mantissa_bits), (one + m) * 2.0 ** (e - 15.0 - mantissa_bits))
    return np.where(e == 31, np.where(m == 0, np.inf, np.nan), v)


@pytest.mark.gpu
def test_decode_of_every_code():
    import torch

    # every code of each channel beside other codes of its neighbours; one image per word,
    # so that a sum is the decoded value
    r, b = _values(6), _values(5)
    c = np.arange(2048, dtype=np.uint32)
    g, z = (c * 37 + 11) % 2048, (c * 5 + 3) % 1024
    words = torch.from_numpy((c | (g << 11) | (z << 22)).view(np.int32)).cuda()
    out = torch.empty(2048, 8, dtype=torch.float64, device="cuda")
    for i in range(2048):
        rc = vg.lib().vlt_image_stats(C.c_void_p(words.data_ptr() + 4 * i), 2, None, 0, 1,
                                      C.c_void_p(out.data_ptr() + 64 * i), None)
        assert rc == 0
    got = out.cpu().numpy()[:, :3]
    np.testing.assert_array_equal(got, np.stack([r[c], r[g], b[z]], 1))
