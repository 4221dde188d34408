"""The branch-free arithmetic (correctly rounded reciprocal, quotient and roots), the word
codec and the selection on the GPU against the IEEE operations and the integer forms: the
reciprocal, the roots, the codec and the range tests over every operand, quotients over 2^32
random pairs and 3 * 2^30 next to the middle of two neighbours, selections over 2^28 draws."""
import ctypes as C
import os
import subprocess

import pytest

from violet_gb300 import build

pytestmark = pytest.mark.gpu

CHECKS = ["rcp", "roots", "div", "div_halfway", "ninths", "encode", "decode", "select", "see"]


@pytest.fixture(scope="module")
def checks(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("exact") / "libexact.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "exact_math_check.cu")
    subprocess.run([build._nvcc()] + build.NVCC_FLAGS + ["-I", build.CSRC, "-shared", "-o", out, src, "-lcudart"],
                   check=True)
    lib = C.CDLL(out)
    assert lib.exact_math_checks() == len(CHECKS)
    return lib


@pytest.mark.parametrize("name", CHECKS)
def test_exact_math(checks, name):
    out = (C.c_ulonglong * 4)()
    assert checks.exact_math_check(CHECKS.index(name), out) == 0
    assert out[0] >= 1 << 28
    assert out[1] == 0, "%s: %d of %d differ, one at %08x, %08x" % (name, out[1], out[0], out[2], out[3])
