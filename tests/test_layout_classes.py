"""The length classes of the device-made processing order, over every length that
a chunk's table can hold: longer payloads never in a later class, absent blocks
last, and no class wider than 4 bytes or 4.2 % of its lengths -- payloads reach
17408 bytes here and 65535 in the format."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "matter-compressor_b200", "csrc")


@pytest.fixture(scope="module")
def classes(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("cls")
    (d / "c.cpp").write_text('#include "mcb_format.h"\nextern "C" int cls(unsigned len) { return mcb::length_class(len); }\n'
                             'extern "C" int count() { return mcb::kLayoutClasses; }\n')
    subprocess.run([gxx, "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "c.so"), str(d / "c.cpp")], check=True)
    lib = C.CDLL(str(d / "c.so"))
    return np.array([lib.cls(n) for n in range(65536)]), lib


def test_order_and_width(classes):
    c, lib = classes
    assert c[0] == lib.count() - 1 and c[1:].max() < lib.count() - 1 and c.min() >= 0
    assert (np.diff(c[1:]) <= 0).all()
    for k in np.unique(c[1:]):
        n = np.flatnonzero(c == k)
        assert n[-1] - n[0] < 4 or n[-1] <= 1.042 * n[0], (k, n[0], n[-1])
    assert lib.cls(1 << 20) == c[65535]
