"""Every kernel that a decode can launch has its code loaded when the library comes
up, so that no call pays for it at its first use: the kernels defined in the decode
sources against those that the preload functions name."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "matter-compressor_b200", "csrc")


def test_decode_kernels_are_preloaded():
    for name, fn in (("mcb_decode.cu", "preload_decode_kernels"), ("mcb_layout.cu", "preload_layout_kernels")):
        src = open(os.path.join(CSRC, name)).read()
        kernels = set(re.findall(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s+)?(k_\w+)", src))
        assert kernels
        i = src.index(f"cudaError_t {fn}() {{")
        body = src[i:src.index("\n}\n", i)]
        assert kernels <= set(re.findall(r"\bk_\w+", body)), name
        assert f"{fn}() != cudaSuccess" in open(os.path.join(CSRC, "mcb_runtime.cpp")).read()
