"""Compile-time knobs of the kernels, checked by compiling the device headers
(no GPU): the values a build may choose compile and take effect."""
import os
import subprocess

import pytest

import differentiablepointrendering_b200.build as B

CSRC = os.path.join(os.path.dirname(B.__file__), "csrc")


def _compile(tmp_path, body, *flags):
    src = tmp_path / "knob.cu"
    src.write_text('#include "kernels.h"\n#include "trace.cuh"\n' + body)
    return subprocess.run([B.nvcc(), *B.ARCH, "-std=c++17", "-I", CSRC, *flags, "-c", str(src), "-o",
                           str(tmp_path / "knob.o")], capture_output=True, text=True)


@pytest.mark.parametrize("half,size", [(0, 64), (1, 32)])
def test_half_nodes_selects_the_traversal_nodes(tmp_path, half, size):
    r = _compile(tmp_path, f'static_assert(sizeof(pale::TravNode) == {size}, "node");\n', f"-DPALE_HALF_NODES={half}")
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("knob,good,bad", [("PALE_LOOKUP_HEAVY", (32, 96, 512), (16, 100, 4096)),
                                           ("PALE_LOOKUP_LANES", (4, 16), (2, 12, 32))])
def test_lookup_knobs_are_guarded(tmp_path, knob, good, bad):
    # other values would write past the group's shared memory or leave parts of it unwritten
    for v in good:
        r = _compile(tmp_path, "", f"-D{knob}={v}")
        assert r.returncode == 0, r.stderr
    for v in bad:
        r = _compile(tmp_path, "", f"-D{knob}={v}")
        assert r.returncode != 0 and knob in r.stderr, v
