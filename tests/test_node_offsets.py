"""Offsets into the per-node arrays beyond 2^31 entries (715,827,883 nodes of three
values), compiled for the host from the header that the kernels use."""
import subprocess

import pytest

from bhut_gb300 import _build

SOURCE = r"""
#include <cstdio>
#include "tree.cuh"
int main()
{
    const int32_t ids[] = {0, 1, 715827882, 715827883, 1073741824, 2147483647};
    for (int width = 2; width <= 3; width++)
        for (int32_t id : ids)
            for (int axis = 0; axis < width; axis++)
                std::printf("%d %d %d %lld\n", width, id, axis, (long long)bhut::node_at(width, id, axis));
}
"""


def test_node_offsets_in_64_bits(tmp_path):
    try:
        nvcc = _build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    src, exe = tmp_path / "offsets.cu", tmp_path / "offsets"
    src.write_text(SOURCE)
    subprocess.run([nvcc, *_build.ARCH, "-std=c++17", "-I" + _build.CSRC, str(src), "-o", str(exe)],
                   check=True, capture_output=True, timeout=300)
    rows = [list(map(int, ln.split())) for ln in
            subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert len(rows) == 6 * 5
    for width, node, axis, at in rows:
        assert at == width * node + axis
