"""bench.py's count of the kernels in a training step: one launch for the weight
gradients of all layers but the first, and one Adam, where the partials of all
layers fit; otherwise one each per layer.  (Counts as a profiler sees them.)"""
import os
import sys

import pytest

from conftest import ROOT

sys.path.insert(0, ROOT)
import bench  # noqa: E402


@pytest.mark.parametrize("layers,batch,launches", [(1, 65536, 6), (2, 65536, 8), (3, 65536, 12), (5, 65536, 16),
                                                   (8, 65536, 22), (8, 4096, 8), (16, 8192, 8), (16, 16384, 38)])
def test_count(layers, batch, launches):
    assert bench.mlp_launches(layers, batch) == launches
