"""The path kernels (tail, training paths) of one-level scenes keep 16 warps per
SM: what bounds them is the latency of their longest paths, and a branch that
only ray batches need, compiled into them, once took them from 128 registers a
thread to 168 and so to 12 warps."""
import ctypes as C
import os

import pytest

pytestmark = pytest.mark.gpu


def test_path_kernels_keep_their_warps(built):
    import foundation_gb300 as fg
    L = C.CDLL(os.path.join(os.path.dirname(os.path.abspath(__file__)), "_build", "libproduct_check.so"))
    with fg.Context(0):
        assert L.product_tail_blocks(0) >= 4
        assert L.product_training_blocks(0) >= 4
        assert L.product_tail_blocks(1) >= 3 and L.product_training_blocks(1) >= 3
