"""The admission estimate counts, beside a solve's matrices, the scratch of its
kernels: the counts of a split Gram and of An_ZtSn, the terms of the bit-plane
product and a worker thread's staging."""
import ctypes as C

import numpy as np
import pytest

from lakcluster_c_gb300 import abi, serve, solve

MB = 1 << 20


@pytest.mark.parametrize("rows,cols", [(100, 500), (900, 1920 * 64 - 8), (3000, 40000)])
def test_estimate_counts_the_scratch(rows, cols):
    lib = serve.bind(solve.load())
    w = np.zeros((rows, (cols + 15) // 16 * 2), np.uint8)
    p = solve.Problem([w], [w], gamma=0.05, packed_ncols=cols)
    est = lib.lakgb_bcc_footprint(C.byref(p.prob))
    rb, cdrop, P = abi.bsize(cols), cols // 8 + 1, abi.psize(cols)
    matrices = 2 * 2 * rows * rb + (16 + 6) * 2 * rows * rows + 33 * 2 * rows * abi.bsize(rows) + 24 * cols * cdrop
    counts, split = min(32 * MB, 2 * rows * 33 * P), min(256 * MB, 2 * rows * rows * P)
    assert est >= matrices + counts + split + 64 * MB + 48 * MB + 30784 * P
