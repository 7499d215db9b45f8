"""lakgb_xcalc_noalloc takes the caller's column offsets as they are: the same
matrix addressed from any of its elements, offsets of -1 and below included,
gives the same planes and scalars."""
import ctypes as C

import numpy as np
import pytest

import test_zz_no_alloc as na
from lakcluster_c_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("base", [1, 7, 40 * 300 - 1])
@pytest.mark.parametrize("wide", [True, False])
def test_offsets_below_the_base_pointer(gpu_lib, base, wide):
    import torch
    lib = na._bind(gpu_lib)
    rows, cols, B = 300, 40, 32
    brows = abi.bsize(rows) if wide else 40
    lf = torch.from_numpy(np.random.default_rng(base).standard_normal(rows * cols) * 9.0).cuda()
    r = torch.arange(rows, device="cuda")
    c = torch.arange(cols, device="cuda") * rows
    got = []
    for shift in (0, base):
        k = c - shift
        planes = torch.full(((B + 1) * cols, brows), 0x5A, dtype=torch.uint8, device="cuda")
        out = (C.c_double * 3)()
        torch.cuda.synchronize()
        a = na.NoAllocArgs(lf.data_ptr() + 8 * shift, r.data_ptr(), rows, r.data_ptr(), rows, k.data_ptr(), cols, None, B,
                           1 << B, brows, planes.data_ptr(), C.cast(out, C.POINTER(C.c_double)), None)
        assert lib.lakgb_xcalc_noalloc(C.byref(a)) == 0
        got.append((planes.cpu().numpy().tobytes(), tuple(out)))
    assert got[0] == got[1]
