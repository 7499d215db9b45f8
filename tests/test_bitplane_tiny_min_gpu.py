"""wrap_At_T_YnWt_S_Zn_ww__run with a minimum so small that the quotients by mlt
are near the smallest doubles (value planes of zeros: the minimum's term alone),
against the C oracle, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import kernel_cases as kc
from test_bitplane_units_gpu import _call, _handles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,mlt", [(-1.74e-307, 2.4661079740013e-15), (-9.81e-303, 2.84749366366689e-11),
                                    (3.06e-299, 2.1993931447575e-17), (-5e-324, 7.0), (0.0, 0.3), (3e-38, 2.9e-20)])
def test_tiny_minimum_equals_oracle(gpu_lib, lo, mlt):
    snps, ny, nw, B, nt = 300, 140, 9, 16, 2
    h = _handles(np.random.default_rng(5), snps, ny, nw, B, nt, 0.9, mlt)
    h["X"].s.min_d = lo
    h["X"].wX[1:] = 0
    want = _call(kc.load_backend("oracle").lako_At_T_YnWt_S_Zn_ww, h, snps, nt, ())
    got = _call(gpu_lib.wrap_At_T_YnWt_S_Zn_ww__run, h, snps, nt, (C.byref(C.c_int(0)), None, None))
    assert gpu_lib.lakgb_device_status() == 0
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
