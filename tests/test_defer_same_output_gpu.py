"""Two calls of a deferral scope that write the same output: the later one's
values stay, whatever way each output comes back (small ones through page-locked
memory, large ones directly)."""
import ctypes as C

import pytest

import kernel_cases as kc
import test_defer_gpu as td
from lakcluster_c_gb300 import abi
from lakcluster_c_gb300.abi import L_handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [(100, 20000), (20000, 100), (100, 90, 20000, 80), (8192, 8193)])
def test_last_call_stays(gpu_lib, rows):
    cases = [td._case(30 + i, n, 20, 1) for i, n in enumerate(rows)]
    out = abi.LHandle(max(rows))
    p = out.ptr
    gpu_lib.lakgb_defer_begin()
    ns = [td._call("gpu", abi.SPACING_a, abi.SPACING_a, c, p) for c in cases]
    gpu_lib.lakgb_defer_end()
    want = out.buf.copy()
    for c, n in zip(cases, ns):
        ref = C.POINTER(L_handle)()
        assert td._call("oracle", abi.SPACING_a, abi.SPACING_a, c, ref) == n
        want[:n] = kc._take(ref, n)
    assert out.buf.tobytes() == want.tobytes()
