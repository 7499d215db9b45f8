"""The kernel choice of lakgb_gram_device does not depend on which launch of a
shape class came first: a large launch runs on the persistent tensor-core kernel
(no counts in scratch) after a small one of the same row and block buckets was
measured, also where its counts exceed the split's scratch; and a split that does
not fit takes the tensor kernel, not the popcount one."""
import ctypes as C

import pytest

from test_scratch_pool_gpu import AUTO, POPCOUNT, SPLIT, TENSOR, bind, device_gram, run

pytestmark = pytest.mark.gpu


def _scratch(lib, a, x, impl):
    """The output, and the scratch and launches of one call."""
    lib.lakgb_pool_high_water.argtypes, lib.lakgb_pool_high_water.restype = [C.c_int], C.c_longlong
    run(lib, a, x, TENSOR)
    base = lib.lakgb_pool_high_water(1)
    lib.lakgb_pool_high_water(1)
    base, n = lib.lakgb_pool_high_water(0), lib.lakgb_kernel_launches()
    out = run(lib, a, x, impl)
    return out, lib.lakgb_pool_high_water(0) - base, lib.lakgb_kernel_launches() - n


@pytest.mark.parametrize("first,later", [((520, 1030, 33), (1020, 2040, 40)), ((520, 1030, 33), (1020, 2040, 64)),
                                         ((130, 4200, 5), (250, 8100, 8))])
def test_large_member_after_a_small_one(gpu_lib, first, later):
    lib = bind(gpu_lib)
    lib.lakgb_gram_autotune_reset()
    a, x = device_gram(*first)
    assert run(lib, a, x, AUTO) == run(lib, a, x, POPCOUNT)
    a, x = device_gram(*later)
    want = run(lib, a, x, POPCOUNT)
    out, scratch, launches = _scratch(lib, a, x, AUTO)
    assert out == want
    assert scratch <= 32000 * later[2] and launches == 2  # the block tables
    assert lib.lakgb_device_status() == 0


def test_split_that_does_not_fit(gpu_lib):
    lib = bind(gpu_lib)
    a, x = device_gram(1020, 2040, 65)
    want = run(lib, a, x, POPCOUNT)
    out, scratch, launches = _scratch(lib, a, x, SPLIT)
    assert out == want and scratch <= 32000 * 65 and launches == 2
