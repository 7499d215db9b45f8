"""The kernel that lakgb_gram_device takes above 60 output tiles, by its scratch
(counts of a split launch or block tables of the persistent one), on both sides of
the costs: narrow last tile columns, few live rows, one to many blocks; and its
outputs against the popcount kernel."""
import pytest

from test_gram_dispatch_gpu import _scratch
from test_scratch_pool_gpu import AUTO, POPCOUNT, bind, device_gram, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nA,nZ,P,split", [(6454, 113, 2, True), (300, 6454, 1, True), (12000, 1, 9, True), (12000, 60, 2, True),
                                           (3000, 230, 33, True), (6454, 300, 9, False), (113, 12000, 9, False),
                                           (230, 12000, 4, False), (1, 30000, 33, False), (900, 1000, 69, False)])
def test_choice_by_cost(gpu_lib, nA, nZ, P, split):
    lib = bind(gpu_lib)
    lib.lakgb_gram_autotune_reset()
    a, x = device_gram(nA, nZ, P)
    want = run(lib, a, x, POPCOUNT)
    out, scratch, launches = _scratch(lib, a, x, AUTO)
    assert out == want
    assert launches == 2
    counts, tables = 2 * nA * nZ * P, 30784 * P
    assert abs(scratch - (counts if split else tables)) < abs(scratch - (tables if split else counts))
    assert lib.lakgb_device_status() == 0
