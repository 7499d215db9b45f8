"""The tensor-core Gram over very many blocks, whose tables estimate the sums so far
from some of the earlier blocks only: the popcount kernel's outputs."""
import pytest

from test_scratch_pool_gpu import POPCOUNT, TENSOR, bind, device_gram, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nA,nZ,P", [(40, 33, 256), (40, 33, 257), (130, 115, 1500)])
def test_many_blocks_equal_popcount(gpu_lib, nA, nZ, P):
    lib = bind(gpu_lib)
    g = device_gram(nA, nZ, P)
    assert run(lib, *g, TENSOR) == run(lib, *g, POPCOUNT)
    assert lib.lakgb_device_status() == 0

