"""AtTYn_vv where its counts stay in the accumulators over many 1920-column
blocks (large counts, a partial last block), narrow and wide tiles, against the
C oracle, bit for bit."""
import pytest

import test_tc_counts_gpu as tc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nA,nY,m,nt", [(10, 9, 131072, 1), (130, 17, 1920 * 12 + 1, 2), (1300, 700, 1920 * 9 - 1, 1)])
def test_many_blocks_equal_oracle(gpu_lib, nA, nY, m, nt):
    tc.test_snp_product_equals_oracle(gpu_lib, nA, nY, m, nt, 0.9)
