"""The fold of a Gram split over blocks against the C oracle, bit for bit, around
the number of blocks it reads ahead (four) and with weights that are not
positive normal numbers: zero, negative, subnormal, far from one."""
import numpy as np
import pytest

import kernel_cases as kc
from lakcluster_c_gb300 import abi
from test_tc_counts_gpu import AUTO, SPLIT, _handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [3, 4, 5, 7, 8, 9, 11, 12, 13, 40])
def test_fold_equals_oracle(gpu_lib, P):
    rng = np.random.default_rng(P)
    MA, MZ = _handle(rng, 131, 1920 * P - 3, 0.8), _handle(rng, 67, 1920 * P - 3, 0.8)
    MZ.set_masks(mc_j=np.unpackbits(MA.mc_j)[: 1920 * P - 3])
    plain = abi.calc_A_ajdk(0.02 + 0.96 * rng.random(P))
    odd = plain.copy()
    odd[5 * P: 6 * P] = rng.permutation(np.resize([0.0, -1.75, 3e-310, 1e300, -0.0, 1.1], P))
    gpu_lib.lakgb_set_gram_impl(SPLIT)
    try:
        for w in (plain, odd, None):
            for t in (abi.TYPE_pm, abi.TYPE_00):
                args = (False, t, abi.SPACING_b, abi.SPACING_j, MA, MZ, w, None, None)
                want, got = kc.call_gram("oracle", *args), kc.call_gram("gpu", *args)
                assert np.array_equal(got.view(np.uint64), want.view(np.uint64)), (t, w is None)
        assert gpu_lib.lakgb_device_status() == 0
    finally:
        gpu_lib.lakgb_set_gram_impl(AUTO)
