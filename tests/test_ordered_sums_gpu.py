"""The ordered sums (AnZt_S_WnYt, AtTYn____WtSZn) and An_ajdk against the C
oracle, bit for bit, at the edges of their tiles: 32 rows, 36 terms (and the
tiles fetched ahead), two rows per warp, four blocks ahead, weights of either
sign, zero, and far from one."""
import ctypes as C

import numpy as np
import pytest

import kernel_cases as kc
import test_defer_gpu as td
from lakcluster_c_gb300 import abi
from lakcluster_c_gb300.abi import L_handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,terms,ns", [(1, 1, 1), (31, 35, 1), (32, 36, 2), (33, 37, 1), (64, 72, 3), (65, 73, 1),
                                           (200, 109, 2), (5000, 3, 1), (40, 2000, 1)])
def test_sums_equal_oracle(gpu_lib, rows, terms, ns):
    rng = np.random.default_rng(rows + 7 * terms)
    ones = lambda n: np.ones(n, np.uint8)  # noqa: E731
    full = lambda n, m: kc.mhandle(kc.random_bits(rng, (n, m)), ones(n), ones(n), ones(m), ones(m))  # noqa: E731
    An, Zn, St = full(rows, 32), full(terms, 32), full(ns, terms)
    wide = lambda s: rng.standard_normal(s) * 10.0 ** rng.integers(-12, 12, s)  # noqa: E731
    c = (An, Zn, St, abi.LHandle.from_matrix(wide((rows, terms))), abi.LHandle.from_matrix(wide((rows, terms))))
    At, Zt, Yt, Tt, S2 = full(rows, 48), full(rows, 40), full(terms, 48), full(ns, 48), full(ns, 40)
    Wt = full(terms, 40)
    w = abi.calc_A_ajdk(0.05 + 0.9 * rng.random(abi.psize(terms)))
    LA, LZ = td._l3(rng, (rows, terms, ns)), td._l3(rng, (rows, terms, ns))

    def products(backend, out):
        args = (abi.SPACING_a, abi.SPACING_j, At.ptr, Tt.ptr, Yt.ptr, Wt.ptr, S2.ptr, Zt.ptr,
                w.ctypes.data_as(C.POINTER(C.c_double)), LA.ptr, LZ.ptr, C.byref(out))
        lib = kc.load_backend(backend)
        if backend == "oracle":
            return lib.lako_AtTYn____WtSZn_vv(*args)
        return lib.wrap_AtTYn____WtSZn_vv__run(*kc._thread_args(), *args)

    for call in (lambda b, o: td._call(b, abi.SPACING_a, abi.SPACING_b, c, o), products):
        got, want = C.POINTER(L_handle)(), C.POINTER(L_handle)()
        assert call("gpu", got) == call("oracle", want) == rows * ns
        assert kc._take(got, rows * ns).tobytes() == kc._take(want, rows * ns).tobytes()


@pytest.mark.parametrize("rows,cols", [(1, 1), (2, 1920), (3, 1921), (31, 7680), (33, 9600), (300, 11521)])
@pytest.mark.parametrize("keep", [1.0, 0.7])
def test_row_terms_equal_oracle(gpu_lib, rows, cols, keep):
    rng = np.random.default_rng(rows + cols)
    mr_j = (rng.random(rows) < keep).astype(np.uint8) | (np.arange(rows) == 0)
    mc_j = (rng.random(cols) < keep).astype(np.uint8)
    M = kc.mhandle(kc.random_bits(rng, (rows, cols)), np.ones(rows, np.uint8), mr_j.astype(np.uint8),
                   np.ones(cols, np.uint8), mc_j)
    P = abi.psize(cols)
    odd = np.concatenate([rng.standard_normal(5 * P), np.zeros(2 * P), 1e-310 * rng.random(P), 1e300 * rng.random(P),
                          rng.random(6 * P)])
    for w in (abi.calc_A_ajdk(0.02 + 0.96 * rng.random(P)), odd):
        for t in (abi.TYPE_pm, abi.TYPE_00):
            got, want = (kc.call_an_ajdk(b, t, abi.SPACING_a, M, w) for b in ("gpu", "oracle"))
            assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
