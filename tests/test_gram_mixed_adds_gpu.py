"""The tensor-core Gram's integer adds and fixed-point row terms against the
popcount kernel (which the oracle tests cover), bit for bit: tile edges (128 A
rows, 112 Z rows, 28 per warp), sums that cross binades, exponents and counts
outside the integer table, and row terms with and without a fixed-point form."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

WEIGHTS = {
    "random": lambda torch, g, P: 0.5 + torch.rand(P, generator=g, dtype=torch.float64),
    "one": lambda torch, g, P: torch.ones(P, dtype=torch.float64),
    "growing": lambda torch, g, P: 1.3 * 2.0 ** torch.arange(P, dtype=torch.float64),
    "falling": lambda torch, g, P: 1.7 * 2.0 ** (-7.0 * torch.arange(P, dtype=torch.float64)),
    "signed": lambda torch, g, P: torch.randn(P, generator=g, dtype=torch.float64),
    "tiny": lambda torch, g, P: 1e-300 * torch.rand(P, generator=g, dtype=torch.float64),
    "zeros": lambda torch, g, P: torch.where(torch.arange(P) % 2 == 0, 0.0, 0.7).double(),
    "huge": lambda torch, g, P: 1e305 * torch.ones(P, dtype=torch.float64),
}
TERMS = {
    "none": None,
    "like": lambda torch, g, n: 400.0 * torch.randn(n, generator=g, dtype=torch.float64),
    "wide": lambda torch, g, n: torch.randn(n, generator=g, dtype=torch.float64) * 10.0 ** torch.arange(-9, 9).double().repeat(n // 18 + 1)[:n],
    "zeros": lambda torch, g, n: torch.zeros(n, dtype=torch.float64) * torch.where(torch.arange(n) % 3 == 0, -1.0, 1.0),
    "whole": lambda torch, g, n: torch.randint(-3000, 3000, (n,), generator=g).double(),
    "infinite": lambda torch, g, n: torch.where(torch.arange(n) % 50 == 7, float("inf"), 100.0).double(),
}


@pytest.mark.parametrize("nA,nZ,P,weights,terms,kind,sym", [
    (1, 1, 1, "random", "like", 1, 0), (127, 111, 2, "random", "like", 1, 0), (128, 112, 40, "random", "like", 1, 0),
    (129, 113, 3, "one", "whole", 1, 0), (300, 28, 9, "one", "none", 2, 0), (97, 141, 20, "growing", "like", 1, 0),
    (130, 29, 20, "falling", "wide", 1, 0), (260, 260, 12, "signed", "zeros", 1, 1), (140, 300, 6, "tiny", "wide", 1, 0),
    (300, 300, 17, "random", "like", 1, 1), (33, 500, 9, "zeros", "infinite", 2, 0), (129, 120, 5, "huge", "like", 1, 0),
    (225, 225, 33, "random", "none", 2, 1), (250, 230, 11, "random", "like", 2, 0)])
def test_tensor_gram_equals_popcount(gpu_lib, nA, nZ, P, weights, terms, kind, sym):
    torch = pytest.importorskip("torch")
    from lakcluster_c_gb300 import abi, gram_pass
    g = torch.Generator().manual_seed(nA + 7 * nZ + 31 * P)
    dev = "cuda"
    nb = 240 * P
    A = torch.randint(0, 256, (nA, nb), generator=g, dtype=torch.uint8)
    Z = A if sym else torch.randint(0, 256, (nZ, nb), generator=g, dtype=torch.uint8)
    if not sym:
        Z[:: 5] = A[torch.arange(0, nZ, 5) % nA]  # equal rows: zero sums
        Z[1:: 9] &= 3                             # few set bits
    mask = torch.randint(0, 256, (nb,), generator=g, dtype=torch.uint8) | 0x55
    D = WEIGHTS[weights](torch, g, P)
    t = TERMS[terms]
    lfA = t(torch, g, nA) if t else None
    lfZ = (lfA if sym else t(torch, g, nZ)) if t else None
    to = lambda x: x.to(dev) if x is not None else None  # noqa: E731
    A, Z, mask, D, lfA, lfZ = map(to, (A, Z, mask, D, lfA, lfZ))
    idx = torch.arange(max(nA, nZ), dtype=torch.int32, device=dev)
    a = gram_pass.GramArgs()
    a.wA, a.a_rowb, a.nA, a.a_row_bytes = A.data_ptr(), idx.data_ptr(), nA, nb
    a.wZ, a.z_rowb, a.nZ, a.z_row_bytes = Z.data_ptr(), idx.data_ptr(), nZ, nb
    a.mask, a.P, a.D = mask.data_ptr(), P, D.data_ptr()
    a.type_flag = abi.TYPE_pm if kind == 1 else abi.TYPE_00
    a.a0d1, a.a2d1 = 1000.3 * float(D.sum()), 77.1
    if t:
        a.lfA, a.lfZ = lfA.data_ptr(), lfZ.data_ptr()
    a.out_r = a.out_c2 = a.out_c = a.out_r2 = idx.data_ptr()
    a.out_stride, a.symmetric = nA, sym
    out = [torch.full((nA * nZ,), 3.25, dtype=torch.float64, device=dev) for _ in range(2)]
    gpu_lib.lakgb_gram_device.argtypes = [C.POINTER(gram_pass.GramArgs)]
    gpu_lib.lakgb_gram_device.restype = C.c_int
    before = gpu_lib.lakgb_gram_impl()
    try:
        for impl in (0, 1):  # popcount, tensor cores
            gpu_lib.lakgb_set_gram_impl(impl)
            a.out, a.stream = out[impl].data_ptr(), torch.cuda.current_stream().cuda_stream
            assert gpu_lib.lakgb_gram_device(C.byref(a)) == 0
            torch.cuda.synchronize()
            assert gpu_lib.lakgb_device_status() == 0
    finally:
        gpu_lib.lakgb_set_gram_impl(before)
    finite = [torch.isfinite(o) for o in out]
    assert torch.equal(out[0].isnan(), out[1].isnan())
    same = out[0].view(torch.int64) == out[1].view(torch.int64)
    assert bool((same | out[0].isnan()).all()), f"{int((~(same | out[0].isnan())).sum())} of {same.numel()} differ ({int((~finite[0]).sum())} not finite)"
