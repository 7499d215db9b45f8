"""The device scratch of lakgb_gram_device: kept over a synchronisation up to a
bound, given back on request, and the graph's own where the launch is captured
(the captured launch, replayed on new rows, gives the plain launch's outputs)."""
import ctypes as C

import pytest

from lakcluster_c_gb300 import abi
from lakcluster_c_gb300.gram_pass import GramArgs

pytestmark = pytest.mark.gpu
AUTO, TENSOR, SPLIT, POPCOUNT = 2, 1, 3, 0
KEPT = 64 << 20


def bind(lib):
    lib.lakgb_gram_device.argtypes, lib.lakgb_gram_device.restype = [C.POINTER(GramArgs)], C.c_int
    lib.lakgb_idle_buffers.argtypes, lib.lakgb_idle_buffers.restype = [C.c_int], C.c_longlong
    return lib


def device_gram(nA, nZ, P, seed=1):
    """The arguments of a Gram of random rows and weights, and its tensors."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = dict(w=[torch.randint(0, 256, (n, 240 * P), generator=g, device="cuda", dtype=torch.uint8) for n in (nA, nZ)],
             mask=torch.randint(0, 256, (240 * P,), generator=g, device="cuda", dtype=torch.uint8),
             D=1.0 + torch.rand(P, generator=g, device="cuda", dtype=torch.float64),
             lf=[torch.randn(n, generator=g, device="cuda", dtype=torch.float64) for n in (nA, nZ)],
             idx=torch.arange(max(nA, nZ), device="cuda", dtype=torch.int32),
             out=torch.full((nA * nZ,), float("nan"), device="cuda", dtype=torch.float64))
    a = GramArgs()
    i = x["idx"].data_ptr()
    a.wA, a.a_rowb, a.nA, a.a_row_bytes = x["w"][0].data_ptr(), i, nA, 240 * P
    a.wZ, a.z_rowb, a.nZ, a.z_row_bytes = x["w"][1].data_ptr(), i, nZ, 240 * P
    a.mask, a.P, a.D, a.type_flag = x["mask"].data_ptr(), P, x["D"].data_ptr(), abi.TYPE_pm
    a.a0d1, a.a2d1, a.lfA, a.lfZ = 3.5, -1.25, x["lf"][0].data_ptr(), x["lf"][1].data_ptr()
    a.out_r = a.out_c = a.out_r2 = a.out_c2 = i
    a.out_stride, a.out = nA, x["out"].data_ptr()
    torch.cuda.synchronize()  # (the tensors are torch's stream's, the launches another's)
    return a, x


def run(lib, a, x, impl):
    import torch
    before = lib.lakgb_gram_impl()
    lib.lakgb_set_gram_impl(impl)
    try:
        x["out"].fill_(float("nan"))
        torch.cuda.synchronize()
        assert lib.lakgb_gram_device(C.byref(a)) == 0
        torch.cuda.synchronize()
    finally:
        lib.lakgb_set_gram_impl(before)
    return x["out"].cpu().numpy().tobytes()


@pytest.mark.parametrize("impl", [TENSOR, SPLIT])
def test_scratch_is_kept_bounded_and_given_back(gpu_lib, impl):
    lib = bind(gpu_lib)
    lib.lakgb_idle_buffers(1)
    small, big = device_gram(300, 500, 9), device_gram(900, 900, 130)
    want = [run(lib, *g, POPCOUNT) for g in (small, big)]
    assert lib.lakgb_idle_buffers(1) == 0
    assert run(lib, *small, impl) == want[0]
    scratch = 300 * 500 * 9 * 2 if impl == SPLIT else 9 * 1921 * 8
    assert lib.lakgb_idle_buffers(0) >= scratch
    assert run(lib, *big, impl) == want[1]  # 210 MB as a split launch
    assert lib.lakgb_idle_buffers(0) <= KEPT + (32 << 20)
    lib.lakgb_idle_buffers(1)
    assert lib.lakgb_idle_buffers(0) == 0
    assert run(lib, *small, impl) == want[0]
    assert lib.lakgb_device_status() == 0


@pytest.mark.parametrize("impl", [TENSOR, SPLIT])
@pytest.mark.parametrize("nA,nZ,P", [(130, 70, 1), (300, 260, 9)])
def test_captured_launch_on_new_rows(gpu_lib, impl, nA, nZ, P):
    import torch
    lib = bind(gpu_lib)
    a, x = device_gram(nA, nZ, P)
    run(lib, a, x, impl)  # module load and attributes, before the capture
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    a.stream = s.cuda_stream
    lib.lakgb_set_gram_impl(impl)
    try:
        with torch.cuda.stream(s):
            with torch.cuda.graph(graph, stream=s):
                assert lib.lakgb_gram_device(C.byref(a)) == 0
    finally:
        lib.lakgb_set_gram_impl(AUTO)
    a.stream = None
    for seed in (2, 3):
        _, y = device_gram(nA, nZ, P, seed)
        for k in (0, 1):
            x["w"][k].copy_(y["w"][k])
        x["D"].copy_(y["D"])
        want = run(lib, a, x, POPCOUNT)
        x["out"].fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert x["out"].cpu().numpy().tobytes() == want
    assert lib.lakgb_device_status() == 0
