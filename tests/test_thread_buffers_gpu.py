"""What a host thread keeps between calls (streams, staging arenas, scope
chunks) goes to the next thread when it ends: batches of solves with fresh
worker threads leave the device memory level, and the buffers of ended threads
are bounded and can be freed."""
import os
import threading
import time

import numpy as np
import pytest

import kernel_cases as kc
from lakcluster_c_gb300 import abi

pytestmark = pytest.mark.gpu
SET_BYTES = 2 * (8 * 4 << 20) + (8 << 20) + 2 * 4 * (4 << 20)  # arenas, outputs, scope chunks


def test_batches_leave_the_device_memory_level(gpu_lib):
    import torch
    from lakcluster_c_gb300 import serve, solve as sv, synth
    insts = [synth.null_instance(300 + s, rows=(128, 256), cols=(512, 1024)) for s in range(8)]
    probs = [sv.Problem(i.A_bins, i.Z_bins, gamma=0.05) for i in insts]
    want = [p.solve() for p in probs]
    free = []
    for _ in range(6):
        got, _, _ = serve.solve_batched(probs, workers=8)
        assert got == want
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    # (one thread's arenas: 32 MB)
    assert free[1] - free[-1] < 32 << 20, [f >> 20 for f in free]


def test_idle_buffers_are_bounded_and_given_back(gpu_lib):
    import ctypes as C
    gpu_lib.lakgb_idle_buffers.argtypes, gpu_lib.lakgb_idle_buffers.restype = [C.c_int], C.c_longlong
    rng = np.random.default_rng(5)
    M = kc.mhandle(kc.random_bits(rng, (70, 3000)), np.ones(70, np.uint8), np.ones(70, np.uint8), np.ones(3000, np.uint8),
                   np.ones(3000, np.uint8))
    w = abi.calc_A_ajdk(0.05 + 0.9 * rng.random(abi.psize(3000)))
    want = kc.call_an_ajdk("oracle", abi.TYPE_pm, abi.SPACING_a, M, w).tobytes()
    before = len(os.listdir("/proc/self/task"))
    for _ in range(2):
        n, got = 20, []
        gate = threading.Barrier(n)

        def work():
            out = kc.call_an_ajdk("gpu", abi.TYPE_pm, abi.SPACING_a, M, w).tobytes()
            gate.wait()
            got.append(out)
        ts = [threading.Thread(target=work) for _ in range(n)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        end = time.monotonic() + 30  # (join returns while the thread still runs its exit handlers)
        while len(os.listdir("/proc/self/task")) > before and time.monotonic() < end:
            time.sleep(0.01)
        assert got == [want] * n
        held = gpu_lib.lakgb_idle_buffers(1)
        assert 0 < held <= 8 * SET_BYTES
        assert gpu_lib.lakgb_idle_buffers(0) == 0
