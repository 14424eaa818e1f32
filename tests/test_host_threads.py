"""The launching side under several host threads: a launch must not depend on what another thread launches at the same time."""
import ctypes as C
import math
import threading

import pytest
import torch

from colinfer_b200 import _lib

pytestmark = pytest.mark.gpu


def _hammer(calls, n):
    """Runs every call n times in a thread of its own, all at once; the error codes other than 0 that came back."""
    codes, start = [], threading.Barrier(len(calls))

    def work(call):
        torch.cuda.set_device(0)
        start.wait()
        bad = [c for c in (call() for _ in range(n)) if c]
        codes.extend(bad)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    return codes


def test_threads_with_different_row_counts_do_not_disturb_each_other():
    """3 rows take clusters of eight CTAs, 20 rows clusters of four with twice the shared memory each: the limit that the larger
    launch needs must stand whatever the smaller one does (ctypes lets go of the interpreter during a call)."""
    V = 151936
    L = _lib.lib()
    x = torch.randn(20, V, device="cuda")
    keep = [torch.ones(20, device="cuda"), torch.full((20,), 20, dtype=torch.int32, device="cuda"), torch.full((20,), 0.9, device="cuda"),
            torch.full((20,), -math.inf, device="cuda"), torch.full((20,), 0.5, device="cuda")]
    p = _lib.SamplerParamsC()
    p.temperature, p.top_k, p.top_p, p.log_min_p = (t.data_ptr() for t in keep[:4])
    streams = [torch.cuda.Stream() for _ in range(4)]
    outs = [torch.zeros(20, dtype=torch.int64, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()

    def call(i, rows):
        return lambda: L.colinfer_sample(x.data_ptr(), _lib.F32, None, 0, 0, C.byref(p), None, 0, keep[4].data_ptr(), outs[i].data_ptr(), None, None,
                                         rows, 1, V, 0, streams[i].cuda_stream)

    assert _hammer([call(0, 3), call(1, 20), call(2, 3), call(3, 20)], 1000) == []
    assert torch.equal(outs[0][:3], outs[1][:3]) and torch.equal(outs[1], outs[3])


@pytest.mark.parametrize("fmt", ["bf16", "nvfp4"])
def test_threads_with_different_hidden_sizes_do_not_disturb_each_other(fmt):
    """Rescoring of hidden sizes whose activations take more than the default 48 KB of shared memory, 50 and 96 KB."""
    L = _lib.lib()
    sizes, rows_w = (25_600, 49_152), 8
    cand = torch.arange(rows_w, device="cuda")[None].contiguous()
    xs = [torch.randn(1, K, device="cuda").bfloat16() for K in sizes]
    ws = [torch.randn(rows_w, K, device="cuda").bfloat16() for K in sizes]
    sf = torch.full((rows_w, sizes[1] // 16), 0x38, dtype=torch.uint8, device="cuda")          # E4M3 1.0
    streams = [torch.cuda.Stream() for _ in range(4)]
    outs = [torch.zeros(1, rows_w, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()

    def call(i):
        x, w, K = xs[i % 2], ws[i % 2], sizes[i % 2]
        if fmt == "bf16":
            return lambda: L.colinfer_rescore_bf16(x.data_ptr(), w.data_ptr(), cand.data_ptr(), outs[i].data_ptr(), 1, K, rows_w, rows_w,
                                                   streams[i].cuda_stream)
        return lambda: L.colinfer_rescore_nvfp4(x.data_ptr(), w.data_ptr(), sf.data_ptr(), 1.0, cand.data_ptr(), outs[i].data_ptr(), 1, K, rows_w, rows_w,
                                                streams[i].cuda_stream)

    assert _hammer([call(i) for i in range(4)], 1000) == []
    assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[3])
