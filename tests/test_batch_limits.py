"""The batched first pass's limit of 2^31 - 1 pixels per layer count. The
injected fault ends every call that passes the checks before its first CUDA
call."""
import ctypes

import pytest

import unblending_b200 as U
from unblending_b200 import synthetic as syn


@pytest.mark.parametrize("sizes,expect", [
    ([(3, 46340, 46340)], U.CUDA_ERROR),
    ([(3, 46340, 23170), (3, 46340, 23170)], U.CUDA_ERROR),
    ([(3, 46340, 46340), (2, 46340, 46340)], U.CUDA_ERROR),
    ([(3, 46340, 46340), (3, 46340, 3)], U.INVALID_ARGUMENT),
    ([(3, 46340, 46340), (2, 46340, 46340), (3, 46340, 46340)], U.INVALID_ARGUMENT),
    ([(2, 32768, 32768), (2, 32768, 32768)], U.INVALID_ARGUMENT),
    ([(2, 32768, 32768), (2, 32768, 32767)], U.CUDA_ERROR),
])
def test_pixels_per_layer_count(monkeypatch, sizes, expect):
    monkeypatch.setenv("UNBLENDING_FAULT", "launch")
    keep, jobs = [], (U.ImageJob * len(sizes))()
    for k, (layers, w, h) in enumerate(sizes):
        arr = syn.layer_array(syn.generate(4, 4, [0] * layers, (1.0, 2.0), seed=k).layers)
        keep.append(arr)
        jobs[k] = U.ImageJob(w, h, 16, ctypes.addressof(arr), layers, 16, None, None)
    rc = U.lib.unblending_unmix_batch_device(jobs, len(sizes), ctypes.byref(U.options()),
                                             ctypes.byref(U.solver_options()), None, None)
    assert rc == expect
