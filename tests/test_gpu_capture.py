"""Calls made while a stream captures a CUDA graph: a call that the capture
refuses leaves nothing behind for the next one."""
import numpy as np
import pytest

from tests import mlp_reference as ref
from tests.test_mlp_reference import random_model
from unblending_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def test_network_of_a_refused_call_is_uploaded_by_the_next(cuda):
    """The prediction waits for its result, which a capturing stream refuses;
    the copy of its network never ran, so the next call has to make it. The
    bound is that of tests/test_gpu_mlp.py; the other network is off by 0.05."""
    import torch

    wl = syn.workload("rgb1024_l5", 23, 13)
    img = torch.from_numpy(wl.image.reshape(-1)).cuda()
    out = torch.empty(wl.pixels * 20, dtype=torch.float32, device="cuda")
    first, second = random_model(11, L=5), random_model(12, L=5)
    torch.cuda.synchronize()

    def predict(model, stream=None):
        cuda.mlp_predict_device(model, wl.width, wl.height, img.data_ptr(), out.data_ptr(), stream=stream)

    predict(first)
    stream = torch.cuda.Stream()
    with pytest.raises(Exception):   # the refused call ends the capture, too
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream, capture_error_mode="relaxed"):
            with pytest.raises(cuda.ExecutionError):
                predict(second, stream.cuda_stream)
    torch.cuda.synchronize()
    predict(second)
    torch.cuda.synchronize()
    want = ref.forward(second, ref.features(wl.image))[0][:, :20]
    err = np.abs(out.cpu().numpy().reshape(-1, 20) - want)
    assert err.max() < 1e-2 and err.mean() < 1e-3, (err.max(), err.mean())
