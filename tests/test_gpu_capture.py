"""Calls made while a stream captures a CUDA graph: a call that the capture
refuses leaves nothing behind for the next one, and a call on another stream
neither is refused nor ends the capture."""
import numpy as np
import pytest

from tests import mlp_reference as ref
from tests.test_gpu_batch_plans import equal_per_image, images
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


@pytest.mark.parametrize("mode", ["relaxed", "thread_local"])
def test_new_batch_while_another_stream_captures(cuda, mode):
    """A batch call with a new job list takes over the last plan's memory; the
    wait for that plan must not touch a capture on another stream of the same
    thread (relaxed) or of another thread (thread_local)."""
    import threading

    import torch

    lists = [images(seed) for seed in (3, 5)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    for jobs, _ in lists:
        cuda.unmix_batch_device(jobs, stream=streams[0].cuda_stream)
    x = torch.zeros(64, device="cuda")
    torch.cuda.synchronize()
    errors = []

    def call():
        try:
            cuda.unmix_batch_device(lists[0][0], stream=streams[0].cuda_stream)
        except Exception as e:
            errors.append(e)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[1], capture_error_mode=mode):
        x.add_(1)
        if mode == "relaxed":
            call()
        else:
            thread = threading.Thread(target=call)
            thread.start()
            thread.join()
    assert not errors
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 1).all()
    for _, keep in lists:
        assert equal_per_image(cuda, keep)
