"""The warm-start network's kernels at the edges of their tiles: pixel and
sample counts around 128, more tiles than an SM's six groups, every layer
count, and buffers that start on 4-byte boundaries, against the CPU
restatement (BF16 rounding at the same places, so the bounds are those of
tests/test_gpu_mlp.py)."""
import numpy as np
import pytest

from tests import mlp_reference as ref
from tests.test_mlp_reference import random_model
from unblending_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,L,offset", [((1, 1), 1, 0), ((127, 1), 2, 0), ((43, 3), 3, 1), ((16, 8), 8, 0),
                                           ((1000, 129), 5, 0), ((337, 339), 4, 3)])
def test_predictions(cuda, size, L, offset):
    import torch

    wl = syn.generate(*size, [0] * 2, (3.0, 9.0), seed=size[0])
    model = random_model(21 + L, L=L)
    img = torch.from_numpy(wl.image.reshape(-1)).cuda()
    out = torch.full((wl.pixels * 4 * L + 4,), -1.0, dtype=torch.float32, device="cuda")
    cuda.mlp_predict_device(model, *size, img.data_ptr(), out.data_ptr() + 4 * offset)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    want = ref.forward(model, ref.features(wl.image))[0][:, :4 * L]
    err = np.abs(got[offset:offset + want.size].reshape(want.shape) - want)
    assert err.max() < 1e-2 and err.mean() < 1e-3, (err.max(), err.mean())
    assert (got[:offset] == -1.0).all() and (got[offset + want.size:] == -1.0).all()


@pytest.mark.parametrize("count,L,offset", [(1, 1, 0), (127, 2, 0), (129, 8, 1), (256, 3, 0), (19000, 5, 2)])
def test_gradients(cuda, count, L, offset):
    import torch

    rng = np.random.default_rng(count)
    model = random_model(31 + L, L=L)
    feats = rng.uniform(0, 1, (count, 32)).astype(np.float32)
    feats[:, 30:] = 0
    targets = rng.uniform(0, 1, (count, 4 * L)).astype(np.float32)
    f = torch.zeros(count * 32 + 4, dtype=torch.float32, device="cuda")
    t = torch.zeros(count * 4 * L + 4, dtype=torch.float32, device="cuda")
    f[offset:offset + feats.size] = torch.from_numpy(feats.reshape(-1)).cuda()
    t[offset:offset + targets.size] = torch.from_numpy(targets.reshape(-1)).cuda()
    torch.cuda.synchronize()
    grad = cuda.mlp_loss_grad_device(model, count, f.data_ptr() + 4 * offset, t.data_ptr() + 4 * offset)
    loss, want = ref.loss_grad(model, feats, targets.astype(np.float64))
    assert abs(grad.loss - loss) <= 1e-3 * loss
    for name, g in want.items():
        used = 4 * L if name in ("w4", "b4") else len(g)
        got = grad.get(name)
        assert np.linalg.norm(got[:used] - g[:used]) < 2e-2 * max(np.linalg.norm(g[:used]), 1e-12), name
        assert (got[used:] == 0).all(), name
