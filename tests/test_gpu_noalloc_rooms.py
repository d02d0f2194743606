"""The allocation-free pass where its array's room for the lanes' records is
one block short of what the re-solve takes on lanes, and just enough: the
results are those of the allocating call."""
import numpy as np
import pytest

from unblending_b200 import synthetic as syn

pytestmark = pytest.mark.gpu

ARRAY = 32 << 20   # bytes for the miss lists (8 a pixel) and the records


@pytest.mark.parametrize("modes,blocks", [([0, 6], 74), ([0, 6, 7], 65), ([0, 1, 2, 3, 6, 9, 7], 37)])
@pytest.mark.parametrize("short", [0, 1])
def test_resolve_at_the_edge_of_its_room(cuda, modes, blocks, short):
    import torch

    L = len(modes)
    record = (16 * L + 2) * 128 * 32   # bytes a block
    w = 256
    h = (ARRAY - (blocks - short) * record) // 8 // w
    tile = syn.generate(w, 256, modes, (20.0, 200.0), seed=3)
    img = torch.from_numpy(np.ascontiguousarray(np.tile(tile.image, (-(-h // 256), 1, 1))[:h])).cuda()
    outs = [torch.full((4 * L * w * h,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
    status = [torch.full((w * h,), -1, dtype=torch.int32, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    so = cuda.solver_options(precision=cuda.PRECISION_FP32)
    args = (w, h, img.data_ptr(), tile.layers)
    stream = torch.cuda.current_stream().cuda_stream
    cuda.unmix_device(*args, outs[0].data_ptr(), solver=so, d_status=status[0].data_ptr(), stream=stream)
    cuda.unmix_device_noalloc(*args, outs[1].data_ptr(), solver=so, d_status=status[1].data_ptr(), stream=stream)
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1]) and torch.equal(status[0], status[1])
