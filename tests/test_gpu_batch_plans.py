"""The batched first pass keeps the last call's captured plan: calls that
differ only in an option of the call must not replay it."""
import pytest

from unblending_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def images(seed, comp=syn.SOURCE_OVER):
    """Two images of three and four layers: jobs, and per job the image, its device copy and the output."""
    import torch

    jobs, keep = [], []
    for k, (size, modes) in enumerate((((40, 30), [0, 1, 2]), ((24, 50), [0, 2, 1, 3]))):
        wl = syn.generate(*size, modes, (5.0, 20.0), seed=seed + k, comp=comp)
        img = torch.from_numpy(wl.image.reshape(-1)).cuda()
        out = torch.full((4 * len(modes) * wl.pixels,), float("nan"), dtype=torch.float64, device="cuda")
        jobs.append(dict(width=wl.width, height=wl.height, d_image=img.data_ptr(), layers=wl.layers,
                         d_output=out.data_ptr()))
        keep.append((wl, img, out))
    torch.cuda.synchronize()
    return jobs, keep


def equal_per_image(cuda, keep, opaque=True):
    """Whether the outputs are those of the single-image calls; clears them."""
    import torch

    torch.cuda.synchronize()
    for wl, img, out in keep:
        ref = torch.empty_like(out)
        cuda.unmix_device(wl.width, wl.height, img.data_ptr(), wl.layers, ref.data_ptr(), opaque=opaque)
        torch.cuda.synchronize()
        if not torch.equal(out, ref):
            return False
        out.fill_(float("nan"))
    torch.cuda.synchronize()
    return True


@pytest.mark.parametrize("comp", [syn.PLUS, syn.SOURCE_OVER])
def test_opaque_background_taken_from_each_call(cuda, comp):
    jobs, keep = images(3, comp)
    for opaque in (True, False, True):
        cuda.unmix_batch_device(jobs, opaque=opaque)
        assert equal_per_image(cuda, keep, opaque), opaque


# Two groups: each has half of the blocks (444 on 148 SMs up to five layers, 296 from six), 128 pixels a block.
@pytest.mark.parametrize("layers", [(2, 3), (3, 6)])
@pytest.mark.parametrize("pixels", [(1, 300), (444, 445), (296, 297), (222 * 128, 148 * 128), (222 * 128 + 1, 148 * 128 + 1)])
@pytest.mark.parametrize("precision", [1, 0])
def test_groups_at_the_edges_of_their_share(cuda, layers, pixels, precision):
    import torch

    so = cuda.solver_options(precision=precision)
    jobs, keep = [], []
    for L, n in zip(layers, pixels):
        wl = syn.generate(n, 1, [0, 1, 2, 6, 3, 9][:L], (3.0, 9.0), seed=n)
        img = torch.from_numpy(wl.image.reshape(-1)).cuda()
        out, ref = (torch.full((4 * L * n,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
        status, ref_status = (torch.full((n,), -1, dtype=torch.int32, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        cuda.unmix_device(n, 1, img.data_ptr(), wl.layers, ref.data_ptr(), solver=so, d_status=ref_status.data_ptr())
        jobs.append(dict(width=n, height=1, d_image=img.data_ptr(), layers=wl.layers, d_output=out.data_ptr(),
                         d_status=status.data_ptr()))
        keep.append((img, out, ref, status, ref_status))
    cuda.unmix_batch_device(jobs, solver=so)
    torch.cuda.synchronize()
    for _, out, ref, status, ref_status in keep:
        assert torch.equal(out, ref) and torch.equal(status, ref_status)
