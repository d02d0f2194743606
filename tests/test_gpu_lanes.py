"""The default solves, one pixel per lane (FP64, and FP32 with its FP64
re-solve), against the quad kernels:
outputs, statuses, counters and evaluation totals are the same bits, over the
layer counts, blend modes, starts, bounds, ragged and tiny pixel counts,
non-finite inputs and buffers that are only 8-byte aligned."""
import numpy as np
import pytest

from unblending_b200 import synthetic as syn

pytestmark = pytest.mark.gpu

QUADS = (3, 7)   # the quad variants of the first pass and of the refinement
QUADS32 = (3, 5)   # the same in FP32


def passes(cuda, wl, opaque=True, smooth=False, starts=1, radius=3, quads=False, image=None, offset=0, precision=1):
    """Both passes through the device entry points; `offset` doubles into larger buffers."""
    import torch

    n, L = wl.pixels, len(wl.layers)
    img = torch.zeros(3 * n + 2, dtype=torch.float64, device="cuda")
    img[offset:offset + 3 * n] = torch.from_numpy(wl.image if image is None else image).cuda().reshape(-1)
    out = [torch.zeros(4 * L * n + 2, dtype=torch.float64, device="cuda") for _ in range(2)]
    status = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2)]
    counters = [torch.zeros(5 * n, dtype=torch.int32, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    d_img, d_out = img.data_ptr() + 8 * offset, [o.data_ptr() + 8 * offset for o in out]
    so = [cuda.solver_options(starts=starts, radius=radius, precision=precision, fp64_variant=QUADS[k] if quads else -1,
                              kernel_variant=QUADS32[k] if quads else -1) for k in range(2)]
    s1 = cuda.unmix_device(wl.width, wl.height, d_img, wl.layers, d_out[0], opaque=opaque, solver=so[0],
                           d_status=status[0].data_ptr(), d_counters=counters[0].data_ptr(), stats=True)
    s2 = cuda.refine_device(wl.width, wl.height, d_img, wl.layers, d_out[0], d_out[1], opaque=opaque, smooth=smooth,
                            solver=so[1], d_status=status[1].data_ptr(), d_counters=counters[1].data_ptr(), stats=True)
    torch.cuda.synchronize()
    totals = [s[k] for s in (s1, s2) for k in ("misses", "failed", "normalization_failed", "fp64_values",
                                               "fp64_gradients", "fp32_values", "fp32_gradients")]
    return [o[offset:offset + 4 * L * n].cpu().numpy() for o in out] + [t.cpu().numpy() for t in status + counters], totals


def same(cuda, wl, **kw):
    lanes, lane_totals = passes(cuda, wl, **kw)
    quads, quad_totals = passes(cuda, wl, quads=True, **kw)
    for k, (a, b) in enumerate(zip(lanes, quads)):
        np.testing.assert_array_equal(a, b, err_msg=f"output {k}")
    assert lane_totals == quad_totals


@pytest.mark.parametrize("precision", [1, 0])
@pytest.mark.parametrize("modes,size,starts,opaque,smooth,comp", [
    ([0], (96, 65), 1, True, True, syn.SOURCE_OVER),
    ([0, 6], (96, 65), 3, True, False, syn.SOURCE_OVER),
    ([0, 1, 2], (96, 65), 2, True, True, syn.SOURCE_OVER),
    ([0, 1, 5], (96, 65), 1, False, False, syn.PLUS),
    ([0, 3, 8, 4], (96, 65), 3, True, True, syn.SOURCE_OVER),
    ([0, 1, 2, 3, 6], (96, 65), 3, True, True, syn.SOURCE_OVER),
    ([0, 7, 9, 10, 11, 12], (64, 33), 2, True, False, syn.SOURCE_OVER),
    ([0, 6, 7, 9, 2, 5, 12], (40, 31), 3, True, True, syn.SOURCE_OVER),
    ([0, 1, 2, 3, 6, 9, 7, 8], (40, 31), 3, False, False, syn.SOURCE_OVER),
])
def test_lanes_equal_quads(cuda, modes, size, starts, opaque, smooth, comp, precision):
    wl = syn.generate(*size, modes, (5.0, 20.0), seed=sum(modes) + size[0], comp=comp)
    same(cuda, wl, starts=starts, opaque=opaque, smooth=smooth, precision=precision)


# One pixel, fewer pixels than warps, one more than the warps (3 x 4 warps on each of 148 SMs), ragged.
@pytest.mark.parametrize("size", [(1, 1), (1, 7), (31, 1), (33, 5), (37, 48), (1777, 1)])
def test_pixel_counts(cuda, size):
    same(cuda, syn.generate(*size, [0, 1, 2, 3, 6], (3.0, 9.0), seed=size[0] + 31 * size[1]), smooth=True)


@pytest.mark.parametrize("precision", [1, 0])
def test_non_finite_and_out_of_range_pixels(cuda, precision):
    wl = syn.generate(48, 40, [0, 1, 6, 7, 9], (5.0, 20.0), seed=11)
    img = wl.image.copy().reshape(-1, 3)
    img[::7, 0], img[3::11, 1], img[5::13] = np.nan, np.inf, -np.inf
    img[2::17], img[4::19] = -3.0, 1e300
    same(cuda, wl, image=img.reshape(wl.image.shape), radius=0, precision=precision)


def test_buffers_aligned_to_eight_bytes(cuda):
    same(cuda, syn.generate(61, 45, [0, 1, 2, 3], (5.0, 20.0), seed=23), smooth=True, offset=1)


def test_in_place_refinement_and_row_bands(cuda):
    import torch

    wl = syn.generate(70, 52, [0, 1, 2, 3, 6], (5.0, 20.0), seed=29)
    (ref1, ref2, *_), _ = passes(cuda, wl, smooth=True, quads=True)
    img = torch.from_numpy(wl.image).cuda()
    buf = torch.zeros(ref1.size, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for rows in ((0, 20), (20, 20), (20, 21), (21, 52)):
        cuda.unmix_device_rows(wl.width, wl.height, img.data_ptr(), wl.layers, buf.data_ptr(), *rows, stats=True)
    np.testing.assert_array_equal(buf.cpu().numpy(), ref1)
    cuda.refine_device(wl.width, wl.height, img.data_ptr(), wl.layers, buf.data_ptr(), buf.data_ptr(), smooth=True,
                       solver=cuda.solver_options(radius=3), stats=True)
    np.testing.assert_array_equal(buf.cpu().numpy(), ref2)


def test_unequal_composite_factors(cuda):
    """Composite factors other than source-over and plus (first pass only):
    composite alphas away from [0, 1]."""
    import torch

    wl = syn.generate(64, 40, [0, 2, 6, 1], (5.0, 20.0), seed=37)
    arr = syn.layer_array(wl.layers)
    for k, comp in enumerate(((1, 1, 1), (3, 2, 1), (0, 1, 2), (1, 0, 1))):
        arr[k].comp_x, arr[k].comp_y, arr[k].comp_z = comp
    img = torch.from_numpy(wl.image).cuda()
    outs = []
    for v in (-1, QUADS[0]):
        out = torch.zeros(4 * 4 * wl.pixels, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        cuda.unmix_device(wl.width, wl.height, img.data_ptr(), arr, out.data_ptr(), opaque=False,
                          solver=cuda.solver_options(fp64_variant=v), stats=True)
        outs.append(out.cpu().numpy())
    np.testing.assert_array_equal(outs[0], outs[1])


@pytest.mark.parametrize("sizes", [((40, 30), (24, 50)), ((3, 2), (200, 120))])
def test_batches_of_changing_job_lists(cuda, sizes):
    """The batched solves' records outlive a job list: lists that take turns, on
    two streams without a wait between the calls, and whose groups need other
    sizes at the same place, still give the single-image results."""
    import torch

    lists, refs = [], []
    for k, layers in enumerate(((3, 5), (6,), (5, 3))):
        jobs, keep = [], []
        for L in layers:
            for w, h in sizes:
                wl = syn.generate(w, h, [0, 1, 2, 5, 0, 3][:L], (20.0, 200.0), 10 * k + L)
                img = torch.from_numpy(wl.image.reshape(-1)).cuda()
                out, ref = (torch.full((4 * L * w * h,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
                cuda.unmix_device(w, h, img.data_ptr(), wl.layers, ref.data_ptr())
                jobs.append(dict(width=w, height=h, d_image=img.data_ptr(), layers=wl.layers, d_output=out.data_ptr()))
                keep.append((img, out, ref))
        lists.append(jobs)
        refs.append(keep)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for turn in range(2):
        for k, jobs in enumerate(lists):
            cuda.unmix_batch_device(jobs, stream=streams[(turn + k) % 2].cuda_stream)
        torch.cuda.synchronize()
        for keep in refs:
            for _, out, ref in keep:
                assert torch.equal(out, ref)
                out.fill_(float("nan"))
        torch.cuda.synchronize()
