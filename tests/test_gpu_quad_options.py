"""The scheduling options of the quad kernels (gradient_quorum, defer_outer),
which calls that name a quad variant run: outputs, statuses and counters do not
depend on them. (Calls that name none run one pixel per lane, where neither
option has an effect.)"""
import numpy as np
import pytest

from unblending_b200 import synthetic as syn

pytestmark = pytest.mark.gpu

FIRST = dict(fp64_variant=3, kernel_variant=3)
REFINE = dict(fp64_variant=7, kernel_variant=5)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("variants", [(FIRST, REFINE), (dict(fp64_variant=0, kernel_variant=1),
                                                        dict(fp64_variant=2, kernel_variant=3))])
def test_gradient_quorum(cuda, precision, variants):
    wl = syn.generate(64, 48, [0, 1, 2, 3, 9], (4.0, 16.0), seed=77)
    outs = []
    for q in (0, 3, 4, 8):
        so = [cuda.solver_options(precision=precision, radius=3, gradient_quorum=q, **v) for v in variants]
        first, st1, c1, _ = cuda.unmix_ex(wl.image, wl.layers, solver=so[0], with_counters=True)
        final, st2, c2, _ = cuda.refine_ex(wl.image, first, wl.layers, smooth=True, solver=so[1], with_counters=True)
        outs.append((first, st1, c1, final, st2, c2))
    for other in outs[1:]:
        for a, b in zip(outs[0], other):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("size,modes,sigma,starts", [((96, 80), [0, 1, 2, 3, 6], (8.0, 40.0), 1),
                                                     ((96, 80), [0, 1, 2, 3, 6], (8.0, 40.0), 3),
                                                     ((64, 48), [0, 6, 7, 9, 1], (8.0, 40.0), 1),
                                                     ((1, 1), [0, 1, 2], (3.0, 9.0), 1)])
def test_deferral(cuda, size, modes, sigma, starts):
    """Pixels deferred at outer step `defer_outer` and resumed, also where the
    slots run out (defer_outer 1 defers most pixels, past the slots for a
    quarter of them), over the whole image and in row bands."""
    import torch

    wl = syn.generate(*size, modes, sigma, seed=8)
    first, _, _, _ = cuda.unmix_ex(wl.image, wl.layers)
    n, L = wl.pixels, len(wl.layers)
    img, d_first = torch.from_numpy(wl.image.reshape(-1)).cuda(), torch.from_numpy(first.reshape(-1)).cuda()
    cuts = sorted({0, wl.height // 3, wl.height})
    runs = []
    for defer in (0, 8, 3, 1):
        so = cuda.solver_options(radius=3, starts=starts, defer_outer=defer, **REFINE)
        out, status, counters, _ = cuda.refine_ex(wl.image, first, wl.layers, smooth=True, solver=so, with_counters=True)
        bands = torch.full((4 * L * n,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for r0, r1 in zip(cuts, cuts[1:]):
            cuda.refine_device_rows(wl.width, wl.height, img.data_ptr(), wl.layers, d_first.data_ptr(),
                                    bands.data_ptr(), r0, r1, smooth=True, solver=so)
        torch.cuda.synchronize()
        assert np.array_equal(bands.cpu().numpy().reshape(out.shape), out), defer
        runs.append((out, status, counters))
    if wl.pixels > 1:
        assert (runs[0][2][:, 4] > 1).sum() > wl.pixels // 4   # more pixels than slots reach outer step 1
    for other in runs[1:]:
        for a, b in zip(runs[0], other):
            assert np.array_equal(a, b)
