"""The lane kernels against the quad kernels where their code differs in form:
zeros of either sign, values far outside the unit cube, non-finite values, and
long schedules whose penalty grows until the arithmetic overflows. Outputs are
compared by their bits (NaN: any), statuses and counters by value."""
import numpy as np
import pytest

from tests.test_gpu_lanes import passes
from unblending_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


def same_bits(cuda, wl, image, precision, **kw):
    lanes, lane_totals = passes(cuda, wl, image=image, precision=precision, **kw)
    quads, quad_totals = passes(cuda, wl, image=image, precision=precision, quads=True, **kw)
    for k, (a, b) in enumerate(zip(lanes, quads)):
        equal = a == b
        if a.dtype.kind == "f":
            equal = (a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))
        assert equal.all(), (k, int((~equal).sum()))
    assert lane_totals == quad_totals


@pytest.mark.parametrize("precision", [1, 0])
@pytest.mark.parametrize("modes,comp,smooth", [([0, 1, 2], syn.SOURCE_OVER, True), ([0, 6, 7, 6], syn.PLUS, False),
                                               ([0, 9, 3, 8, 6, 7], syn.SOURCE_OVER, True),
                                               ([0, 6, 6, 6, 6, 6, 6, 6], syn.SOURCE_OVER, False)])
@pytest.mark.parametrize("values", ["image", "large", "mixed", "zeros"])
def test_bits(cuda, values, modes, comp, smooth, precision):
    wl = syn.generate(24, 17, modes, (3.0, 12.0), seed=len(modes), comp=comp)
    rng = np.random.default_rng(len(values))
    img = wl.image.copy()
    if values == "large":
        img *= 10.0 ** rng.uniform(-300, 150, img.shape[:2] + (1,))
    elif values == "mixed":
        img = np.where(rng.random(img.shape) < 0.3, 10.0 ** rng.uniform(10, 154, img.shape), img)
    elif values == "zeros":
        img = np.where(rng.random(img.shape) < 0.3, -0.0, img)
        img[::5, ::3], img[1::5, ::3] = np.nan, np.inf
    same_bits(cuda, wl, img, precision, opaque=smooth, smooth=smooth, starts=2)


# Penalties of up to 1e302 (FP32: infinity) in pixels that the method cannot solve.
@pytest.mark.parametrize("precision", [1, 0])
@pytest.mark.parametrize("modes", [[0, 1, 6], [0, 7, 9, 6, 6]])
def test_long_schedules(cuda, modes, precision, monkeypatch):
    wl = syn.generate(24, 17, modes, (3.0, 12.0), seed=41)
    img = wl.image.copy()
    img[::2, ::3] += 0.5
    options = cuda.solver_options
    monkeypatch.setattr(cuda, "solver_options",
                        lambda **kw: options(outer=300, inner=8, frozen_stop=0, resolve_misses=0, **kw))
    same_bits(cuda, wl, img, precision, smooth=True)
