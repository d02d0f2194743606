"""The guided filter's targets at the edges of its passes: rows and columns
around the column pass's batches of eight and segments of 128, few rows (the
row pass shares their planes among CTAs) and more rows than one wave of CTAs,
windows larger than the image, against the oracle's filter (FP64, 1e-12, as
tests/test_gpu_parity.py)."""
import numpy as np
import pytest

import oracle
from unblending_b200 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,radius", [((5, 1), 1), ((1, 9), 2), ((33, 7), 3), ((40, 8), 9), ((17, 127), 4),
                                         ((20, 129), 60), ((3, 1190), 5), ((257, 16), 8)])
def test_targets(cuda, size, radius):
    wl = syn.generate(*size, [0, 1], (3.0, 9.0), seed=size[0] + size[1])
    first, _, _, _ = cuda.unmix_ex(wl.image, wl.layers)
    L = len(wl.layers)
    out, _, _, stats = cuda.refine_ex(wl.image, first, wl.layers, smooth=True, solver=cuda.solver_options(radius=radius))
    assert stats["radius"] == radius
    _, _, targets, _ = oracle.refine(wl.image, oracle.unpack(first, L), wl.layers, opaque=True, smooth=True,
                                     radius=radius, opts=oracle.options())
    alpha = targets[:L].copy()
    alpha[0] = 1.0   # (the opaque background's written alpha)
    np.testing.assert_allclose(out[..., 3].reshape(L, -1), alpha, rtol=0, atol=1e-12)
    np.testing.assert_allclose(out[0, ..., :3].reshape(-1, 3), targets[L:].T, rtol=0, atol=1e-12)
