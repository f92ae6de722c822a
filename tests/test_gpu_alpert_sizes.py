"""The FP64 self-interaction matrices at point counts whose products with the
interpolation matrices run as transforms (powers of two and three times one,
one to four row pairs per CTA, a last CTA with fewer rows) and at counts that
fall back to the dense products.  Against the oracle's matrices at 1e-11 of
the largest entry: both sum at most N ceil(sqrt(N)) products twice in FP64."""
import numpy as np
import pytest
import torch

from oracle import ves2d_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nv", [(8, 3), (12, 2), (16, 1), (20, 2), (24, 3), (32, 5), (48, 1), (64, 2), (96, 1), (128, 1)])
def test_fp64_matrix(N, nv):
    from ves2dpy_gb300.capsules import capsules
    from ves2dpy_gb300.poten import Poten
    from ves2dpy_gb300.suspension import vesicle_shape
    rng = np.random.default_rng(N)
    X = np.zeros((2 * N, nv))
    for k in range(nv):
        x, y = vesicle_shape(N, rng, 0.8)
        X[:N, k], X[N:, k] = x + 3.0 * k, y
    ref = O.stokes_sl_matrix(X, O.PotenTables(N))
    Xd = torch.tensor(X, dtype=torch.float64, device="cuda:0")
    got = Poten(N).stokesSLmatrix(capsules(Xd, None, None, 1.0, 1.0)).cpu().numpy()
    ref = np.asarray(ref)
    if ref.shape != got.shape:
        ref = np.moveaxis(ref, 0, -1)
    assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max()
