"""The FP32 self-interaction matrices at point counts off the row and thread
blocks of their kernel and at the largest one, against the FP64 ones of the
device: 2e-5 of the largest entry (rounding of 1.2e-7 per FP32 value and
product, sums of up to a few thousand terms of one size)."""
import numpy as np
import pytest
import torch

from ves2dpy_gb300 import _native as nat
from ves2dpy_gb300.suspension import vesicle_shape

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nv", [(8, 3), (12, 2), (20, 2), (32, 5), (36, 1), (64, 3), (128, 2), (256, 1)])
def test_fp32_matrix(N, nv):
    rng = np.random.default_rng(N)
    dev = torch.device("cuda:0")
    X = np.zeros((nv, 2 * N))
    for k in range(nv):
        x, y = vesicle_shape(N, rng, 0.8)
        X[k, :N], X[k, N:] = x + 3.0 * k, y
    Xd = torch.tensor(X, dtype=torch.float64, device=dev)
    ctx, out = nat.context(N, dev), {}
    for prec in ("fp64", "fp32c"):
        p = nat.PREC[prec]
        ws = torch.empty(ctx.lib.ves_stokes_sl_matrix_workspace(ctx.handle, nv, p), dtype=torch.uint8, device=dev)
        G = torch.empty(nv, 4 * N * N, dtype=torch.float64, device=dev)
        nat.check(ctx.lib.ves_stokes_sl_matrix(ctx.handle, nv, Xd.data_ptr(), p, G.data_ptr(), ws.data_ptr(),
                                               ws.numel(), nat.stream_ptr(dev)), "sl")
        out[prec] = G
    err = (out["fp64"] - out["fp32c"]).abs().amax(1) / out["fp64"].abs().amax(1)
    assert float(err.max()) <= 2e-5, err
