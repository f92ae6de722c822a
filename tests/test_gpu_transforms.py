"""The shared-memory transform at lengths with an even and an odd number of
radix-2 stages, with and without the factor three, through the upsampling
(1e-13 of the largest coordinate: at most 12 stages of FP64), and the arc-length
redistribution at more vesicles than fit the device at once: twice over and six
at a time the same bits, and those against the oracle (1e-10, as
tests/test_gpu_parity.py)."""
import numpy as np
import pytest
import torch

from oracle import ves2d_oracle as O
from ves2dpy_gb300 import _native as nat
from ves2dpy_gb300.suspension import vesicle_shape

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


def _shapes(N, nv):
    """[nv][2N], six shapes of about unit length in turn."""
    rng = np.random.default_rng(N)
    base = []
    for _ in range(6):
        x, y = vesicle_shape(N, rng, 0.7)
        z = x + 1j * y
        base.append(np.concatenate((x, y)) / np.abs(np.roll(z, -1) - z).sum())
    return np.stack([base[k % 6] for k in range(nv)])


@pytest.mark.parametrize("N", [8, 16, 32, 64, 128, 256])
def test_upsample(N):
    X = _shapes(N, 5)
    Nup = N * int(np.ceil(np.sqrt(N)))
    ctx = nat.context(N, DEV)
    Xd = torch.tensor(X, device=DEV)
    U = torch.empty(5, 2 * Nup, dtype=torch.float64, device=DEV)
    nat.check(ctx.lib.ves_upsample(ctx.handle, 5, 2, Xd.data_ptr(), U.data_ptr(), nat.stream_ptr(DEV)), "upsample")
    ref = O.interpft_vec(X.T, Nup).T
    assert np.abs(U.cpu().numpy() - ref).max() <= 1e-13 * np.abs(X).max()


@pytest.mark.parametrize("N", [16, 32, 128])
def test_redistribute_many(N):
    from ves2dpy_gb300 import curve
    X = torch.tensor(_shapes(N, 1500).T.copy(), device=DEV)
    oc = curve.Curve()  # updates its argument in place
    a, _ = oc.redistributeArcLength(X.clone())
    b, _ = oc.redistributeArcLength(X.clone())
    assert torch.equal(a, b)
    few, _ = oc.redistributeArcLength(X[:, :6].clone())  # every spread is above the threshold
    assert torch.equal(a, few.repeat(1, 250))
    ref = O.redistribute_arc_length(X[:, :6].cpu().numpy())[0]
    assert np.abs(few.cpu().numpy() - ref).max() <= 1e-10 * np.abs(ref).max()
