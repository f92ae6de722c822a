"""A suspension handed over as several point sets of one point count is the
suspension: the multipole sum runs over the sets one after the other, with
stages of sources that end short at each set, and adds a target point's
contributions in the order of the joined suspension.  Without near
corrections (whose width is each set's own) the step is the same bit for bit,
with one, four and eight warps per 32 target points."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("counts, N", [((45, 38), 32), ((33, 1, 70), 32), ((64, 32), 32), ((20, 50, 33, 65), 48),
                                       ((200, 150), 64), ((900, 700), 32), ((1, 95, 320), 128)])
def test_sets_are_the_suspension(counts, N):
    from ves2dpy_gb300 import TStepBiem, TStepBiemMixed
    nv = sum(counts)
    rng = np.random.default_rng(nv)
    n = math.isqrt(nv - 1) + 1
    k, t = rng.permutation(nv), 2 * math.pi * np.arange(N)[:, None] / N
    r = 0.16 * (1.0 + rng.uniform(0.0, 0.1, nv))
    x = 0.5 * (k % n) + rng.uniform(-0.03, 0.03, nv) + r * np.cos(t) * 0.9
    y = 0.5 * (k // n) + rng.uniform(-0.03, 0.03, nv) + r * np.sin(t)
    X = torch.tensor(np.concatenate([x, y]), dtype=torch.float64, device=DEV)
    zero = torch.zeros(N, nv, dtype=torch.float64, device=DEV)
    prams = dict(dt=1e-5, kappa=1.0, gmresTol=1e-8, gmresMaxIter=200, farFieldSpeed=1.0, viscCont=1.0)
    opts = dict(farField="shear", usePreco=True, repulsion=False)
    kw = dict(near="none", farfield_precision="fp32m", sl_precision="fp32c")
    one = TStepBiem(X, None, opts, prams, **kw)
    Xr, sr, _, _, it, flag = one.time_step(X, zero)
    Xs = [a.contiguous() for a in X.split(counts, dim=1)]
    Xo, so, it2, flag2 = TStepBiemMixed(Xs, opts, prams, **kw).time_step(
        Xs, [a.contiguous() for a in zero.split(counts, dim=1)])
    assert not flag and not flag2 and it == it2
    assert torch.equal(torch.cat(list(so), 1), sr) and torch.equal(torch.cat(list(Xo), 1), Xr)
