"""The multipole all-pairs sum at the sizes where its split of the work can go
wrong: source counts around a stage of 32, target columns off a warp, one, four
and eight warps per 32 points, near-pair exclusions of close and of separated
sources.  Against the FP64 direct rule at 1e-6 (the accuracy of the FP32 series
and direct rule, tests/test_gpu_farfield_mp.py), and bit for bit between the
splits, which add a point's contributions in the same order."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


def _case(nsrc, ns, nt, ntp, seed):
    g = torch.Generator().manual_seed(seed)
    r = dict(dtype=torch.float64, generator=g)
    side = 1.2 * math.sqrt(max(nsrc, nt))
    c = side * torch.rand(max(nsrc, nt), 2, 1, **r)
    th = lambda n: 2 * math.pi * torch.arange(n, dtype=torch.float64) / n  # noqa: E731

    def curves(k, n):
        t = th(n)
        e = torch.stack((0.35 * torch.cos(t), 0.2 * torch.sin(t)))
        return (c[:k] + e).reshape(k, 2 * n).contiguous().to(DEV)

    den = torch.randn(nsrc, 2 * ns, **r) * (2 * math.pi / ns)
    return curves(nsrc, ns), den.to(DEV), curves(nt, ntp)


@pytest.mark.parametrize("nsrc,ns,nt,ntp", [(1, 48, 1, 16), (31, 64, 31, 20), (32, 100, 32, 32), (33, 96, 33, 33),
                                            (65, 192, 9, 96), (90, 33, 90, 128), (700, 40, 700, 64)])
def test_sizes(nsrc, ns, nt, ntp):
    from ves2dpy_gb300.biem_support import _farfield
    Xs, den, Xt = _case(nsrc, ns, nt, ntp, nsrc + ntp)
    Xt = Xt + 0.05  # no target point on a source point
    idx = torch.arange(nt, dtype=torch.int32, device=DEV)
    ref = _farfield("fp64", Xs, den, Xt, idx, None, ntp)
    got = _farfield("fp32m", Xs, den, Xt, idx, None, ntp)
    assert float((got - ref).abs().max()) <= 1e-6 * max(float(ref.abs().max()), 1e-3 * float(den.abs().sum()))


@pytest.mark.parametrize("ntp", [32, 48])
def test_result_does_not_depend_on_the_split(ntp):
    from ves2dpy_gb300.biem_support import _farfield
    nt = 1400
    Xs, den, Xt = _case(nt, 64, nt, ntp, 5)
    Xt = Xt + 0.05
    idx = torch.arange(nt, dtype=torch.int32, device=DEV)
    whole = _farfield("fp32m", Xs, den, Xt, idx, None, ntp)          # one warp per 32 points
    for k0, k1 in ((0, 400), (400, 420), (1399, 1400)):              # four, eight, eight
        part = _farfield("fp32m", Xs, den, Xt[k0:k1].contiguous(), idx[k0:k1].contiguous(), None, ntp)
        assert torch.equal(part, whole[k0:k1])


def test_exclusions_of_close_and_separated_sources():
    from ves2dpy_gb300 import biem_support as B
    nsrc, ns, N = 40, 64, 40
    Xs, den, Xt = _case(nsrc, ns, nsrc, N, 11)
    Xt = Xt + 0.05
    rng = np.random.default_rng(2)
    rows = sorted({(int(rng.integers(nsrc - 1)), int(rng.integers(N)), int(rng.integers(nsrc))) for _ in range(300)})
    ids = [[r[k] for r in rows] for k in range(3)]
    sa = torch.ones(ns, nsrc, dtype=torch.float64, device=DEV)
    f = (den * ns / (2 * math.pi)).t().contiguous()
    args = (Xs.t().contiguous(), sa, f, Xt.t().contiguous(), *ids)
    ref = B.allExactStokesSLTarget_compare2(*args, precision="fp64")
    got = B.allExactStokesSLTarget_compare2(*args, precision="fp32m")
    assert float((got - ref).abs().max()) <= 1e-6 * float(ref.abs().max())
