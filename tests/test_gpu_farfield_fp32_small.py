"""The direct FP32 rule where its plan changes: from one source vesicle over
splits of one and of a few to the sizes that fill the chip with whole stages,
twice the same bits.  Against the FP64 rule at
1e-5 (the accuracy of the FP32 rule, tests/test_gpu_parity.py)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("nsrc,ns,nt,ntp", [(1, 48, 1, 16), (2, 192, 2, 32), (16, 192, 16, 32), (17, 48, 3, 128),
                                            (40, 64, 40, 16), (101, 192, 101, 32), (61, 1536, 61, 128),
                                            (310, 40, 1, 7), (700, 40, 40, 64)])
def test_sizes(nsrc, ns, nt, ntp):
    from ves2dpy_gb300.biem_support import _farfield
    r = dict(dtype=torch.float64, generator=torch.Generator().manual_seed(nsrc + ntp))
    c = 1.2 * math.sqrt(max(nsrc, nt)) * torch.rand(max(nsrc, nt), 2, 1, **r)

    def curves(k, n):
        t = 2 * math.pi * torch.arange(n, dtype=torch.float64) / n
        return (c[:k] + torch.stack((0.35 * torch.cos(t), 0.2 * torch.sin(t)))).reshape(k, 2 * n).contiguous().to(DEV)

    Xs, Xt = curves(nsrc, ns), curves(nt, ntp) + 0.05  # no target point on a source point
    den = (torch.randn(nsrc, 2 * ns, **r) * (2 * math.pi / ns)).to(DEV)
    idx = torch.arange(nt, dtype=torch.int32, device=DEV)
    ref = _farfield("fp64", Xs, den, Xt, idx, None, ntp)
    got = _farfield("fp32c", Xs, den, Xt, idx, None, ntp)
    assert torch.equal(got, _farfield("fp32c", Xs, den, Xt, idx, None, ntp))
    assert float((got - ref).abs().max()) <= 1e-5 * max(float(ref.abs().max()), 1e-3 * float(den.abs().sum()))
