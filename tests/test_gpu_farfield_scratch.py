"""One scratch buffer serves every all-pairs sum up to the one it was sized
for: a smaller problem, which is cut into more pieces to fill the chip, takes
fewer of them where the buffer does not hold their partial sums."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("precision", ["fp32c", "fp64"])
@pytest.mark.parametrize("nsrc,ns,most,ntp", [(16, 192, 640, 32), (40, 64, 40, 16), (33, 96, 130, 48)])
def test_smaller_calls_fit_the_largest_call_s_buffer(nsrc, ns, most, ntp, precision):
    from ves2dpy_gb300 import _native as nat
    from ves2dpy_gb300.biem_support import _farfield
    ctx, prec = nat.context(ntp, DEV), nat.PREC[precision]
    g = torch.Generator().manual_seed(nsrc)
    r = dict(dtype=torch.float64, generator=g)
    c = 400.0 * torch.rand(most, 2, 1, **r)
    t = lambda n: 2 * math.pi * torch.arange(n, dtype=torch.float64) / n  # noqa: E731
    e = lambda n: torch.stack((0.3 * torch.cos(t(n)), 0.2 * torch.sin(t(n))))  # noqa: E731
    cs = c[:nsrc] if most >= nsrc else 400.0 * torch.rand(nsrc, 2, 1, **r)
    Xs = (cs + 0.03 + e(ns)).reshape(nsrc, 2 * ns).contiguous().to(DEV)
    Xt = (c + e(ntp)).reshape(most, 2 * ntp).contiguous().to(DEV)
    den = (torch.randn(nsrc, 2 * ns, **r) * (2 * math.pi / ns)).to(DEV)
    idx = torch.arange(most, dtype=torch.int32, device=DEV)
    size = ctx.lib.ves_farfield_workspace(ctx.handle, prec, nsrc, ns, most, ntp)
    ws = torch.empty(size, dtype=torch.uint8, device=DEV)
    ref = _farfield("fp64", Xs, den, Xt, idx, None, ntp)
    scale = max(float(ref.abs().max()), 1e-3 * float(den.abs().sum()))
    tol = 1e-5 if precision == "fp32c" else 1e-12  # the FP32 rule's accuracy; a sum regrouped
    for nt in sorted({1, 2, 3, 5, 31, 33, most - 1, most} | set(range(1, most, max(1, most // 20)))):
        out = torch.full((nt, 2 * ntp), float("nan"), dtype=torch.float64, device=DEV)
        rc = ctx.lib.ves_farfield(ctx.handle, prec, nsrc, ns, Xs.data_ptr(), den.data_ptr(), nt, ntp, Xt.data_ptr(),
                                  idx.data_ptr(), None, out.data_ptr(), ws.data_ptr(), size, nat.stream_ptr(DEV))
        assert rc == 0, (nt, rc)
        assert float((out - ref[:nt]).abs().max()) <= tol * scale, nt


def test_static_scratch_filled_by_the_records():
    """2.09 million FP64 sources leave 0.2 of the fixed 64 MiB to the targets and
    the partial sums: fewer pieces than the plan for a caller's buffer takes."""
    from ves2dpy_gb300 import _native as nat
    from ves2dpy_gb300.biem_support import _farfield
    nsrc, ns, nt, ntp = 1000, 2090, 16, 32
    r = dict(dtype=torch.float64, generator=torch.Generator().manual_seed(1))
    t = lambda n: 2 * math.pi * torch.arange(n, dtype=torch.float64) / n  # noqa: E731
    e = lambda n: torch.stack((0.3 * torch.cos(t(n)), 0.2 * torch.sin(t(n))))  # noqa: E731
    Xs = (400.0 * torch.rand(nsrc, 2, 1, **r) + e(ns)).reshape(nsrc, 2 * ns).contiguous().to(DEV)
    Xt = (-2.0 - 40.0 * torch.rand(nt, 2, 1, **r) + e(ntp)).reshape(nt, 2 * ntp).contiguous().to(DEV)
    den = (torch.randn(nsrc, 2 * ns, **r) * (2 * math.pi / ns)).to(DEV)
    ref = _farfield("fp64", Xs, den, Xt, None, None, ntp)
    out = torch.empty(nt, 2 * ntp, dtype=torch.float64, device=DEV)
    nat.check(nat.load_library().ves_farfield_static_scratch(
        nat.PREC["fp64"], nsrc, ns, Xs.data_ptr(), den.data_ptr(), nt, ntp, Xt.data_ptr(), None, out.data_ptr(),
        nat.stream_ptr(DEV)), "static scratch")
    assert float((out - ref).abs().max()) <= 1e-12 * max(float(ref.abs().max()), 1e-3 * float(den.abs().sum()))
