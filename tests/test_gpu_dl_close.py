"""The double layer's multipole path at the sizes where its close pairs can go
wrong: point counts off a multiple of 8, 32 and 256, few and many points of a
warp within 12 source spacings (summed in FP64, four at a time), and one, four
and eight warps per 32 points.  Against the direct FP64 rule: the close points
at 1e-12 of the sum of their terms' sizes (FP64 against FP64, at most 600 terms
of rounding 1.1e-16 each), the rest at 1e-6 of it (FP32 terms and series)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


def _circles(nv, ns, side, seed):
    g = torch.Generator().manual_seed(seed)
    th = 2 * math.pi * torch.arange(ns, dtype=torch.float64) / ns
    c = torch.stack((torch.arange(nv) % side, torch.arange(nv) // side), 1).to(torch.float64)
    t = torch.stack((-torch.sin(th), torch.cos(th)))[None].expand(nv, 2, ns)
    X = c[:, :, None] + 0.3 * torch.stack((torch.cos(th), torch.sin(th)))
    sa = torch.full((nv, ns), 0.3, dtype=torch.float64)
    f = torch.randn(nv, 2, ns, dtype=torch.float64, generator=g)
    flat = lambda a: a.reshape(nv, -1).contiguous().to(DEV)  # noqa: E731
    return flat(X), flat(t), flat(sa), flat(f)


def _run(prec, X, t, sa, f, visc, Xt, idx):
    from ves2dpy_gb300 import _native as nat
    lib, st, nv, ns = nat.load_library(), nat.stream_ptr(DEV), X.shape[0], sa.shape[1]
    nt, ntp = Xt.shape[0], Xt.shape[1] // 2
    ctx, p = nat.context(32, DEV), nat.PREC[prec]
    den, out = torch.empty_like(f), torch.empty_like(Xt)
    nat.check(lib.ves_dl_density(nv, ns, f.data_ptr(), sa.data_ptr(), visc.data_ptr(), den.data_ptr(), st), "density")
    ws = torch.empty(lib.ves_farfield_dl_workspace(p, nv, nt, max(ns, ntp)) + nv * ns * 32 + (1 << 20),
                     dtype=torch.uint8, device=DEV)
    nat.check(lib.ves_farfield_dl(ctx.handle, p, nv, ns, X.data_ptr(), t.data_ptr(), den.data_ptr(), sa.data_ptr(),
                                  visc.data_ptr(), nt, ntp, Xt.data_ptr(), idx.data_ptr(), None, out.data_ptr(),
                                  ws.data_ptr(), ws.numel(), st), "dl")
    return out, den


@pytest.mark.parametrize("nv,ns,ntp,nclose", [(9, 33, 40, 1), (9, 64, 40, 5), (12, 100, 33, 33), (49, 255, 64, 3),
                                              (400, 257, 32, 4), (400, 513, 32, 9), (1400, 96, 32, 2)])
def test_close_points(nv, ns, ntp, nclose):
    X, t, sa, f = _circles(nv, ns, int(math.sqrt(nv)), ns)
    visc = torch.full((nv,), 3.0, dtype=torch.float64, device=DEV)
    h = 0.6 * math.pi / ns
    # a column sits around the next circle but one: nclose points 2 to 6 spacings
    # off that circle, the others midway to its neighbours (all outside every
    # curve, where the rule with the mean taken off holds)
    k = torch.arange(ntp, dtype=torch.float64)
    near = k < nclose
    rad = torch.where(near, 0.3 + (2 + k % 5) * h, 0.5 * torch.ones(ntp, dtype=torch.float64))
    th = 2.399963 * k
    off = torch.stack((rad * torch.cos(th), rad * torch.sin(th)))
    c = X.reshape(nv, 2, ns).mean(2).roll(-2, 0).cpu()
    Xt = (c[:, :, None] + off).reshape(nv, -1).contiguous().to(DEV)
    idx = torch.arange(nv, dtype=torch.int32, device=DEV)
    ref, den = _run("fp64", X, t, sa, f, visc, Xt, idx)
    got, _ = _run("fp32m", X, t, sa, f, visc, Xt, idx)
    size = float(den.abs().sum(1).max()) / (4 * h * h) ** 0.5 / math.pi  # a source's terms at two spacings
    err = (got - ref).abs().reshape(nv, 2, ntp).amax((0, 1)).cpu()
    assert bool((err[near] <= 1e-6 * size).all()) and bool((err <= 1e-6 * size).all())
    # one source alone, no series and no FP32 sum: the close points to FP64 rounding
    one = lambda a: a[2:3].contiguous()  # noqa: E731
    own = torch.tensor([-1], dtype=torch.int32, device=DEV)
    a, _ = _run("fp64", one(X), one(t), one(sa), one(f), one(visc), Xt[:1].contiguous(), own)
    b, _ = _run("fp32m", one(X), one(t), one(sa), one(f), one(visc), Xt[:1].contiguous(), own)
    err = (a - b).abs().reshape(2, ntp).amax(0).cpu()
    assert bool((err[near] <= 1e-12 * size).all()), err[near].max() / size
