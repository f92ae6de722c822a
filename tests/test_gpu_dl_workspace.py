"""The double layer's workspace queries count the sources' points: the sum runs
in exactly what they ask for, and in Python on a context that has none yet.
Against the FP64 direct sum at 1e-6 (as tests/test_gpu_dl.py's multipole
tests)."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


def circles(nv, n, seed):
    r = dict(dtype=torch.float64, generator=torch.Generator().manual_seed(seed))
    k = torch.arange(nv, dtype=torch.float64)
    side = math.isqrt(nv - 1) + 1
    c = 2.6 * torch.stack((k % side, torch.div(k, side, rounding_mode="floor"))) + 0.1 * torch.rand(2, nv, **r)
    t = 2 * math.pi * torch.arange(n, dtype=torch.float64)[:, None] / n
    return torch.cat((c[0] + torch.cos(t), c[1] + 0.9 * torch.sin(t))).to(DEV), torch.randn(2 * n, nv, **r).to(DEV)


@pytest.mark.parametrize("nv, N", [(3, 32), (200, 128), (900, 64)])
def test_python_call_on_a_new_context(nv, N, monkeypatch):
    from ves2dpy_gb300 import Poten
    from ves2dpy_gb300.capsules import capsules
    X, f = circles(nv, N, nv)
    ves = capsules(X, None, None, 1.0, 3.0)
    op = Poten(N)
    Xt = torch.cat((X[:N, :1], X[N:, :1] - 20.0))  # a column away from the vesicles
    ref = op.exactStokesDL(ves, f, Xt)
    monkeypatch.setattr(op._ctx, "_ws", None)  # as no call has made one yet
    got = op.exactStokesDL(ves, f, Xt, precision="fp32m")
    assert float((got - ref).abs().max()) <= 1e-6 * float(ref.abs().max())


def test_queries_cover_the_call():
    from ves2dpy_gb300 import _native as nat
    lib = nat.load_library()
    for prec in ("fp32c", "fp32m"):
        p = nat.PREC[prec]
        for nsrc, nt, ntp in ((1, 1, 16), (700, 700, 64)):
            sizes = [lib.ves_farfield_dl_workspace_ns(p, nsrc, ns, nt, ntp) for ns in (16, 512, 8533)]
            assert sizes[0] + 24 * 496 * nsrc <= sizes[1] + 1024 and sizes[1] < sizes[2]
            assert lib.ves_farfield_dl_workspace(p, nsrc, nt, ntp) == sizes[2]
