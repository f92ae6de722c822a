"""The FP64 all-pairs sum at the sizes where its split of the work can go
wrong: one source, pieces of a source vesicle with a remainder, target counts
off a warp and off a CTA, more pieces than splits, near-pair exclusions.  The
reference is the same sum in plain torch FP64; both add at most 6e4 terms of
one sign-changing sum, so 1e-12 of the largest value covers their rounding."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("nsrc,ns,nt,ntp", [(1, 7, 1, 1), (1, 33, 3, 20), (2, 16, 2, 32), (5, 100, 5, 24),
                                            (16, 192, 16, 32), (40, 1536, 3, 128), (300, 31, 300, 16)])
@pytest.mark.parametrize("near", [False, True])
def test_fp64_direct_rule(nsrc, ns, nt, ntp, near):
    from ves2dpy_gb300 import biem_support as B
    g = torch.Generator().manual_seed(nsrc * 1000 + ns)
    r = dict(dtype=torch.float64, generator=g)
    c = 5.0 * torch.rand(2, max(nsrc, nt), **r)
    Xs = torch.cat((c[0, :nsrc] + 0.3 * torch.rand(ns, nsrc, **r), c[1, :nsrc] + 0.3 * torch.rand(ns, nsrc, **r)))
    Xt = torch.cat((c[0, :nt] + 0.3 * torch.rand(ntp, nt, **r), c[1, :nt] + 0.3 * torch.rand(ntp, nt, **r)))
    f = torch.randn(2 * ns, nsrc, **r)
    sa = 0.5 + torch.rand(ns, nsrc, **r)
    off = 0 if nt == nsrc else nsrc - nt if nsrc > nt else 0
    ids = [], [], []
    keep = torch.ones(nt, ntp, nsrc, dtype=torch.bool)
    for t in range(nt):
        if off + t < nsrc:
            keep[t, :, off + t] = False
    if near and nsrc > 1:
        rng = np.random.default_rng(3)
        pairs = set()
        while len(pairs) < min(40, nt * ntp):
            t, i, s = int(rng.integers(nt)), int(rng.integers(ntp)), int(rng.integers(nsrc))
            if s != off + t:
                pairs.add((s - (1 if s > off + t else 0), i, t, s))
            elif nsrc == 1:
                break
        for j, i, t, s in sorted(pairs):
            ids[0].append(j), ids[1].append(i), ids[2].append(t)
            keep[t, i, s] = False
    den = f * torch.cat((sa, sa)) * (2 * np.pi / ns)
    x, y = Xt[:ntp].t(), Xt[ntp:].t()
    ref = torch.zeros(2 * ntp, nt, dtype=torch.float64)
    for s in range(nsrc):
        dx, dy = x[..., None] - Xs[:ns, s], y[..., None] - Xs[ns:, s]
        r2 = dx * dx + dy * dy
        lg, dot = -0.5 * torch.log(r2), (dx * den[:ns, s] + dy * den[ns:, s]) / r2
        m = keep[:, :, s].double()
        ref[:ntp] += (((lg * den[:ns, s] + dot * dx).sum(-1)) * m).t() / (4 * np.pi)
        ref[ntp:] += (((lg * den[ns:, s] + dot * dy).sum(-1)) * m).t() / (4 * np.pi)
    d = lambda a: a.to(DEV)  # noqa: E731
    got = B.allExactStokesSLTarget_compare2(d(Xs), d(sa), d(f), d(Xt), *ids, offset=off, precision="fp64").cpu()
    scale = max(float(ref.abs().max()), 1e-300)
    assert float((got - ref).abs().max()) <= 1e-12 * max(scale, 1.0)
