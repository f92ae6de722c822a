"""The near corrections add to a target point in a fixed order.

A point near several source vesicles takes one addition per source.  The sum
is the same, bit for bit, whatever the order of the near entries in the lists
and of the warps that work on them: with the entries shuffled, over repeated
calls, and between point sets.
"""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


def T(a):
    return torch.tensor(np.asarray(a), dtype=torch.float64, device=DEV)


def packed_circles(rows, cols, gap, seed=0):
    """Centres and radii of a triangular packing of nearly unit circles."""
    rng = np.random.default_rng(seed)
    d = 2.0 + gap
    c = np.array([(d * (i + 0.5 * (j % 2)), d * math.sqrt(0.75) * j) for j in range(rows) for i in range(cols)])
    return c + rng.uniform(-0.1 * gap, 0.1 * gap, c.shape), 1.0 + rng.uniform(-0.1 * gap, 0.1 * gap, len(c))


def circles(c, r, N, turn=0.0):
    t = 2 * math.pi * np.arange(N)[:, None] / N + turn
    return np.concatenate([c[:, 0] + r * np.cos(t), c[:, 1] + 0.97 * r * np.sin(t)])


def shuffled(near, perm):
    """The near lists with their entries in another order (in place)."""
    n = len(perm)
    for a, w in ((near.ent_tsj, 3), (near.ent_icp, 1), (near.ent_geo, 4)):
        rows = a[:n * w].reshape(n, w)
        rows.copy_(rows[torch.as_tensor(perm, device=a.device)].clone())


@pytest.mark.parametrize("double", [False, True])
@pytest.mark.parametrize("N, room", [(16, 1024), (32, 1024), (32, 8192)])  # lists searched, lists with an index
def test_entries_in_any_order(N, room, double):
    from ves2dpy_gb300 import Poten
    from ves2dpy_gb300.biem_support import NearZone
    from ves2dpy_gb300.capsules import capsules
    from ves2dpy_gb300.layout import to_vm
    X = T(circles(*packed_circles(6, 6, 0.05), N))
    ves = capsules(X, None, None, 1.0, 3.0 if double else 1.0)
    near = NearZone.build_matlab(to_vm(X), N, h=0.9, max_entries=room)
    n = int(near.n_entries[0].item())
    assert (near.max_entries >= 4096) == (room >= 4096)
    tsj = near.ent_tsj[:3 * n].reshape(n, 3).cpu().numpy()
    _, of_point = np.unique(tsj[:, [0, 2]], axis=0, return_counts=True)
    assert (of_point == 2).sum() >= 20 and (of_point >= 3).sum() >= 3
    op = Poten(N)
    G = op.stokesDLmatrix(ves) if double else op.stokesSLmatrix(ves)
    f = torch.randn(X.shape, dtype=torch.float64, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1))

    def potential():
        return op.nearSingInt(ves, f, lambda F: op.exactStokesSLdiag(ves, G, F), near,
                              op.exactStokesDL if double else op.exactStokesSL, ves, True, precision="fp64")

    ref = potential()
    assert torch.isfinite(ref).all()
    rng = np.random.default_rng(2)
    for k in range(20):
        shuffled(near, np.arange(n)[::-1].copy() if k == 0 else rng.permutation(n))
        assert torch.equal(potential(), ref), k


def test_step_of_two_point_sets_repeats():
    from ves2dpy_gb300 import TStepBiemMixed
    c, r = packed_circles(8, 8, 0.05)
    sets = [np.arange(len(c)) % 2 == q for q in range(2)]
    Xs = [circles(c[m], r[m], N, 0.3) for m, N in zip(sets, (16, 20))]
    # points within the near zone (width: the source set's point distance) of sources of both sets
    p = np.stack([Xs[1][:20].ravel(), Xs[1][20:].ravel()], axis=1)
    dist = np.hypot(*(p[:, None, :] - c[None]).transpose(2, 0, 1)) - r
    dist[:, sets[1]] += 9.0 * np.tile(np.eye(sets[1].sum()), (20, 1))  # the point's own vesicle
    near = [(dist[:, m] < 0.95 * 2 * math.pi / N).any(axis=1) for m, N in zip(sets, (16, 20))]
    assert (near[0] & near[1]).sum() >= 20
    prams = dict(dt=1e-5, kappa=1.0, gmresTol=1e-8, gmresMaxIter=200, farFieldSpeed=1.0, viscCont=1.0, chanWidth=60.0)
    Xs = [T(X) for X in Xs]
    step = TStepBiemMixed(Xs, dict(farField="parabolic", usePreco=True, repulsion=False), prams, near="matlab",
                          farfield_precision="fp32m", sl_precision="fp32c")
    zero = [torch.zeros(X.shape[0] // 2, X.shape[1], dtype=torch.float64, device=DEV) for X in Xs]
    ref = None
    for k in range(20):
        Xn, sig, _, flag = step.time_step(Xs, zero)
        assert not flag
        out = [a.clone() for a in list(Xn) + list(sig)]
        ref = ref or out
        assert all(torch.equal(a, b) for a, b in zip(out, ref)), k


def hedgehog(N, thresh, maxc=32, nrow=5):
    from ves2dpy_gb300 import Poten
    from ves2dpy_gb300.biem_support import NearZone
    from ves2dpy_gb300.capsules import capsules
    from ves2dpy_gb300.layout import to_vm
    X = T(circles(*packed_circles(nrow, nrow, 0.05), N))
    near = NearZone.build_py(to_vm(X), N, thresh=thresh, maxc=maxc)
    f = torch.randn(X.shape, dtype=torch.float64, device=DEV, generator=torch.Generator(device=DEV).manual_seed(3))
    op = Poten(N)
    ves = capsules(X, None, None, 1.0, 1.0)

    def correction():
        """The far field with the correction, and the correction alone, of self velocities f."""
        return op.nearSingInt_hh(ves, f, lambda F: F, near, precision="fp64")

    return X, near, f, correction


def test_hedgehog_stays_in_its_lists():
    """A candidate count above the lists' capacity is read as the capacity."""
    _, near, _, correction = hedgehog(16, 0.2)
    need = int(near.cand_count.max().item())
    _, near, _, correction = hedgehog(16, 0.2, maxc=need)
    assert near.maxc == need
    LP, only = correction()
    near.cand_count[near.cand_count == need] = need + 1000
    LP2, only2 = correction()
    assert torch.equal(LP, LP2) and torch.equal(only, only2) and float(only.abs().max()) > 0


@pytest.mark.parametrize("N, thresh, most", [(16, 0.7, 2), (16, 2.0, 7), (16, 3.0, 13), (32, 1.2, 3)])
def test_hedgehog_adds_in_ascending_order(N, thresh, most):
    """The correction alone, bit for bit, against additions in ascending order
    of the vesicle whose self velocity is added; hedgehog points of up to `most`
    vesicles."""
    X, near, f, correction = hedgehog(N, thresh)
    nv, Nup = X.shape[1], near.Nup
    Xh, fh = X.cpu().numpy(), f.cpu().numpy()
    up = torch.fft.fft(torch.complex(X[:N], X[N:]), dim=0).cpu().numpy()
    pad = np.zeros((Nup, nv), dtype=complex)
    pad[:N // 2], pad[Nup - N // 2:] = up[:N // 2], up[N // 2:]
    z = np.fft.ifft(pad, axis=0) * (Nup / N)
    ref, times = np.zeros((2 * N, nv)), np.zeros((N, nv), dtype=int)
    for id1, t in zip(*near.hh()):  # ascending t
        k2, J = divmod(int(id1), N)
        if k2 >= nv or k2 == t:
            continue
        d2 = (Xh[:N, t] - z[J, k2].real) ** 2 + (Xh[N:, t] - z[J, k2].imag) ** 2
        p = (int(np.argmin(d2)) - 3) % N
        two = np.sort(d2)[:2]
        assert two[1] - two[0] > 1e-9  # no tie decides
        ref[J, k2] += fh[p, t]
        ref[N + J, k2] += fh[N + p, t]
        times[J, k2] += 1
    assert times.max() == most
    LP, only = correction()
    assert np.array_equal(only.cpu().numpy(), ref)
    for _ in range(20):
        LP2, only2 = correction()
        assert torch.equal(LP, LP2) and torch.equal(only, only2)
