"""The work users have this package do, as measurable cases.

A case is a dict of plain values.  ``listed()`` names the fixed ones,
``draw(rng)`` gives more of the same ranges, ``prepare(case, seed)`` makes what
a program holds before the call, ``run(state)`` is one pass through the public
entry points, ``work(case)`` what such a pass cannot do without and
``exact(case, seed)`` the outputs in 64 bits by plain torch where that takes
seconds.

Kinds of case:

* ``biem``   one implicit step, ``TStepBiem.time_step``;
* ``mixed``  one implicit step of a suspension of two point counts,
  ``TStepBiemMixed.time_step``;
* ``mlarm``  one surrogate step, ``MLARM_manyfree_py.time_step_many_noinfo``,
  with the trained networks on the tensor cores;
* ``net``    one network on its own, ``mlarm.Network``;
* ``layer``  one layer potential with its near-singular part,
  ``Poten.nearSingInt``;
* ``far``    one all-pairs sum, ``allExactStokesSLTarget_compare2``;
* ``slmat``  the self-interaction matrices, ``Poten.stokesSLmatrix``;
* ``train``  one training step of one network (forward, backward, Adam).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

DEV = "cuda:0"
UNIT_AREA = 0.65 / (4 * math.pi)   # reduced area 0.65 at unit length, the surrogate's vesicles
UNIT_GAP = 0.05 / 7.79             # the 0.05 gap of vesicles of area pi (length 7.79) at unit length


def listed():
    return [
        # the smallest simulation: the reference's own test size in its own
        # arithmetic (FP64, near rule py_hh), ten thousands of steps long in
        # earnest, so launches and latency are the cost
        dict(name="biem-16xN32-fp64", kind="biem", nv=16, N=32, precision="fp64", near="py_hh", precond="fp64",
             flow="shear", contrast=1.0, tol=1e-10, dt=1e-4),
        # the implicit step at the resolution of the benchmark, on the
        # settings its comparison arm uses
        dict(name="biem-1024xN128", kind="biem", nv=1024, N=128, precision="fp32m", near="py_hh", precond="fp32",
             flow="shear", contrast=1.0, tol=1e-8, dt=1e-5),
        # a large suspension of coarse vesicles in a Taylor-Green flow
        dict(name="biem-8192xN32", kind="biem", nv=8192, N=32, precision="fp32m", near="py_hh", precond="fp64",
             flow="taylorGreen", contrast=1.0, tol=1e-8, dt=1e-5),
        # vesicles more viscous than the fluid (double layer in every matvec), an odd count
        dict(name="biem-301xN64-contrast", kind="biem", nv=301, N=64, precision="fp32m", near="py_hh", precond="fp64",
             flow="shear", contrast=3.0, tol=1e-8, dt=1e-5),
        # an uneven suspension in a channel flow: coarse and fine vesicles in one system
        dict(name="mixed-3000xN32-1000xN128", kind="mixed", nv32=3000, nv128=1000),
        # the headline: the surrogate step of a full suspension
        dict(name="mlarm-4096", kind="mlarm", nv=4096),
        # the surrogate step of a small, odd suspension
        dict(name="mlarm-61", kind="mlarm", nv=61),
        # one network on its own batch, as when networks are judged or tuned
        dict(name="net-adv-128", kind="net", net="adv", nv=128),
        # one layer potential over all vesicles with the MATLAB near rule
        dict(name="layer-1024xN128", kind="layer", nv=1024, N=128, precision="fp32m"),
        # one all-pairs sum between a few hundred vesicles
        dict(name="far-333xN64", kind="far", nv=333, N=64, precision="fp32m"),
        # the self-interaction matrices in the default precision
        dict(name="slmat-200xN96-fp64", kind="slmat", nv=200, N=96, precision="fp64"),
        # one step of surrogate training
        dict(name="train-relax-128", kind="train", net="relax", batch=128),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["biem", "biem", "biem", "mixed", "mlarm", "mlarm", "net", "net", "layer", "far", "slmat", "train"])
    if kind == "biem":
        N = rng.choice([16, 32, 48, 64, 96, 128])
        if rng.random() < 0.25:  # the FP64 form is for small suspensions
            near = rng.choice(["py_hh", "py_rbf", "matlab"])  # the RBF rule's width is set for N = 32
            return dict(kind=kind, nv=_size(rng, 2, 40), N=32 if near == "py_rbf" else rng.choice([16, 32, 48]),
                        precision="fp64", near=near, precond="fp64", flow="shear", contrast=1.0, tol=1e-10, dt=1e-4)
        contrast = rng.choice([1.0, 1.0, 1.0, 3.0])
        hi = {16: 6000, 32: 6000, 48: 4000, 64: 2500, 96: 1200, 128: 900}[N]
        return dict(kind=kind, nv=_size(rng, 8, hi if contrast == 1.0 else hi // 4), N=N, precision="fp32m",
                    near=rng.choice(["py_hh", "matlab"]), precond=rng.choice(["fp32", "fp64"]),
                    flow=rng.choice(["shear", "taylorGreen", "parabolic"]), contrast=contrast, tol=1e-8, dt=1e-5)
    if kind == "mixed":
        return dict(kind=kind, nv32=_size(rng, 20, 3000), nv128=_size(rng, 7, 800))
    if kind == "mlarm":
        return dict(kind=kind, nv=_size(rng, 3, 3000))
    if kind == "net":
        return dict(kind=kind, net=rng.choice(["adv", "advten", "near", "relax", "selften"]), nv=_size(rng, 1, 256))
    if kind == "layer":
        N = rng.choice([32, 64, 128])
        return dict(kind=kind, nv=_size(rng, 16, {32: 8192, 64: 3000, 128: 1500}[N]), N=N,
                    precision=rng.choice(["fp32m", "fp32m", "fp32c"]) if N < 128 else "fp32m")
    if kind == "far":
        return dict(kind=kind, nv=_size(rng, 4, 500), N=rng.choice([16, 32, 64, 96]),
                    precision=rng.choice(["fp32m", "fp32m", "fp32c", "fp64"]))
    if kind == "slmat":
        N = rng.choice([16, 32, 48, 64, 96])
        return dict(kind=kind, nv=_size(rng, 1, {16: 2000, 32: 1500, 48: 900, 64: 500, 96: 220}[N]), N=N,
                    precision=rng.choice(["fp64", "fp32c"]))
    return dict(kind=kind, net=rng.choice(["relax", "selften", "adv", "advten"]), batch=_size(rng, 16, 256))


# ---------------------------------------------------------------------------
# inputs

def _dev(a):
    return torch.tensor(np.asarray(a), dtype=torch.float64, device=DEV)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) % (1 << 62))


@functools.lru_cache(maxsize=16)
def _arrangement(nv, N, unit, fraction):
    from ves2dpy_gb300 import random_suspension
    return random_suspension(nv, N, fraction, min_gap=UNIT_GAP if unit else 0.05,
                             area=UNIT_AREA if unit else math.pi, seed=7)


@functools.lru_cache(maxsize=4)
def _uneven(nv32, nv128):
    from ves2dpy_gb300 import mixed_suspension
    return mixed_suspension([(nv32, 32), (nv128, 128)], 0.20, box_aspect=5.0, min_gap=0.1, reduced_area=(0.6, 0.9),
                            seed=7)


def _moved(X, rng, gap, turn):
    """An arrangement turned by a random angle (``turn``), every vesicle moved
    by up to a quarter of the smallest gap and its first point taken anywhere."""
    N, nv = X.shape[0] // 2, X.shape[1]
    a = rng.uniform(0, 2 * math.pi) if turn else 0.0
    x = math.cos(a) * X[:N] - math.sin(a) * X[N:] + rng.uniform(-0.25 * gap, 0.25 * gap, nv)
    y = math.sin(a) * X[:N] + math.cos(a) * X[N:] + rng.uniform(-0.25 * gap, 0.25 * gap, nv)
    first = (np.arange(N)[:, None] + rng.integers(0, N, nv)) % N
    return np.concatenate((np.take_along_axis(x, first, 0), np.take_along_axis(y, first, 0)))


def _suspension(nv, N, seed, unit=True, fraction=0.15):
    """Vesicles at random places, 15 to 25% of the area, close pairs among them."""
    X = _arrangement(nv, N, unit, fraction)
    return _moved(X, np.random.default_rng(int(seed) % (1 << 31)), UNIT_GAP if unit else 0.05, True)


def _upsampled(X):
    """The upsampled curve and its jacobian, as the callers of the all-pairs sum hold them."""
    from ves2dpy_gb300.biem_support import upsample_factor
    N, nv = X.shape[0] // 2, X.shape[1]
    Nup = upsample_factor(N)
    z = torch.fft.fft(torch.complex(X[:N], X[N:]), dim=0)
    k = torch.fft.fftfreq(N, 1.0 / N, device=X.device, dtype=torch.float64)
    pad = torch.zeros(Nup, nv, dtype=torch.complex128, device=X.device)
    pad[:N // 2], pad[Nup - N // 2:] = z[:N // 2], z[N // 2:]
    kk = torch.zeros(Nup, dtype=torch.float64, device=X.device)
    kk[:N // 2], kk[Nup - N // 2:] = k[:N // 2], k[N // 2:]
    up = torch.fft.ifft(pad, dim=0) * (Nup / N)
    d = torch.fft.ifft(pad * (1j * kk)[:, None], dim=0) * (Nup / N)
    return torch.cat((up.real, up.imag)).contiguous(), d.abs().contiguous()


@functools.lru_cache(maxsize=1)
def _trained():
    from ves2dpy_gb300 import training
    return training.load()


@functools.lru_cache(maxsize=None)
def _network(name):
    from ves2dpy_gb300.mlarm import Network
    return Network(name, _trained()[0][name], "bf16", DEV)


@functools.lru_cache(maxsize=1)
def _surrogate():
    """The surrogate a driver keeps for the whole simulation."""
    from ves2dpy_gb300.curve import Curve
    from ves2dpy_gb300.mlarm import MLARM_manyfree_py
    sds, norms = _trained()
    n = {k: torch.from_numpy(np.asarray(v, dtype=np.float64)) for k, v in norms.items()}

    def vinf(X):  # shear of rate 2
        h = X.shape[0] // 2
        return 2.0 * torch.vstack((X[h:], torch.zeros_like(X[:h])))

    return MLARM_manyfree_py(1e-5, vinf, Curve(), False, 1e2, -1, n["adv_in"], n["adv_out"], n["relax_in"],
                             n["relax_out"], n["near_in"], n["near_out"], n["selften_in"], n["selften_out"],
                             n["advten_in"], n["advten_out"], DEV, state_dicts=sds, net_precision="bf16",
                             farfield_precision="fp32m")


def _train_arrays(case, seed):
    """The trained group's weights, a batch of normalised inputs and targets."""
    from ves2dpy_gb300 import training as T
    spec = T.group_spec(case["net"])
    sd = T.init_state_dict(spec, seed=1 + int(seed) % 1000)
    g = _gen(seed)
    x = torch.randn(case["batch"], spec.blocks[0].cin, spec.L, generator=g, device=DEV)
    t = torch.randn(case["batch"], spec.blocks[-1].cout, spec.L, generator=g, device=DEV)
    return spec, sd, x, t


def _net_input(case, seed):
    from ves2dpy_gb300.mlarm_weights import NETS
    spec = NETS[case["net"]]
    return torch.randn(case["nv"], spec.rep * spec.cin, spec.L, generator=_gen(seed), device=DEV)


def _far_input(case, seed):
    X = _dev(_suspension(case["nv"], case["N"], seed, unit=False, fraction=0.2))
    Xup, sa = _upsampled(X)
    f = torch.randn(Xup.shape, dtype=torch.float64, device=DEV, generator=_gen(seed))
    return X, Xup, sa, f


def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind)
    if kind == "biem":
        from ves2dpy_gb300 import TStepBiem
        nv, N = case["nv"], case["N"]
        if case["precision"] == "fp64":
            X = _dev(_suspension(nv, N, seed, unit=False, fraction=0.2))
        else:
            X = _dev(_suspension(nv, N, seed, fraction=0.25 if case["flow"] == "taylorGreen" else 0.15))
        side = math.sqrt(nv * UNIT_AREA / 0.25)
        prams = dict(dt=case["dt"], kappa=1.0, gmresTol=case["tol"], gmresMaxIter=200, farFieldSpeed=2.0,
                     viscCont=case["contrast"], chanWidth=2 * side, vortexSize=side / 8)
        sl = "fp64" if case["precision"] == "fp64" else "fp32c"
        st["step"] = TStepBiem(X, None, dict(farField=case["flow"], usePreco=True, repulsion=False), prams,
                               near=case["near"], farfield_precision=case["precision"], sl_precision=sl,
                               precond_precision=case["precond"])
        st["X"], st["sig"] = X, torch.zeros(N, nv, dtype=torch.float64, device=DEV)
    elif kind == "mixed":
        from ves2dpy_gb300 import TStepBiemMixed
        rng = np.random.default_rng(int(seed) % (1 << 31))
        Xs = [_dev(_moved(X, rng, 0.1, False)) for X in _uneven(case["nv32"], case["nv128"])]
        prams = dict(dt=1e-5, kappa=1.0, gmresTol=1e-8, gmresMaxIter=200, farFieldSpeed=1.0, chanWidth=60.0,
                     viscCont=1.0)
        st["step"] = TStepBiemMixed(Xs, dict(farField="parabolic", usePreco=True, repulsion=False), prams,
                                    near="matlab", farfield_precision="fp32m", sl_precision="fp32c")
        st["X"] = Xs
        st["sig"] = [torch.zeros(X.shape[0] // 2, X.shape[1], dtype=torch.float64, device=DEV) for X in Xs]
    elif kind == "mlarm":
        from ves2dpy_gb300.curve import Curve
        X = _dev(_suspension(case["nv"], 128, seed))
        cv = Curve()
        _, st["area0"], st["len0"] = cv.geomProp(X)
        for _ in range(10):  # the driver's equal-arclength passes
            X, good = cv.redistributeArcLength(X)
            if good:
                break
        st["step"] = _surrogate()
        st["X"], st["ten"] = X, torch.zeros(128, case["nv"], dtype=torch.float64, device=DEV)
    elif kind == "net":
        st["net"], st["x"] = _network(case["net"]), _net_input(case, seed)
    elif kind == "layer":
        from ves2dpy_gb300 import Poten
        from ves2dpy_gb300.capsules import capsules
        X = _dev(_suspension(case["nv"], case["N"], seed, unit=False, fraction=0.2))
        ves = capsules(X, None, None, 1.0, 1.0)
        st["op"], st["ves"], st["near"] = Poten(case["N"]), ves, ves.getZone()
        st["G"] = st["op"].stokesSLmatrix(ves, "fp32c")
        st["f"] = torch.randn(X.shape, dtype=torch.float64, device=DEV, generator=_gen(seed))
        st["precision"] = case["precision"]
    elif kind == "far":
        st["X"], st["Xup"], st["sa"], st["f"] = _far_input(case, seed)
        st["precision"] = case["precision"]
    elif kind == "slmat":
        from ves2dpy_gb300 import Poten
        from ves2dpy_gb300.capsules import capsules
        X = _dev(_suspension(case["nv"], case["N"], seed, unit=False, fraction=0.2))
        st["op"], st["ves"] = Poten(case["N"]), capsules(X, None, None, 1.0, 1.0)
        st["precision"] = case["precision"]
    elif kind == "train":
        from ves2dpy_gb300.training import Trainer
        spec, sd, st["x"], st["t"] = _train_arrays(case, seed)
        st["trainer"] = Trainer(spec, sd, "fp32", case["batch"], DEV)
    else:
        raise ValueError(kind)
    return st


def run(st):
    kind = st["kind"]
    if kind == "biem":
        X, sig, _, _, _, _ = st["step"].time_step(st["X"], st["sig"])
        return X, sig
    if kind == "mixed":
        Xs, sigs, _, _ = st["step"].time_step(st["X"], st["sig"])
        return Xs, sigs
    if kind == "mlarm":
        m = st["step"]
        m.area0, m.len0 = st["area0"], st["len0"]
        return m.time_step_many_noinfo(st["X"], st["ten"], 3)
    if kind == "net":
        return st["net"](st["x"])
    if kind == "layer":
        op, ves, G = st["op"], st["ves"], st["G"]
        return op.nearSingInt(ves, st["f"], lambda F: op.exactStokesSLdiag(ves, G, F), st["near"], op.exactStokesSL,
                              ves, True, precision=st["precision"])
    if kind == "far":
        from ves2dpy_gb300.biem_support import allExactStokesSLTarget_compare2
        return allExactStokesSLTarget_compare2(st["Xup"], st["sa"], st["f"], st["X"], [], [], [],
                                               precision=st["precision"])
    if kind == "slmat":
        return st["op"].stokesSLmatrix(st["ves"], st["precision"])
    loss = st["trainer"].train_step(st["x"], st["t"], 1e-4, want_loss=True)
    sd = st["trainer"].state_dict()
    return loss, np.concatenate([sd[k].reshape(-1) for k in sorted(sd)])


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _nup(N):
    return N * math.ceil(math.sqrt(N))


def _pairs_flops(targets, sources, precision, Nup):
    """An all-pairs sum: the direct rule's 12 operations per point pair, or the
    series' 6 orders of 32 operations per (target point, source vesicle)."""
    return targets * sources * (6 * 32.0 if precision == "fp32m" else 12.0 * Nup)


def _step_work(nv, N, precision, precond, iters=20):
    """Self matrices and preconditioner blocks made once and read once per
    iteration; an all-pairs sum per iteration."""
    es = 4 if precond == "fp32" else 8
    b = nv * (4 * N * N * 8.0 + 9 * N * N * es) * (iters + 1) + 6 * nv * 3 * N * 8.0
    f = nv * (2.0 / 3.0) * (3 * N) ** 3 + iters * nv * 2.0 * 13 * N * N
    f += iters * _pairs_flops(nv * N, nv, precision, _nup(N))
    return b, f


def _net_flops(spec, groups):
    f = 0
    for b in spec.blocks:
        d, L = 2 * b.c2, spec.L
        f += 2 * (L // 2) * b.c1 * b.cin * 7 + 2 * (L // 4) * b.c2 * 2 * b.c1 * 7
        f += (L // 2) * d * d * 5 + L * d * d * 5 + L * b.cmix * d * 3
    return 2.0 * f * groups


def _net_params(spec):
    return sum(2 * 7 * (b.c1 * b.cin + b.c2 * 2 * b.c1) + 20 * (2 * b.c2) ** 2 + 6 * b.cmix * b.c2 for b in spec.blocks)


def work(case):
    from ves2dpy_gb300.mlarm_weights import NETS
    kind = case["kind"]
    if kind == "biem":
        b, f = _step_work(case["nv"], case["N"], case["precision"], case["precond"])
    elif kind == "mixed":
        n1, n2 = case["nv32"], case["nv128"]
        b1, f1 = _step_work(n1, 32, "fp32m", "fp64")
        b2, f2 = _step_work(n2, 128, "fp32m", "fp64")
        b, f = b1 + b2, f1 + f2 + 20 * (_pairs_flops(n1 * 32, n2, "fp32m", 0) + _pairs_flops(n2 * 128, n1, "fp32m", 0))
    elif kind == "mlarm":
        nv = case["nv"]
        f = sum(_net_flops(s, s.rep) for s in NETS.values()) * nv + 2 * _pairs_flops(nv * 128, nv, "fp32m", 0)
        b = sum(2.0 * _net_params(s) * s.rep for s in NETS.values()) + 8.0 * nv * 128 * 6
    elif kind == "net":
        s = NETS[case["net"]]
        f = _net_flops(s, s.rep) * case["nv"]
        b = 2.0 * _net_params(s) * s.rep + 4.0 * case["nv"] * s.rep * (s.cin + s.cout) * s.L
    elif kind == "layer":
        nv, N = case["nv"], case["N"]
        f = nv * 8.0 * N * N + _pairs_flops(nv * N, nv, case["precision"], _nup(N))
        b = nv * (32.0 * N * N + 6 * N * 8)
    elif kind == "far":
        nv, N, Nup = case["nv"], case["N"], _nup(case["N"])
        f = _pairs_flops(nv * N, nv, case["precision"], Nup)
        b = nv * (5.0 * Nup + 4 * N) * 8
    elif kind == "slmat":
        # per vesicle Nup^2 kernel values of three fields, restricted to N points by fast transforms
        nv, N, Nup = case["nv"], case["N"], _nup(case["N"])
        f = nv * 20.0 * Nup * Nup
        b = nv * (4.0 * N * N + 2 * N) * 8
    else:
        s = NETS[case["net"]]
        f = 3 * _net_flops(s, 1) * case["batch"]
        b = 4.0 * _net_params(s) * 7 + 4.0 * case["batch"] * s.L * (s.cin + s.cout)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# 64 bits by plain torch

def _windows(x, taps, stride):
    """x[G, C, B, P] -> the taps' windows [G, C * len(taps), B * Lout], tap t starting at column t."""
    lout = x.shape[-1] - max(taps)
    lout = (lout + stride - 1) // stride
    cols = [x[..., t:t + stride * (lout - 1) + 1:stride] for t in taps]
    w = torch.stack(cols, dim=2)  # [G, C, T, B, Lout]
    return w.reshape(x.shape[0], -1, x.shape[2] * lout), lout


def _conv(x, w, b, taps, stride):
    """x[G, C, B, P], w[G*O, C, T] -> [G, O, B, Lout]."""
    G, C, B, _ = x.shape
    X, lout = _windows(x, taps, stride)
    y = torch.baddbmm(b.reshape(G, -1, 1), w.reshape(G, -1, C * len(taps)), X)
    return y.reshape(G, -1, B, lout)


def _deconv(x, w, b):
    """Transposed convolution, kernel 10, stride 2, padding 4: w[G*C, O, 10]."""
    G, C, B, P = x.shape
    xp = torch.nn.functional.pad(x, (2, 2))
    w = w.reshape(G, C, -1, 10)
    out = []
    for r in range(2):  # out[2q + r] = sum_u w[r + 2u] x[q + 2 - u]
        wr = torch.stack([w[..., r + 2 * u] for u in (4, 3, 2, 1, 0)], dim=-1)
        out.append(_conv(xp, wr.permute(0, 2, 1, 3).reshape(-1, C, 5), b, (0, 1, 2, 3, 4), 1))
    return torch.stack(out, dim=-1).reshape(G, -1, B, 2 * P)


def _bn(x, W, name):
    G, C = x.shape[:2]
    s = W[name + ".weight"] / torch.sqrt(W[name + ".running_var"] + 1e-5)
    t = W[name + ".bias"] - W[name + ".running_mean"] * s
    return x * s.reshape(G, C, 1, 1) + t.reshape(G, C, 1, 1)


def _forward(spec, W, x):
    """The network in plain torch on x[B, G*C, L]."""
    G, B = spec.rep, x.shape[0]
    x = x.reshape(B, G, -1, spec.L).permute(1, 2, 0, 3)
    circ = functools.partial(torch.nn.functional.pad, mode="circular")

    def pair(v, p, k):
        flat = v.reshape(-1, *v.shape[2:])
        one, two = circ(flat, (3, 3)).reshape(*v.shape[:3], -1), circ(flat, (6, 6)).reshape(*v.shape[:3], -1)
        a = _conv(one, W[p + ".conv%d_1.weight" % k], W[p + ".conv%d_1.bias" % k], range(7), 2)
        b = _conv(two, W[p + ".conv%d_2.weight" % k], W[p + ".conv%d_2.bias" % k], range(0, 14, 2), 2)
        return torch.relu(torch.cat((a, b), dim=1))

    for blk in spec.blocks:
        p = blk.prefix
        b = _bn(pair(_bn(pair(x, p, 1), W, p + ".bn1"), p, 2), W, p + ".bn2")
        c = _bn(torch.relu(_deconv(b, W[p + ".deconv1.weight"], W[p + ".deconv1.bias"])), W, p + ".bn3")
        d = _bn(torch.relu(_deconv(c, W[p + ".deconv2.weight"], W[p + ".deconv2.bias"])), W, p + ".bn4")
        m = _conv(torch.nn.functional.pad(d, (1, 1)), W[p + ".mix.weight"], W[p + ".mix.bias"], (0, 1, 2), 1)
        if blk.residual:
            m = m + x[:, :blk.cmix]
        x = torch.cat((m, x[:, blk.cin - blk.npass:]), dim=1) if blk.npass else m
    return x.permute(2, 0, 1, 3).reshape(B, -1, spec.L)


def _weights64(sd):
    return {k: torch.as_tensor(np.asarray(v)).to(DEV, torch.float64) for k, v in sd.items()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "net":
        from ves2dpy_gb300.mlarm_weights import NETS
        spec = NETS[case["net"]]
        W = _weights64(_trained()[0][case["net"]])
        x = _net_input(case, seed).double()
        return torch.cat([_forward(spec, W, x[i:i + 16]) for i in range(0, x.shape[0], 16)])
    if kind == "far":
        X, Xup, sa, f = _far_input(case, seed)
        nv, N, Nup = case["nv"], case["N"], sa.shape[0]
        if nv * nv * N * Nup > 3e10:
            return None
        f = f * torch.cat((sa, sa)) * (2 * math.pi / Nup)
        out = torch.zeros_like(X)
        for k in range(nv):
            keep = torch.arange(nv, device=X.device) != k
            sx, sy = Xup[:Nup, keep].reshape(-1), Xup[Nup:, keep].reshape(-1)
            fx, fy = f[:Nup, keep].reshape(-1), f[Nup:, keep].reshape(-1)
            dx, dy = X[:N, k, None] - sx, X[N:, k, None] - sy
            r2 = dx * dx + dy * dy
            lg, dot = -0.5 * torch.log(r2), (dx * fx + dy * fy) / r2
            out[:N, k] = (lg @ fx + (dot * dx).sum(1)) / (4 * math.pi)
            out[N:, k] = (lg @ fy + (dot * dy).sum(1)) / (4 * math.pi)
        return out
    if kind == "train":
        spec, sd, x, t = _train_arrays(case, seed)
        W = _weights64(sd)
        learn = [k for k in W if "running" not in k]
        for k in learn:
            W[k].requires_grad_(True)
        loss = ((_forward(spec, W, x.double()) - t.double()) ** 2).mean()
        loss.backward()
        new = {}
        for k in W:  # the first step of Adam
            g = W[k].grad if k in learn else None
            new[k] = W[k].detach() if g is None else W[k].detach() - 1e-4 * g / (g.abs() + 1e-8)
        return float(loss.detach()), torch.cat([new[k].reshape(-1) for k in sorted(new)])
    return None
