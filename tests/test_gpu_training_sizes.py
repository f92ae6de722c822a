"""The trainer's convolutions at lengths whose rows are not whole vectors (20 and
120: quarter lengths 5 and 30) beside one where they are (48), one sample and
several per CTA.  FP64 against autograd of the oracle's forward pass at
1e-10 and FP32 at 5e-3 of each gradient's 2-norm (both as tests/test_gpu_training.py)."""
import dataclasses

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("L,B", [(20, 3), (120, 2), (48, 130), (20, 310)])
def test_gradients(L, B):
    from oracle import mlarm_oracle as M
    from ves2dpy_gb300 import training as T
    spec = dataclasses.replace(T.group_spec("relax"), L=L)
    sd = T.init_state_dict(spec, seed=5)
    rng = np.random.default_rng(L)
    x, t = torch.from_numpy(rng.normal(size=(B, spec.cin, L))), torch.from_numpy(rng.normal(size=(B, spec.cout, L)))
    grads = {}
    for prec in ("fp64", "fp32"):
        tr = T.Trainer(spec, sd, prec, B, DEV)
        tr.forward(x)
        tr.backward(t)
        grads[prec] = tr.grads_f64() if prec == "fp64" else tr.grads()
    W = {k: torch.tensor(np.asarray(v, dtype=np.float64),
                         requires_grad=not k.endswith(("running_mean", "running_var"))) for k, v in sd.items()}
    ((M.net_forward_t(spec, W, x) - t) ** 2).mean().backward()
    off = 0
    for b in spec.blocks:
        for key in T.ORDER:
            w = W[f"{b.prefix}.{key}"]
            n = w.numel()
            if w.requires_grad:
                ref, name = w.grad.numpy().reshape(-1), f"{b.prefix}.{key}"
                err = np.abs(grads["fp64"][off:off + n] - ref).max() / max(np.abs(ref).max(), 1e-300)
                assert err < 1e-10, (name, err)
                diff = np.linalg.norm(np.asarray(grads["fp32"][name]).reshape(-1) - ref)
                assert diff <= 5e-3 * max(np.linalg.norm(ref), 1e-30), (name, diff)
            off += n
