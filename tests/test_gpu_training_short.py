"""The trainer at the shortest rows that circular padding allows (12 points: the
second pair of convolutions sees rows as long as its padding of 6), FP64
against autograd of the oracle's forward pass at 1e-10 (as
tests/test_gpu_training_sizes.py), and its refusal of shorter ones."""
import dataclasses

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("L", [4, 8])
def test_shorter_rows_are_refused(L):
    from ves2dpy_gb300 import training as T
    spec = dataclasses.replace(T.group_spec("relax"), L=L)
    with pytest.raises(Exception, match="circular padding"):
        T.Trainer(spec, T.init_state_dict(spec, seed=5), "fp32", 2, DEV)


@pytest.mark.parametrize("B", [1, 5])
def test_gradients_of_the_shortest_rows(B):
    from oracle import mlarm_oracle as M
    from ves2dpy_gb300 import training as T
    spec = dataclasses.replace(T.group_spec("relax"), L=12)
    sd = T.init_state_dict(spec, seed=5)
    rng = np.random.default_rng(B)
    x, t = torch.from_numpy(rng.normal(size=(B, spec.cin, 12))), torch.from_numpy(rng.normal(size=(B, spec.cout, 12)))
    tr = T.Trainer(spec, sd, "fp64", B, DEV)
    tr.forward(x)
    tr.backward(t)
    grads = tr.grads_f64()
    W = {k: torch.tensor(np.asarray(v, dtype=np.float64),
                         requires_grad=not k.endswith(("running_mean", "running_var"))) for k, v in sd.items()}
    ((M.net_forward_t(spec, W, x) - t) ** 2).mean().backward()
    off = 0
    for b in spec.blocks:
        for key in T.ORDER:
            w = W[f"{b.prefix}.{key}"]
            if w.requires_grad:
                ref = w.grad.numpy().reshape(-1)
                err = np.abs(grads[off:off + w.numel()] - ref).max() / max(np.abs(ref).max(), 1e-300)
                assert err < 1e-10, (b.prefix, key, err)
            off += w.numel()
