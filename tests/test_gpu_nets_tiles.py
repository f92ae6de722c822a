"""The tensor-core network kernels at vesicle counts off their tiles of two and
four vesicles: a vesicle's output is the same bits whatever batch it is in,
and agrees with the FP64 engine to the BF16 tolerance of the suite."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["relax", "selften", "adv", "advten", "near"])
def test_batches_around_a_tile(name):
    from ves2dpy_gb300.mlarm import Network
    from ves2dpy_gb300.mlarm_weights import NETS, net_test_input, synthetic_state_dict
    sd = synthetic_state_dict(name, 0)
    x = torch.from_numpy(net_test_input(name, nv=9, seed=4)).to("cuda:0")
    net = Network(name, sd, "bf16", "cuda:0")
    whole = net(x)
    for nv in (1, 2, 3, 5, 8):
        assert torch.equal(net(x[:nv].contiguous()), whole[:nv]), nv
    fixed = Network(name, sd, "bf16", "cuda:0", autotune=False)
    assert torch.equal(fixed(x), whole)
    ref = Network(name, sd, "fp64", "cuda:0")(x[:2].contiguous())
    assert float((whole[:2].double() - ref).abs().max()) <= 3e-2 * float(ref.abs().max())
