"""The implicit step where the factorisation of its preconditioner changes its
split: 3N = 126 and 132 unknowns per vesicle around the step from 128 to 256
threads, 252 and 258 around the one from one panel row per thread to two, 438
near the largest FP64 size, 516 with four rows per thread in FP32; all but two
with a last panel and tiles of fewer than 32 columns.  Against the FP64 oracle
step; GMRES stops at a relative residual of 1e-10, which the block-diagonal
preconditioner keeps within a factor of ten in the positions."""
import numpy as np
import pytest
import torch

from oracle import ves2d_oracle as O

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


@pytest.mark.parametrize("N,precond", [(42, "fp64"), (44, "fp32"), (84, "fp64"), (86, "fp64"), (86, "fp32"),
                                       (146, "fp64"), (172, "fp32")])
def test_step_matches_oracle(N, precond):
    from ves2dpy_gb300.suspension import lattice_suspension
    from ves2dpy_gb300.tstep_biem import TStepBiem
    X = lattice_suspension(2, N, spacing=2.2, jitter=0.05, min_gap=0.02, reduced_area=0.9, seed=3)
    nv = X.shape[1]
    ref = O.time_step(X, np.zeros((N, nv)), O.StepParams(dt=1e-4, speed=2.0), O.PotenTables(N))
    t = lambda a: torch.tensor(a, dtype=torch.float64, device=DEV)  # noqa: E731
    prams = dict(dt=1e-4, kappa=1.0, gmresTol=1e-10, gmresMaxIter=200, farFieldSpeed=2.0, viscCont=[1.0] * nv)
    tt = TStepBiem(t(X), None, dict(farField="shear", usePreco=True, repulsion=False), prams, near="py_hh",
                   farfield_precision="fp64", sl_precision="fp64", precond_precision=precond)
    Xn, sn, _, _, it, iflag = tt.time_step(t(X), torch.zeros(N, nv, dtype=torch.float64, device=DEV))
    assert not iflag
    assert np.abs(Xn.cpu().numpy() - ref.X).max() <= 1e-9 * np.abs(ref.X).max()
