"""A NaN in a factor, a right-hand side or a matrix is reported, never taken for a
solution: the norms of the stopping test keep it."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,at", [(1, 0), (33, 0), (1000, 999), (70001, 40000)])
def test_infnorm_keeps_nan(mxp, torch_cuda, n, at):
    torch = torch_cuda
    x = torch.ones(n, dtype=torch.float64, device="cuda")
    ws = mxp.Workspace(max(n, 64), 64, 0)
    for v in (float("nan"), float("-inf")):
        x[at] = v
        got = mxp.infnorm(x, ws)
        assert math.isnan(got) if math.isnan(v) else got == math.inf


@pytest.mark.parametrize("chain", [False, True])
def test_refinement_with_nan_in_the_factor(mxp, torch_cuda, chain):
    """Both triangular solves hand the NaN on; the next residual is all NaN."""
    p = mxp.panel_matgen(512, 3)
    ws = mxp.Workspace(512, 128, 0)
    mxp.panel_lu(p, 128, ws)
    if chain:
        ws.set_option(mxp.OPT_TRSV_INV, 0)
    p.A[511] = float("nan")  # L(511, 0)
    x, st, status = mxp.iterative_refinement(p, ws, raise_on_fail=False)
    assert status == mxp.NONFINITE and st["converged"] == 0 and math.isnan(st["residual"])


@pytest.mark.parametrize("higham", [False, True])
def test_refinement_with_nan_in_the_right_hand_side(mxp, torch_cuda, higham):
    n, b = 512, 128
    ws = mxp.Workspace(n, b, 0)
    if higham:
        alpha, beta = mxp.higham_params(n)
        p = mxp.higham_matgen(n, alpha, beta)
        ws.set_matrix_higham(alpha, beta)
    else:
        p = mxp.panel_matgen(n, 3)
    mxp.panel_lu(p, b, ws)
    p.rhs[100] = float("nan")
    x, st, status = mxp.iterative_refinement(p, ws, raise_on_fail=False)
    assert status == mxp.NONFINITE and st["converged"] == 0


@pytest.mark.parametrize("where", ["matrix", "rhs", "d"])
def test_batch_system_with_nan(mxp, torch_cuda, where):
    """The system that holds the NaN is not converged (and its pivots are reported
    when the matrix holds it); the others are solved."""
    bt = mxp.Batch([256, 384, 128], [4, 5, 6])
    bt.set_config(64, 128, 3)
    bt.matgen()
    if where == "matrix":
        bt.matrix(1)[3, 200] = float("nan")
    else:
        bt.vec(getattr(bt, where), 1)[7] = float("nan")
    bt.solve()
    got = bt.results()
    assert got[1]["converged"] == 0 and math.isnan(got[1]["hpl_harness"])
    assert (got[1]["info"] > 0) == (where == "matrix")
    for i in (0, 2):
        assert got[i]["converged"] == 1 and got[i]["hpl_harness"] < 16.0 and got[i]["info"] == 0
    bt.close()
