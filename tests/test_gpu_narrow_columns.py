"""16-bit columns of the sliced layout (long lists): the FP32 apply against the
bound pass of the error-budget apply, which sums the same terms from the 32-bit
columns, bit for bit: lattice order (every slice narrow), no order at all (none),
renumbered (some), lists with the particle itself, one to four outputs; and a
Gray-Scott step and its adjoint against the CSR kernels."""
import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.odeint import GrayScottRK4
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu

LAP = [[(2, 0, 0), (0, 2, 0), (0, 0, 2)]]


@pytest.mark.parametrize("outputs", [LAP, LAP + [[(1, 0, 0)]], LAP + [[(1, 0, 0)], [(0, 1, 0)]], W.grad_lap_outputs(3)])
@pytest.mark.parametrize("shuffled,reorder,self_skip", [(False, 0, True), (True, -1, True), (True, 0, True),
                                                        (False, 0, False)])
def test_narrow_apply_matches_the_wide_columns(cuda, outputs, shuffled, reorder, self_skip):
    pos, h = W.lattice(61, 3, jitter=0.1, seed=51)
    rng = np.random.default_rng(52)
    if shuffled:
        pos = pos[rng.permutation(pos.shape[0])]
    pt = torch.tensor(pos, device="cuda")
    f = torch.tensor(rng.standard_normal(pos.shape[0]), device="cuda")
    plan = DcpsePlan(3, outputs)
    plan.set_support(None, self_skip=self_skip)
    plan.set_reorder(reorder)
    plan.build_neighbors(pt, 2.8 * h)
    plan.assemble(pt, C.ASSEMBLE_FAST | C.STORE_OUT_F32 | C.STORE_OUT_F32_CORR)
    assert plan.info()["nnz"] * (4 + 4 * len(outputs)) > 128 << 20
    plan.set_error_budget(0.9)  # no row is corrected
    wide = plan.apply(f, C.F32_BUDGET)
    for schedule in (0, C.APPLY_SLICE_WINDOWS, C.APPLY_SLICE_WARPS):
        plan.set_apply_config(0, schedule)
        assert torch.equal(torch.nan_to_num(plan.apply(f, C.F32), nan=5.0), torch.nan_to_num(wide, nan=5.0))
    plan.close()


def test_gray_scott_narrow_against_csr(cuda):
    nside = 60
    h = 1.0 / nside
    pos, _ = W.lattice(nside, 3, h=h, jitter=0.1, seed=53)
    pos = np.mod(pos, 1.0)
    plan = DcpsePlan(3, LAP, box=((0.0,) * 3, (1.0,) * 3, (1, 1, 1)))
    pt = torch.tensor(pos, device="cuda")
    plan.build_neighbors(pt, 2.8 * h)
    plan.assemble(pt, C.ASSEMBLE_FAST | C.STORE_OUT_F32)
    assert plan.info()["nnz"] * 8 > 128 << 20
    u0, v0 = (torch.tensor(x, device="cuda", dtype=torch.float32) for x in W.gray_scott_initial(pos))
    got = []
    for mode in (0, 1):  # sliced, CSR
        plan.set_apply_config(0, mode)
        gs = GrayScottRK4(plan, u0, v0, 2e-5, 1e-5, 0.04, 0.06, 0.2 * h * h / 2e-5)
        for _ in range(2):
            gs.step()
        ub, vb = gs.backward([(u0, v0)], 2, (torch.zeros_like(u0), torch.ones_like(v0)))
        got.append([x.double().clone() for x in (gs.u, gs.v, ub, vb)])
    for a, b in zip(*got):
        # 92 FP32 terms in another order, ten Laplacians deep
        assert (a - b).abs().max() <= 2e-5 * b.abs().max()
    plan.close()
