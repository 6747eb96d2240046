"""The warp-scheduled sliced kernels: a warp's first slice is its own index, the
others come from a counter.  Bit-identical to one window of 8 slices per block
where the slices number fewer than the grid's warps (a window, and almost all
warps of the chip) and a few more than those."""
import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu


# five outputs: four blocks of 8 warps per SM, 4,864 slices of 32 rows at once on 152 SMs
@pytest.mark.parametrize("side", [14, 394, 396, 500])
def test_slices_around_the_grid(cuda, side):
    pos_np, h = W.lattice(side, 2, jitter=0.15, seed=side)
    pos = torch.tensor(pos_np, device="cuda")
    plan = DcpsePlan(2, W.five_ops_2d(), order=2)
    plan.build_neighbors(pos, 2.8 * h)
    plan.assemble(pos, C.ASSEMBLE_FAST | C.STORE_OUT_F32 | C.STORE_OUT_F32_CORR)
    f = torch.tensor(np.sin(3 * pos_np[:, 0]) * np.cos(2 * pos_np[:, 1]), device="cuda")
    for prec in (C.F32, C.F32_PAIR):
        plan.set_apply_config(0, C.APPLY_SLICE_WINDOWS)
        want = plan.apply(f, prec).clone()
        plan.set_apply_config(0, C.APPLY_SLICE_WARPS)
        for _ in range(2):  # the counter starts again
            assert torch.equal(plan.apply(f, prec), want)
    plan.close()
