"""The FP32 and bf16 residuals of the FP32 weights, wherever the integer pipes or
the FP64 pipe narrowed them: r32 = float(w64 - double(w32)), r16 = bf16(r32),
read entry by entry through applies of unit fields."""
import pytest
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu

TERMS = [(1, 0), (2, 0), (1, 1)]


@pytest.mark.parametrize("scale,eps", [(1.0, None), (1e-17, None), (1e16, None), (1e21, None), (1e-19, None), (1.0, 1e-7)])
def test_residuals_are_the_conversions(cuda, scale, eps):
    pos, h = W.lattice(10, 2, jitter=0.1, seed=93)
    p = torch.tensor(pos * scale, device="cuda")
    h *= scale
    n = p.shape[0]
    plan = DcpsePlan(2, [[s] for s in TERMS])
    plan.build_neighbors(p, 3.1 * h)
    plan.assemble(p, C.ASSEMBLE_FAST | C.STORE_OUT_F64 | C.STORE_OUT_F32 | C.STORE_OUT_F32_CORR | C.STORE_OUT_F32_RESID,
                  eps_fixed=None if eps is None else torch.full((n,), eps * h, dtype=torch.float64, device="cuda"))
    plan.set_error_budget(1e-300)  # every row is corrected by its r32
    rp, cols = plan.neighbors()
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), rp[1:] - rp[:-1])
    got = {C.F32_BUDGET: [], C.F32_RESID: []}
    for prec in got:
        at = torch.empty((len(TERMS), n, n), dtype=torch.float64, device="cuda")
        for q in range(n):
            f = torch.zeros(n, dtype=torch.float64, device="cuda")
            f[q] = 1.0
            at[:, :, q] = plan.apply(f, prec)
        got[prec] = at[:, rows, cols.long()]
    torch.cuda.synchronize()
    seen = 0
    for o in range(len(TERMS)):
        w64, w32 = (x.clone() for x in plan.output_weights(o))
        r32 = (w64 - w32.double()).float()
        # (an entry that overflows makes every entry of its row NaN)
        fine = torch.zeros(n, device="cuda").index_add_(0, rows, (~torch.isfinite(w32)).float())[rows] == 0
        seen += int(fine.sum())
        # one product with 1, the others with 0: exact; w32 + r32 spans 49 bits
        assert torch.equal(got[C.F32_BUDGET][o][fine], (w32.double() + r32.double())[fine])
        assert torch.equal(got[C.F32_RESID][o][fine], (w32.double() + r32.bfloat16().double())[fine])
    assert seen > 0
    plan.close()
