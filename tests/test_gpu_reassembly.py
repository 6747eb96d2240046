"""Re-assembly on one list: the sliced layout stays and its weight buffers are
used again; every precision gives the bits of a plan assembled once, also when
the stored weights, the numbering or the stream change in between."""
import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu

ALL = C.ASSEMBLE_FAST | C.STORE_OUT_F64 | C.STORE_OUT_F32 | C.STORE_OUT_F32_RESID | C.STORE_OUT_F32_CORR


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("first", [ALL, C.ASSEMBLE_FAST | C.STORE_OUT_F32, C.ASSEMBLE_FAST | C.STORE_OUT_F64])
def test_reassembly_matches_a_fresh_plan(cuda, shuffled, first):
    rng = np.random.default_rng(61)
    pos, h = W.lattice(15, 3, jitter=0.1, seed=62)
    if shuffled:
        pos = pos[rng.permutation(pos.shape[0])]
    moved = pos + rng.uniform(-0.02 * h, 0.02 * h, pos.shape)
    p0, p1 = torch.tensor(pos, device="cuda"), torch.tensor(moved, device="cuda")
    f = torch.tensor(rng.standard_normal(pos.shape[0]), device="cuda")
    g = torch.tensor(rng.standard_normal((4, pos.shape[0])), device="cuda")

    def applies(plan):
        out = [plan.apply(f, p) for p in (C.F32, C.F32_RESID, C.F32_PAIR, C.F32_BUDGET, C.F64)]
        return out + [plan.vjp_field(g, C.F64), plan.vjp_field(g, C.F32)]

    fresh = DcpsePlan(3, W.grad_lap_outputs(3))
    fresh.build_neighbors(p0, 2.8 * h)
    fresh.assemble(p1, ALL)
    ref = applies(fresh)
    plan = DcpsePlan(3, W.grad_lap_outputs(3))
    plan.build_neighbors(p0, 2.8 * h)
    plan.assemble(p0, first)
    for prec, need in ((C.F32, C.STORE_OUT_F32), (C.F64, C.STORE_OUT_F64)):
        if first & need:
            plan.apply(f, prec)
    for stream in (None, torch.cuda.Stream()):
        torch.cuda.synchronize()
        plan.set_stream(stream)
        plan.assemble(p1, ALL)
        got = applies(plan)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, ref))
    # numbering policy changed between assemblies: the layout is built again
    plan.set_reorder(-1 if shuffled else 1)
    plan.assemble(p1, ALL)
    got = applies(plan)
    torch.cuda.synchronize()
    assert plan.reorder_info()[0] == (not shuffled)
    assert all(torch.equal(a, b) for a, b in zip(got, ref))
    # weights no longer stored are gone
    plan.assemble(p1, C.ASSEMBLE_FAST | C.STORE_OUT_F64)
    with pytest.raises(C.DcpseError):
        plan.apply(f, C.F32)
    got = plan.apply(f, C.F64)
    torch.cuda.synchronize()
    assert torch.equal(got, ref[4])
    plan.close()
    fresh.close()
