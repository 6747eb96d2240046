"""16-bit columns of an interpolation between two sets (rows and columns of
different sets, a column may equal its row's index): the sliced FP32 kernel
against the CSR kernel, which reads the list itself."""
import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("ncomp", [1, 2])
def test_interpolation_through_narrow_columns(cuda, shuffled, ncomp):
    side = 62
    sup, h = W.lattice(side, 3, jitter=0.1, seed=91)
    dom, _ = W.lattice(side - 2, 3, h=h, origin=0.7 * h)
    rng = np.random.default_rng(92)
    if shuffled:  # (few slices fit 16 bits: the 32-bit columns serve)
        sup = sup[rng.permutation(sup.shape[0])]
    f = torch.tensor(rng.standard_normal((sup.shape[0], ncomp)), device="cuda")
    plan = DcpsePlan(3, [[(0, 0, 0)]])
    plan.set_support(torch.tensor(sup, device="cuda"))
    pd = torch.tensor(dom, device="cuda")
    plan.build_neighbors(pd, 2.8 * h)
    assert plan.info()["nnz"] * 8 > 128 << 20
    plan.assemble(pd, C.ASSEMBLE_FAST | C.STORE_OUT_F32)
    got = plan.p2p(f, C.F32)
    plan.set_apply_config(0, 1)
    ref = plan.p2p(f, C.F32)
    torch.cuda.synchronize()
    # the same FP32 products of about 90 entries of order one, summed in another
    # order: 90 ulps of 2^-24 at most on either side
    rp, cols = plan.neighbors()
    rows = torch.repeat_interleave(torch.arange(dom.shape[0], device="cuda"), rp[1:] - rp[:-1])
    w = plan.output_weights(0)[1].double().abs()
    terms = torch.zeros(dom.shape[0], ncomp, dtype=torch.float64, device="cuda")
    terms.index_add_(0, rows, w[:, None] * f[cols.long()].abs())
    bound = 2 * 90 * 2.0 ** -24 * terms
    assert (got[0] - ref[0]).abs().le(bound).all()
    plan.close()
