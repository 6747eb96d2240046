"""Weights kernel on and off the integer pipes: unjittered lattices (monomials
that are zero), offsets and coefficients outside the integer products' range,
FP32 weights that are denormal or overflow, rows concatenated over the particles of
a warp in list and binned order.  Kernels bit for bit against the oracle, the
FP32 weights and residuals against the FP64 ones' conversions."""
import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu

TERMS = [(1, 0), (0, 1), (2, 0), (0, 2), (1, 1)]


@pytest.mark.parametrize("nside,jitter,scale,eps,bins", [
    (12, 0.1, 1.0, None, 0),
    (13, 0.0, 1.0, None, 4),
    (12, 0.1, 1e-60, None, 0),      # eps^-2 beyond 2^257
    (12, 0.1, 1e21, None, 0),       # weights that are denormal floats
    (12, 0.1, 1.0, 2e5, 0),         # u below 2^-16
    (12, 0.1, 1.0, 1e-7, 0),        # u above 2^17: weights that are zero
    (8, 0.0, 1.0, 2e30, 16),        # coefficients beyond 2^101
])
def test_weights_bitexact_in_every_range(cuda, orc, nside, jitter, scale, eps, bins):
    pos, h = W.lattice(nside, 2, jitter=jitter, seed=91)
    pos, h = pos * scale, h * scale
    n = pos.shape[0]
    epsv = None if eps is None else np.full(n, h * eps)
    plan = DcpsePlan(2, [[s] for s in TERMS])
    plan.set_assembly_config(bin_width=bins)
    pt = torch.tensor(pos, device="cuda")
    plan.build_neighbors(pt, 3.1 * h)
    plan.assemble(pt, C.STORE_TERMS_F64 | C.STORE_OUT_F64 | C.STORE_OUT_F32 | C.STORE_OUT_F32_CORR
                  | C.STORE_OUT_F32_RESID, eps_fixed=None if epsv is None else torch.tensor(epsv, device="cuda"))
    rp, cols = (x.cpu().numpy() for x in plan.neighbors())
    for t, sig in enumerate(TERMS):
        _, eip, K, _ = orc.assemble(pos, rp, cols, sig, 2, eps_fixed=epsv)
        k, e = (x.cpu().numpy() for x in plan.term_kernels(t))
        assert np.array_equal(k, K, equal_nan=True) and np.array_equal(e, eip, equal_nan=True), (sig, t)
        w64, w32 = plan.output_weights(t)
        assert torch.equal(torch.nan_to_num(w64.float(), nan=7.0), torch.nan_to_num(w32, nan=7.0))
    plan.close()
