"""Position VJP through the split kernels (Gram with the extra column, QR of
two right-hand sides, chain rule): rows of one to five chunks of 32 entries,
one to three basis groups, a row that cannot be assembled, several QR lane
groupings, against the oracle's reference adjoint at its 1e-9 bar; a fixed eps
against central differences."""
import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nside,rc,outputs", [
    (1, 40, 4.3, [[(1,)], [(2,)]]),
    (2, 17, 3.1, [[(1, 1)]]),
    (2, 17, 4.2, [[(1, 0)], [(2, 0), (0, 2)], [(2, 1)]]),
    (3, 9, 2.8, W.grad_lap_outputs(3)),
    (3, 11, 3.4, [[(2, 0, 0), (0, 2, 0), (0, 0, 2)]]),
])
@pytest.mark.parametrize("lanes", [0, 8])
def test_split_vjp_vs_reference_adjoint(cuda, orc, dim, nside, rc, outputs, lanes):
    pos, h = W.lattice(nside, dim, jitter=0.1, seed=70 + dim)
    inside = W.interior_mask(pos, rc * h)
    # one particle out of everybody's reach: no neighbours, no gradient
    pos = np.vstack([pos, np.full((1, dim), 9.0)])
    inside = np.append(inside, True)
    n = pos.shape[0]
    rng = np.random.default_rng(71)
    f, g = rng.standard_normal(n), rng.standard_normal((len(outputs), n)) * inside
    plan = DcpsePlan(dim, outputs)
    plan.set_assembly_config(qr_lanes=lanes)
    pt = torch.tensor(pos, device="cuda")
    plan.build_neighbors(pt, rc * h)
    rp, cols = (x.cpu().numpy() for x in plan.neighbors())
    got = plan.vjp_positions(pt, torch.tensor(f, device="cuda"), torch.tensor(g, device="cuda")).cpu().numpy()
    g[:, -1] = 0.0  # (the adjoint of a row without neighbours is not defined)
    ref = orc.vjp_positions(pos, rp, cols, outputs, f, g)
    assert np.all(got[-1] == 0.0)
    assert np.abs(got - ref).max() <= 1e-9 * np.abs(ref).max()
    plan.close()


def test_split_vjp_fixed_eps(cuda):
    pos, h = W.lattice(14, 2, jitter=0.1, seed=75)
    outputs = [[(2, 0), (0, 2)], [(1, 0)]]
    inside = W.interior_mask(pos, 3.1 * h)
    n = pos.shape[0]
    rng = np.random.default_rng(76)
    f = torch.tensor(rng.standard_normal(n), device="cuda")
    g = torch.tensor(rng.standard_normal((2, n)) * inside, device="cuda")
    eps = torch.tensor(h * rng.uniform(1.4, 2.0, n), device="cuda")
    plan = DcpsePlan(2, outputs)
    pt = torch.tensor(pos, device="cuda")
    plan.build_neighbors(pt, 3.1 * h)
    ad = plan.vjp_positions(pt, f, g, eps_fixed=eps).cpu().numpy()

    def phi(P):
        plan.assemble(P, C.ASSEMBLE_FAST | C.STORE_OUT_F64, eps_fixed=eps)
        return plan.apply(f, C.F64) * g

    fd = []
    coords = rng.choice(2 * n, 40, replace=False)
    for c in coords:
        i, d = divmod(int(c), 2)
        P, M = pt.clone(), pt.clone()
        P[i, d] += 1e-6 * h
        M[i, d] -= 1e-6 * h
        fd.append(float((phi(P) - phi(M)).sum()) / (2e-6 * h))
    fd = np.array(fd)
    got = ad[coords // 2, coords % 2]
    assert np.abs(fd - got).max() <= 1e-5 * np.abs(fd).max()
    plan.close()
