"""Reference-order applies: runs of one to five terms of both signs, and fields
whose differences leave the integer product's range (zero, tiny, huge,
non-finite), bit for bit against the oracle."""
import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import _capi as C
from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu

OUTPUTS = [
    [(1, 1)],
    [(2, 0), (0, 2)],
    [(1, 0), (0, 1), (2, 0), (0, 2), (1, 1)],  # two odd terms, then three even ones
    [(2, 0), (0, 2), (1, 1), (2, 0)],          # a run longer than one launch takes
    [(2, 0), (1, 0), (0, 2)],                  # the sign changes twice
]


@pytest.mark.parametrize("kind", ["smooth", "constant", "tiny", "huge", "mixed"])
def test_terms_bitexact(cuda, orc, kind):
    pos, h = W.lattice(21, 2, jitter=0.1, seed=81)
    n = pos.shape[0]
    rng = np.random.default_rng(82)
    f = {"smooth": np.sin(5 * pos[:, 0]) * pos[:, 1], "constant": np.full(n, 0.1),
         "tiny": rng.standard_normal(n) * 1e-290, "huge": rng.standard_normal(n) * 1e290,
         "mixed": rng.standard_normal(n) * 10.0 ** rng.integers(-300, 280, n)}[kind]
    if kind == "mixed":
        f[::7] = 0.0
        f[5], f[200] = np.inf, np.nan
    pt, ft = torch.tensor(pos, device="cuda"), torch.tensor(f, device="cuda")
    for sigs in OUTPUTS:
        plan = DcpsePlan(2, [[(0, 1)], sigs])
        plan.build_neighbors(pt, 3.1 * h)
        plan.assemble(pt, C.STORE_TERMS_F64)
        rp, cols = (x.cpu().numpy() for x in plan.neighbors())
        Ks, es = zip(*[[x.cpu().numpy() for x in plan.term_kernels(1 + t)] for t in range(len(sigs))])
        got = plan.apply_output_f64(1, ft).cpu().numpy()
        with np.errstate(all="ignore"):
            ref = orc.apply_sum(f, rp, cols, list(Ks), list(es), [sum(s) for s in sigs])
        assert np.array_equal(got, ref, equal_nan=True), (sigs, kind)
        plan.close()


@pytest.mark.parametrize("ncomp", [1, 3])
def test_p2p_bitexact_out_of_range(cuda, orc, ncomp):
    sup, h = W.lattice(15, 2, jitter=0.1, seed=83)
    dom = sup[30:180:3] + 0.3 * h
    rng = np.random.default_rng(84)
    f = rng.standard_normal((sup.shape[0], ncomp)) * 10.0 ** rng.integers(-300, 280, (sup.shape[0], ncomp))
    f[::5] = 0.0
    plan = DcpsePlan(2, [[(0, 0)]])
    plan.set_support(torch.tensor(sup, device="cuda"))
    dt = torch.tensor(dom, device="cuda")
    plan.build_neighbors(dt, 3.1 * h)
    plan.assemble(dt, C.STORE_TERMS_F64)
    rp, cols = (x.cpu().numpy() for x in plan.neighbors())
    K, e = (x.cpu().numpy() for x in plan.term_kernels(0))
    got = plan.p2p_f64(0, torch.tensor(f if ncomp > 1 else f[:, 0], device="cuda")).cpu().numpy().reshape(-1, ncomp)
    for c in range(ncomp):
        ref = orc.p2p(np.ascontiguousarray(f[:, c]), rp, cols, K, e)
        assert np.array_equal(got[:, c], ref)
    plan.close()
