"""Neighbour builds at the ends of their ranges, bit for bit against the oracle
or against the two-pass search."""
import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import workloads as W  # noqa: F401
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu


def _build(pos, rcut, box=None, rcut_pp=None, self_skip=True):
    dim = pos.shape[1]
    plan = DcpsePlan(dim, [[(1,) + (0,) * (dim - 1)]], box=box)
    if not self_skip:
        plan.set_support(None, self_skip=False)
    plan.build_neighbors(torch.tensor(pos, device="cuda"), rcut,
                         None if rcut_pp is None else torch.tensor(rcut_pp, device="cuda"))
    rp, cols = (x.cpu().numpy() for x in plan.neighbors())
    plan.close()
    return rp, cols


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("rcut", [4.0, 1e25, 1e200, float("inf")])
def test_cutoffs_beyond_the_set(cuda, dim, rcut):
    """Every particle is everybody's neighbour, also where the cutoff, its
    square or the expected number of neighbours is infinite."""
    n = 301
    pos = np.random.default_rng(71).random((n, dim))
    rp, cols = _build(pos, rcut)
    every = np.arange(n)
    assert np.array_equal(rp, np.arange(n + 1) * (n - 1))
    assert np.array_equal(cols.reshape(n, n - 1), np.array([np.delete(every, p) for p in range(n)]))
