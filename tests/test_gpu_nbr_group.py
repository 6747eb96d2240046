"""Neighbour search by groups of cells, bit for bit against the oracle: groups
of one, two and four cells, odd cell counts, periodic axes down to the fewest
cells it takes, rows longer than the staging rows, uneven radii, exact ties,
particles outside the box, lists with the particle itself."""
import numpy as np
import pytest
import torch

from openfpm_numerics_gb300 import workloads as W
from openfpm_numerics_gb300.plan import DcpsePlan

pytestmark = pytest.mark.gpu


def _check(orc, pos, rcut, box=None, rcut_pp=None, self_skip=True):
    dim = pos.shape[1]
    plan = DcpsePlan(dim, [[(1,) + (0,) * (dim - 1)]], box=box)
    if not self_skip:
        plan.set_support(None, self_skip=False)
    plan.build_neighbors(torch.tensor(pos, device="cuda"), rcut,
                         None if rcut_pp is None else torch.tensor(rcut_pp, device="cuda"))
    rp, cols = (x.cpu().numpy() for x in plan.neighbors())
    erp, ecols = orc.neighbors(pos, rcut, rcut_pp=rcut_pp, box=box, self_skip=self_skip)
    assert np.array_equal(rp, erp) and np.array_equal(cols, ecols)
    assert plan.info()["max_neighbors"] == (int(np.diff(erp).max()) if pos.shape[0] else 0)
    plan.close()


@pytest.mark.parametrize("dim,nside,jitter", [(2, 9, 0.1), (2, 90, 0.3), (2, 257, 0.1), (2, 260, 0.0),
                                              (3, 7, 0.1), (3, 37, 0.15), (3, 38, 0.0)])
def test_lattices(cuda, orc, dim, nside, jitter):
    pos, h = W.lattice(nside, dim, jitter=jitter, seed=41)
    # without jitter the cutoff falls on lattice distances
    _check(orc, pos, (3.1 if dim == 2 else 2.8) * h if jitter else (5.0 * h if dim == 2 else 3.0 * h),
           self_skip=nside % 2 == 1)


@pytest.mark.parametrize("dim,nside", [(2, 8), (2, 9), (2, 11), (2, 13), (2, 230), (3, 8), (3, 9), (3, 11), (3, 33)])
def test_periodic(cuda, orc, dim, nside):
    h = 1.0 / nside
    pos, _ = W.lattice(nside, dim, h=h, jitter=0.2, seed=42)
    pos = np.mod(pos, 1.0)
    box = ((0.0,) * dim, (1.0,) * dim, (1, 1, 0)[:dim] if nside % 2 else (1,) * dim)
    _check(orc, pos, (3.1 if dim == 2 else 2.6) * h, box=box)


def test_uneven_and_clustered(cuda, orc):
    cfg = W.config3(60_000, seed=43)
    _check(orc, cfg["pos"], 0.0, rcut_pp=cfg["rcut_pp"])
    rng = np.random.default_rng(44)
    # rows far longer than the mean occupancy suggests
    pos = np.vstack([rng.random((5000, 3)), 0.4 + 0.03 * rng.random((1500, 3))])
    _check(orc, pos, 0.08)
    _check(orc, rng.random((3, 2)), 0.5)


def test_outside_the_box(cuda, orc):
    rng = np.random.default_rng(45)
    pos = rng.random((4000, 2)) * 1.2 - 0.1
    _check(orc, pos, 0.05, box=((0.0, 0.0), (1.0, 1.0), (0, 0)))
