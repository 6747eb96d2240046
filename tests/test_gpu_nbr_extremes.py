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


def _patch(n, dim, ratio, share, seed):
    """n points, `share` of them in a patch whose spacing is `ratio` times
    smaller, each with a radius of about 30 (2D) or 90 neighbours."""
    rng = np.random.default_rng(seed)
    nd = int(n * share)
    h = (1.0 / (n - nd)) ** (1.0 / dim)
    side = nd ** (1.0 / dim) * h / ratio
    wide, dense = rng.random((n - nd, dim)), 0.6 - side / 2 + side * rng.random((nd, dim))
    rc = (3.1 if dim == 2 else 2.8) * h
    near = np.all(np.abs(wide - 0.6) < side / 2, axis=1)
    radii = np.concatenate([np.where(near, rc / ratio, rc), np.full(nd, rc / ratio)])
    order = rng.permutation(n)
    return np.vstack([wide, dense])[order], radii[order]


@pytest.mark.parametrize("dim,n,ratio,share", [(2, 6000, 4, 0.1), (2, 6000, 8, 0.3), (3, 6000, 3, 0.3), (3, 4000, 4, 0.5)])
@pytest.mark.parametrize("periodic", [False, True])
def test_crowded_groups(cuda, orc, dim, n, ratio, share, periodic):
    """Groups of cells too crowded for one warp, beside ordinary ones; the longest
    rows are longer than the staging rows in some of these sets."""
    pos, radii = _patch(n, dim, ratio, share, 72)
    if periodic:  # (the patch across the box's faces)
        pos = np.mod(pos + 0.4, 1.0)
    box = ((0.0,) * dim, (1.0,) * dim, (1,) * dim) if periodic else None
    for self_skip in (True, False):
        rp, cols = _build(pos, 0.0, box, radii, self_skip)
        erp, ecols = orc.neighbors(pos, 0.0, rcut_pp=radii, box=box, self_skip=self_skip)
        assert np.array_equal(rp, erp) and np.array_equal(cols, ecols)


@pytest.mark.parametrize("dim", [2, 3])
def test_crowds_of_long_rows(cuda, orc, dim):
    """A cluster under one cutoff: rows longer than the staging rows, found by both
    searches of one build."""
    rng = np.random.default_rng(73)
    pos = np.vstack([rng.random((4000, dim)), 0.45 + 0.1 * rng.random((3000, dim))])
    rcut = 2.5 * 7000 ** (-1.0 / dim)
    rp, cols = _build(pos, rcut)
    erp, ecols = orc.neighbors(pos, rcut)
    assert np.diff(erp).max() > 300
    assert np.array_equal(rp, erp) and np.array_equal(cols, ecols)


def test_a_refused_build_leaves_no_list(cuda):
    """After positions or a list that are refused the plan has no list: calls that
    need one say so (they would read arrays that were never filled)."""
    from openfpm_numerics_gb300 import _capi as C

    pos = torch.tensor(W.lattice(12, 2)[0], device="cuda")
    bad = pos.clone()
    bad[3, 0] = float("inf")
    plan = DcpsePlan(2, [[(1, 0)]])
    rp = torch.arange(145, dtype=torch.int64, device="cuda")
    for refused in (lambda: plan.build_neighbors(bad, 0.3),
                    lambda: plan.set_neighbors(rp, torch.full((144,), 144, device="cuda"))):
        plan.build_neighbors(pos, 0.3)
        with pytest.raises(C.DcpseError):
            refused()
        assert plan.info()["n"] == -1
        with pytest.raises(C.DcpseError) as e:
            plan.assemble(pos, C.ASSEMBLE_FAST | C.STORE_OUT_F64)
        assert e.value.code == C.ERR_STATE
    plan.build_neighbors(pos, 0.3)
    plan.assemble(pos, C.ASSEMBLE_FAST | C.STORE_OUT_F64)
    plan.close()


@pytest.mark.parametrize("dim,cells", [(2, 30), (2, 100), (2, 160), (3, 8), (3, 24)])
def test_outside_a_periodic_box(cuda, dim, cells):
    """Particles just inside, just beyond and well outside a box with periodic
    axes, in groups of one, two and four cells: the search by groups against the
    two-pass search, which serves where the columns are a second set (here the
    same positions)."""
    rng = np.random.default_rng(74)
    side = 1.0 / (cells + 0.5)
    rcut = 2.0 * side
    n = int((10 if dim == 2 else 2.5) * cells ** dim / (3.1 if dim == 2 else 1.0))
    pos = rng.random((n, dim))
    k = n // 8
    edge = rng.integers(0, 2, (k, dim)).astype(float)
    off = side * rng.choice([0.0, 1e-16, 1e-9, 1e-7, 9e-7, 1.1e-6, 1e-5, 0.3, 0.6, 3.0], (k, dim)) * rng.choice([-1, 1], (k, dim))
    axes = rng.random((k, dim)) < 0.6
    pos[:k] = np.where(axes, edge + off, pos[:k])
    for per in ((1,) * dim, (0,) + (1,) * (dim - 1), (1,) + (0,) * (dim - 1)):
        box = ((0.0,) * dim, (1.0,) * dim, per)
        rp, cols = _build(pos, rcut, box, self_skip=False)
        plan = DcpsePlan(dim, [[(1,) + (0,) * (dim - 1)]], box=box)
        t = torch.tensor(pos, device="cuda")
        plan.set_support(t.clone())
        plan.build_neighbors(t, rcut)
        rp2, cols2 = (x.cpu().numpy() for x in plan.neighbors())
        plan.close()
        assert np.array_equal(rp, rp2) and np.array_equal(cols, cols2)
