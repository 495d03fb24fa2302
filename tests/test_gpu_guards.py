"""Periodic guard fill and fold in one launch against the oracle's axis by
axis exchanges: sizes from one cell above the guards up, rows longer than a
warp, no guards, one to three arrays; and the x-z form against the slab
operations written out.  Equal bit for bit."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from picsar_b200 import _lib
from picsar_b200 import picsar as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,g", [((4, 5, 4), 3), ((5, 7, 6), 3), ((37, 9, 12), 4), ((70, 33, 8), 2),
                                 ((3, 2, 4), 0), ((128, 16, 40), 1)])
@pytest.mark.parametrize("fold", [False, True])
def test_guards_match_the_slab_exchanges(cuda, n, g, fold):
    rng = np.random.default_rng(sum(n) + g)
    for count in (1, 2, 3):
        ref = [O.zeros_grid(*n, g) for _ in range(count)]
        for a in ref:
            a[...] = rng.standard_normal(a.shape)
        got = [P.to_fortran(a) for a in ref]
        for a in ref:
            (O.summation_bcs if fold else O.field_bc)(a, n, g)
            if fold:
                O.field_bc(a, n, g)
        ptr = [a.data_ptr() for a in got] + [None] * (3 - count)
        _lib.call("pxrb_summation_bcs_periodic" if fold else "pxrb_field_bc_periodic", *ptr, *n,
                  g, g, g, torch.cuda.current_stream().cuda_stream)
        for a, b in zip(ref, got):
            assert np.array_equal(a, b.cpu().numpy())


def _slabs(a, n, g, fold):
    """field_bc, or summation_bcs and field_bc after it, slab by slab on the
    axes that have cells (a's first node is -g)."""
    for fill in ([False, True] if fold else [True]):
        for ax in range(3):
            if n[ax] == 0:
                continue
            v = np.moveaxis(a, ax, 0)
            at = lambda lo: slice(lo + g[ax], lo + 2 * g[ax] + 1)       # nodes lo .. lo + g
            N = n[ax]
            if fill:
                v[at(N)] = v[at(0)].copy()
                v[at(-g[ax])] = v[at(N - g[ax])].copy()
            else:
                v[at(0)] += v[at(N)].copy()
                v[at(N - g[ax])] += v[at(-g[ax])].copy()


@pytest.mark.parametrize("n,g", [((40, 0, 9), (3, 0, 3)), ((5, 0, 70), (4, 0, 2)),
                                 ((9, 7, 8), (3, 1, 2))])
@pytest.mark.parametrize("fold", [False, True])
def test_guards_of_x_z_grids(cuda, n, g, fold):
    """An axis without cells and guards (y of x-z grids), and guards that
    differ per axis."""
    rng = np.random.default_rng(sum(n) + sum(g))
    ref = [rng.standard_normal([v + 1 + 2 * h for v, h in zip(n, g)]) for _ in range(3)]
    got = [P.to_fortran(a) for a in ref]
    for a in ref:
        _slabs(a, n, g, fold)
    _lib.call("pxrb_summation_bcs_periodic" if fold else "pxrb_field_bc_periodic",
              *[a.data_ptr() for a in got], *n, *g, torch.cuda.current_stream().cuda_stream)
    for a, b in zip(ref, got):
        assert np.array_equal(a, b.cpu().numpy())
