"""bound_prim's single launch and its per-direction path at the edges of their ranges, against the
oracle: the smallest grids either takes (n2 = ng + 1 and n3 = ng for the single launch, n2 = ng or
n3 < ng for the other, whose outer x3 ghost planes repeat planes that are ghosts of ghosts), one
plane and several.  FP64 in the oracle's operations: equal to the last bits of the math library's
log and exp.  With n2 = ng the outermost polar ghost row mirrors the other pole's first row, which
the oracle has already rewritten there: it is left out."""
import numpy as np
import pytest

from helpers import make_torus, rel_err
from harm_harm_b200 import Harm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1,n2,n3,lim", [(3, 5, 1, 0), (5, 7, 6, 2), (37, 9, 4, 0), (16, 12, 7, 2), (130, 33, 1, 2),
                                          (9, 4, 1, 0), (12, 6, 8, 2), (20, 9, 3, 1), (33, 15, 2, 2)])
def test_bound_edges(cuda, n1, n2, n3, lim):
    g, geom, conn, aux, P = make_torus(n1, n2, n3, lim=lim)
    rng = np.random.default_rng(n1)
    P[:2] = 10.0 ** rng.uniform(-6, 0, P[:2].shape)
    P[2:] = rng.normal(0.0, 0.3, P[2:].shape)
    Po, Pd = P.copy(), cuda.from_numpy(P).cuda()
    O.Oracle(g, geom, conn, aux).bound_prim(Po)
    dev = Harm(g, geom, conn, aux)
    dev.bound_prim(Pd)
    once = Pd.cpu().numpy()
    rows = slice(None) if n2 > g.g.ng else slice(1, -1)
    assert rel_err(once[:, :, rows], Po[:, :, rows]) < 1e-13
    if n2 > g.g.ng:  # bounding a bounded state changes nothing (what a step's second bound relies on)
        dev.bound_prim(Pd)
        assert np.array_equal(Pd.cpu().numpy(), once)
