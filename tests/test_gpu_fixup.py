"""post_fixup on planted failure flags, against the oracle: flags in the corners and along every
boundary (whose neighbours' flags follow the boundary order and are never read from the ghost cells
that the same launch writes), few and many, on grids whose ghost flags the fixup itself fills and on
those too small for that (n2 <= ng, n3 < ng3), one plane and several.  FP64 in the oracle's order:
equal to round-off, flags equal."""
import numpy as np
import pytest

from helpers import make_torus, rel_err
from harm_harm_b200 import Harm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.05, 0.6])
@pytest.mark.parametrize("finalstep", [0, 1])
@pytest.mark.parametrize("shape,lim", [((5, 7, 1), 0), ((37, 9, 6), 0), ((16, 12, 7), 2), ((9, 4, 1), 0), ((12, 4, 3), 1), ((130, 33, 1), 3)])
def test_planted_flags(cuda, shape, lim, finalstep, share):
    g, geom, conn, aux, P = make_torus(*shape, lim=lim)
    rng = np.random.default_rng(shape[0])
    P[:2] *= 10.0 ** rng.uniform(-1, 1, P[:2].shape)
    P[2:5] += rng.normal(0.0, 0.05, P[2:5].shape)
    orc = O.Oracle(g, geom, conn, aux)
    orc.bound_prim(P)
    flag = np.where(rng.random(P.shape[1:]) < share, rng.choice([1, 5, 9, 10, 11, 14, 15], P.shape[1:]), 0).astype(np.int8)
    act = flag[g.active]
    act[:, [0, 0, -1, -1], [0, -1, 0, -1]] = 1
    act[:, -1, ::3] = 14
    act[:, 0, 1::3] = 9
    act[:, ::2, -1] = 10
    Po, fo = P.copy(), flag.copy()
    orc.post_fixup(Po, fo, finalstep)
    dev = Harm(g, geom, conn, aux)
    Pd, fd = cuda.from_numpy(P).cuda(), cuda.from_numpy(flag).cuda()
    dev.post_fixup(Pd, fd, finalstep)
    near = slice(max(g.g.ng3 - 1, 0), g.g.ng3 + g.g.n3 + 1)  # with n3 < ng3 the planes beyond, which nothing reads, differ
    assert np.array_equal(fd.cpu().numpy()[near], fo[near])
    assert rel_err(Pd.cpu().numpy()[(slice(None), *g.active)], Po[(slice(None), *g.active)]) < 1e-13
    assert not np.array_equal(Po, P)
