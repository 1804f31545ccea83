"""Utoprimgen over points at the sizes where its kernels can go wrong: one point, the edges of a block
of 128, the line between the one kernel for few points and the two for many, several windows of 1024
flags per block of the second, and sets dense in points that do not converge within the first's
steps (low u/rho at high B^2/rho, whose residual rounds more coarsely than the test) or that the hot
inversion cannot invert.  FP64 against the oracle point by point: the same flags, primitives to 1e-9
of each point's largest (W' of the slow points is only defined to 1e-12 of D, 1e-6 of itself and of
u)."""
import numpy as np
import pytest

from helpers import make_torus
from harm_harm_b200 import Harm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _points(g, geom, n, kind, seed):
    rng = np.random.default_rng(seed)
    cell = rng.integers(geom.shape[2] * geom.shape[3], size=n)
    rec = np.ascontiguousarray(geom[0].reshape(28, -1)[:, cell])
    P = np.zeros((8, n))
    P[0] = 10.0 ** rng.uniform(-4, 0, n)
    P[1] = P[0] * 10.0 ** (rng.uniform(-3, 0, n) if kind != "slow" else rng.uniform(-6, -5, n))
    P[2:5] = rng.normal(0.0, 0.05, (3, n)) / np.sqrt(rec[[4, 7, 9]])
    P[5:] = rng.normal(0.0, 1.0, (3, n)) * np.sqrt(P[0] * (10.0 if kind == "slow" else 0.01)) / np.sqrt(rec[[4, 7, 9]])
    U = np.stack([O.primtoU_point(np.ascontiguousarray(rec[:, k]), P[:, k]) for k in range(n)], axis=1)
    if kind == "failing":
        bad = rng.random(n) < 0.5
        U[1, bad] *= -3.0  # no root: the hot inversion fails, the cold one may take over
    return U, rec, P * rng.uniform(0.99, 1.01, P.shape)


@pytest.mark.parametrize("n,kind", [(1, "plain"), (127, "plain"), (129, "slow"), (1025, "slow"), (2300, "failing"), (1, "failing")])
def test_points(cuda, n, kind):
    g, geom, conn, aux, _ = make_torus(16, 16, 1)
    U, rec, guess = _points(g, geom, n, kind, seed=n)
    dev = Harm(g, geom, conn, aux)
    Pd = cuda.from_numpy(guess.copy()).cuda()
    flag = cuda.zeros(n, dtype=cuda.int8, device="cuda")
    it = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    dev.Utoprimgen(cuda.from_numpy(U).cuda(), cuda.from_numpy(rec).cuda(), Pd, flag, it)
    P, flag, it = Pd.cpu().numpy(), flag.cpu().numpy(), it.cpu().numpy()
    for k in range(n):
        pr, fl, _ = O.utoprimgen_point(g, np.ascontiguousarray(rec[:, k]), U[:, k], guess[:, k])
        assert flag[k] == fl, (k, flag[k], fl)
        assert np.abs(P[:, k] - pr).max() <= 1e-9 * np.abs(pr).max(), k
    if kind == "slow":
        assert (it > 12).any()
    if kind == "failing" and n > 1:
        assert (flag != 0).any()


@pytest.mark.parametrize("per_sm,more", [(512, 0), (512, 1), (2 * 2 * 1024, 517)])
@pytest.mark.parametrize("dense", [0.02, 0.7])
def test_many_points(cuda, dense, per_sm, more):
    """The most points that one kernel takes, the fewest that two do (a window of the second with a
    remainder), and more than two windows per block of the second: what a block's list carries from
    one window into the next, full passes with windows still to come (dense) and lists that fill over
    all of them (sparse).  Slow, failing and plain points, checked against the oracle once, at random
    places: the kernels' operations on a point do not depend on its place, so its copies are equal bit
    for bit."""
    g, geom, conn, aux, _ = make_torus(16, 16, 1)
    sets = [_points(g, geom, m, kind, seed=m) for m, kind in ((700, "plain"), (150, "slow"), (400, "failing"))]
    U, rec, guess = (np.concatenate([s[q] for s in sets], axis=1) for q in range(3))
    ref = [O.utoprimgen_point(g, np.ascontiguousarray(rec[:, k]), U[:, k], guess[:, k]) for k in range(U.shape[1])]
    Pr, fr = (np.array([r[q] for r in ref]) for q in range(2))
    n = per_sm * cuda.cuda.get_device_properties(0).multi_processor_count + more
    rng = np.random.default_rng(11)
    at = np.where(rng.random(n) < dense, rng.integers(700, U.shape[1], n), rng.integers(0, 700, n))
    idx = cuda.from_numpy(at).cuda()
    dev = Harm(g, geom, conn, aux)
    Ud, recd, Pd = (cuda.from_numpy(a).cuda()[:, idx].contiguous() for a in (U, rec, guess))
    flag = cuda.full((n,), 77, dtype=cuda.int8, device="cuda")
    it = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    dev.Utoprimgen(Ud, recd, Pd, flag, it)
    P, flag, it = Pd.cpu().numpy(), flag.cpu().numpy(), it.cpu().numpy()
    assert (flag == fr[at]).all()
    assert (np.abs(P - Pr[at].T).max(axis=0) <= 1e-9 * np.abs(Pr[at]).max(axis=1)).all()
    first = np.zeros(U.shape[1], dtype=np.int64)
    first[at[::-1]] = np.arange(n)[::-1]
    assert np.array_equal(P, P[:, first[at]]) and np.array_equal(it, it[first[at]])
    assert (it[flag == 0] > 12).any() and (fr != 0).any()
