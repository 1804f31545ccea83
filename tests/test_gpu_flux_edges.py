"""The flux stage's two kernels at the edges of their ranges: lines shorter than a warp's 32 or 64,
grids of a few cells, segments and chunks with a remainder, one plane and several, the directions
in joint launches and each in its own, with the reduction of WENO5BND (a planted pressure jump) and
the PARALINE flattener active.  FP64 against the oracle to 1e-12 of each field's largest face value,
and to the bit against the tile kernel of the entry point without allocations, which has the same
arithmetic and none of these kernels; FP32 (mixed path) against the FP64 path: both reconstruct the
same state, and a face flux carries the rounding of a few dozen FP32 operations on the face's
largest terms, of which a substep adds dt/dx < 1: 64 half-ulps of a field's largest value (of the
state's, for the vectors, whose components share their terms)."""
import ctypes as C
from fractions import Fraction

import numpy as np
import pytest

from helpers import make_torus, plant_compression, rel_err
from harm_harm_b200 import HARM_PREC_FP64, HARM_PREC_MIXED, Grid, Harm
from harm_harm_b200 import _native as N
from oracle import oracle as O

SHAPES = [(5, 7, 1), (59, 9, 1), (33, 21, 6), (64, 13, 7), (131, 8, 12), (17, 70, 9)]
# larger ones, of which (41, 45, 37) takes a launch per direction for FP64 WENO5 and the last two do for all
LARGE = [(131, 70, 33), (29, 37, 230), (41, 45, 37), (133, 70, 90), (1390, 740, 1)]


def _faces(g, d):
    gg = g.g
    return (slice(None), slice(gg.ng3, gg.ng3 + gg.n3 + (d == 3)), slice(gg.ng, gg.ng + gg.n2 + (d == 2)),
            slice(gg.ng, gg.ng + gg.n1 + (d == 1)))


@pytest.mark.gpu
@pytest.mark.parametrize("lim", [0, 1, 2, 3])
@pytest.mark.parametrize("shape", SHAPES + LARGE)
def test_flux_edges(cuda, shape, lim):
    g, geom, conn, aux, P = make_torus(*shape, lim=lim)
    plant_compression(g, P)
    orc = O.Oracle(g, geom, conn, aux)
    orc.bound_prim(P)
    Fo = [np.zeros_like(P) for _ in range(3)]
    ndt = orc.fluxcalc(P, *Fo)
    dev = Harm(g, geom, conn, aux)
    Pd = cuda.from_numpy(P).cuda()
    Fd = [cuda.zeros_like(Pd) for _ in range(3)]
    got = dev.fluxcalc(Pd, *Fd)
    for d in range(3 if shape[2] > 1 else 2):
        a, b = Fd[d].cpu().numpy()[_faces(g, d + 1)], Fo[d][_faces(g, d + 1)]
        for pl in range(8):
            assert rel_err(a[pl], b[pl]) < 1e-12, (d + 1, pl)
        assert abs(got[d] - ndt[d]) <= 1e-12 * ndt[d]
    if g.cells <= N.HARM_NOALLOC_MAX_CELLS:  # the tile kernel, to the bit
        Gd = cuda.from_numpy(np.ascontiguousarray(geom)).cuda()
        Fn, nn = [cuda.zeros_like(Pd) for _ in range(3)], (C.c_double * 3)()
        cuda.cuda.synchronize()
        assert N.device_lib().harm_b200_fluxcalc_noalloc(C.byref(g.g), Gd.data_ptr(), Pd.data_ptr(), *(f.data_ptr() for f in Fn), nn, None) == 0
        assert list(nn)[:2] == list(got)[:2] and (shape[2] == 1 or nn[2] == got[2])
        for d in range(3 if shape[2] > 1 else 2):
            f = (slice(None), *_faces(g, d + 1)[1:])
            assert np.array_equal(Fn[d].cpu().numpy()[f], Fd[d].cpu().numpy()[f]), d + 1
    dt = 0.2 / sum(1.0 / x for x in ndt if x < 1e99)
    if lim != 2:  # the other limiters switch at the jump, and FP32 may take the other branch there
        Ps = make_torus(*shape, lim=lim)[4]
        if lim == 3:
            # the flattener tests the sign of a flux difference, which is zero in gas at rest: a drift,
            # slow enough for the floor's cold gas that the rounding of its kinetic energy does not
            # show in its velocity
            Ps[2] += 0.05
            Ps[3:5] += 0.01
        Pd = cuda.from_numpy(Ps).cuda()
        dev.bound_prim(Pd)
    out, ok = [], True
    for prec in (HARM_PREC_FP64, HARM_PREC_MIXED):
        pf, flag = cuda.zeros_like(Pd), cuda.zeros(P.shape[1:], dtype=cuda.int8, device="cuda")
        dev.advance(0, Pd, Pd, pf, flag, dt, precision=prec)
        out.append(pf.cpu().numpy()[(slice(None), *g.active)])
        ok = ok & (flag.cpu().numpy()[g.active] == 0)  # the jump leaves a few cells without a solution
    assert ok.mean() > 0.9
    for pl in range(8):
        own, most = np.abs(out[0][pl]).max(), np.abs(out[0]).max()
        assert np.abs(out[1][pl] - out[0][pl])[ok].max() < 64 * 2.0**-24 * (own + (pl >= 2) * most), pl


def test_corrected_quotients_are_ieee():
    """The WENO sums' division by a shared denominator (a y corrected by its exact remainder, y the
    rounded reciprocal), in exact rational arithmetic with each operation rounded: the IEEE quotient
    for random operands and for the constants it divides by (the formula; test_quotients.py runs the
header's functions)."""
    rng = np.random.default_rng(5)
    dens = list(10.0 ** rng.uniform(-12, 12, 300)) + [12.0, 1.6 - 1.3, 0.8 * (1 / 3) - 0.2 * (1 / 3), 1 - 1.2 * (1 / 3), 2.2250738585072014e-308]
    for b in dens:
        y = 1.0 / b
        for a in rng.uniform(-1, 1, 20) * b * 10.0 ** rng.uniform(-9, 3, 20):
            q = float(a) * y
            r = float(Fraction(float(a)) - Fraction(b) * Fraction(q))  # fma(-b, q, a): one rounding
            got = float(Fraction(r) * Fraction(y) + Fraction(q))       # fma(r, y, q)
            assert got == float(a) / b


def _narrowed(g, geom, P, ng, ng3):
    """the same active grid with ng (x3: ng3) ghost zones, its tables and its state; and the state of
    the wide grid whose ghost zones beyond those repeat the last one of them"""
    a, b = g.g, type(g.g)()
    C.memmove(C.byref(b), C.byref(a), C.sizeof(a))
    b.ng, b.ng3 = ng, ng3
    b.n1e, b.n2e, b.n3e = a.n1 + 2 * ng, a.n2 + 2 * ng, a.n3 + 2 * ng3
    cut, cut3 = a.ng - ng, a.ng3 - ng3
    inner = slice(cut, -cut or None)
    tables = [np.ascontiguousarray(t[..., inner, inner]) for t in geom]
    Pn = np.ascontiguousarray(P[:, cut3:P.shape[1] - cut3, inner, inner])
    k, j, i = (np.clip(np.arange(n) - c, 0, m - 1) for n, c, m in zip(P.shape[1:], (cut3, cut, cut), Pn.shape[1:]))
    return Grid(b), tables, Pn, np.ascontiguousarray(Pn[:, k][:, :, j][:, :, :, i])


@pytest.mark.gpu
@pytest.mark.parametrize("shape,lim,ng,ng3", [((40, 33, 1), 0, 1, 0), ((19, 70, 9), 0, 1, 1), ((70, 12, 7), 1, 1, 1), ((33, 21, 1), 1, 2, 0),
                                              ((12, 9, 35), 1, 2, 2), ((37, 12, 9), 2, 6, 5), ((20, 9, 40), 2, 6, 1), ((33, 9, 8), 3, 4, 3),
                                              ((70, 8, 9), 3, 4, 1)])
def test_fewer_ghost_zones_than_the_stencil(cuda, shape, lim, ng, ng3):
    """A caller's grid with fewer ghost zones than the reconstruction reads: a cell beyond the grid is
    the grid's last one, so the fluxes are those of a wide grid whose outer ghost zones repeat it.
    FP64 to the bit; the mixed path to a few FP32 roundings of the largest (as above)."""
    g, geom, conn, aux, P = make_torus(*shape, lim=lim)
    O.Oracle(g, geom, conn, aux).bound_prim(P)
    gn, tables, Pn, Pw = _narrowed(g, (geom, conn, aux), P, ng, ng3)
    got = []
    for grid, tabs, p in ((g, (geom, conn, aux), Pw), (gn, tables, Pn)):
        dev, Pd = Harm(grid, *tabs), cuda.from_numpy(p).cuda()
        Fd = [cuda.zeros_like(Pd) for _ in range(3)]
        ndt = dev.fluxcalc(Pd, *Fd)
        pf, flag = cuda.zeros_like(Pd), cuda.zeros(p.shape[1:], dtype=cuda.int8, device="cuda")
        dev.advance(0, Pd, Pd, pf, flag, 0.2 / sum(1.0 / x for x in ndt if x < 1e99), precision=HARM_PREC_MIXED)
        ok = flag.cpu().numpy()[grid.active] == 0
        got.append((ndt, [f.cpu().numpy()[_faces(grid, d + 1)] for d, f in enumerate(Fd)], pf.cpu().numpy()[(slice(None), *grid.active)], ok))
    assert got[0][0] == got[1][0]
    for d in range(3 if shape[2] > 1 else 2):
        assert np.array_equal(got[0][1][d], got[1][1][d]), d + 1
    ok = got[0][3] & got[1][3]
    assert ok.mean() > 0.9
    for pl in range(8):
        own, most = np.abs(got[0][2][pl]).max(), np.abs(got[0][2]).max()
        assert np.abs(got[1][2][pl] - got[0][2][pl])[ok].max() < 64 * 2.0**-24 * (own + (pl >= 2) * most), pl
