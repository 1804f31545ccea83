"""A substep in other units of mass: density and energy times s = 2^-176 (1e-53), the field times
sqrt(s), and the floors with them.  Every term of the equations scales alike and the powers of two
are exact, so the result is the unscaled one times the same factors: the inversion must not form
powers of its enthalpy that leave the range of FP64 where the quotients it needs do not."""
import numpy as np
import pytest

from helpers import make_torus, rel_err
from harm_harm_b200 import HARM_PREC_FP64, HARM_PREC_FP64_FMA, Harm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [HARM_PREC_FP64, HARM_PREC_FP64_FMA])
def test_advance_in_small_units(cuda, prec):
    g, geom, conn, aux, P = make_torus(32, 24, 8, lim=0)
    s = np.array([2.0**-176] * 2 + [1.0] * 3 + [2.0**-88] * 3)
    small = aux.copy()
    small[1:] *= 2.0**-176
    out = []
    for a, f in ((aux, np.ones(8)), (small, s)):
        dev = Harm(g, geom, conn, a)
        Pd = cuda.from_numpy(P * f[:, None, None, None]).cuda()
        pf, flag = cuda.zeros_like(Pd), cuda.zeros(P.shape[1:], dtype=cuda.int8, device="cuda")
        dev.advance(0, Pd, Pd, pf, flag, 1e-3, precision=prec)
        out.append((pf.cpu().numpy()[(slice(None), *g.active)] / f[:, None, None, None], flag.cpu().numpy()))
    assert np.array_equal(out[0][1], out[1][1])
    for pl in range(8):
        assert rel_err(out[1][0][pl], out[0][0][pl]) < 1e-13, pl
