"""Multi-shift CG, whose shifted systems take several iterations at once: solves that end
at every place among those, with shifts that converge in different iterations, in FP64
and with the FP32 inner solve, against the oracle's solutions and iteration counts."""
import numpy as np
import pytest

import oracle as O
from hirep_b200 import fields as F
from hirep_b200 import hrgpu as G

pytestmark = pytest.mark.gpu

M = 0.2


def setup(ng, rep, dims, clover):
    o = O.Oracle(*dims, ng, rep)
    u = F.smooth_gauge(5, o.V, ng, 0.3)
    uf = o.represent_gauge_field(u, True)
    o.set_gauge(uf)
    o.set_mass(M)
    lat = G.Lattice(*dims, ng, rep, ipt=o.geometry()[0])
    lat.set_gauge_f(uf)
    if clover:
        o.clover_init(1.0)
        o.compute_clover_term()
        lat.clover_init(1.0)
    return o, lat


@pytest.mark.parametrize("op,par,clover", [(G.OP_G5DPHI_EOPRE_SQ, G.EVEN, False), (G.OP_G5CPHI_EOPRE_SQ, G.EVEN, True),
                                           (G.OP_G5DPHI_SQ, G.FULL, False)])
@pytest.mark.parametrize("ng,rep", [(3, O.FUND), (4, O.ASYM)])
def test_ends_of_a_solve(ng, rep, op, par, clover):
    o, lat = setup(ng, rep, (4, 6, 2, 4), clover)
    shifts = [-0.02, -3.0, -0.3, -40.0, -300.0]
    b = F.gaussian_spinor(3, lat.nsites(par), o.nf)
    fb = lat.field(par, host=b)
    for n in (1, 2, 5):
        ends = set()
        for e in range(4, 16):
            err2 = 10.0 ** -e
            outs = [lat.field(par) for _ in range(n)]
            if n == 1:
                lat.la("zero", outs[0])
            it, ok = lat.cg_mshift(op, M, shifts[:n], err2, fb, outs)
            xo, it_o = o.cg_mshift(op, shifts[:n], err2, b)
            assert ok
            if it == it_o:  # (a stopping test within rounding of its limit may fall either way)
                ends.add((it - n) % 4)
                # the same recursion in FP64: rounding of some tens of iterations times the
                # condition number (below 1e3), far below one iteration's change (err2 >= 1e-15)
                for x, y in zip(outs, xo):
                    assert np.linalg.norm(x.download() - y) < 1e-11 * np.linalg.norm(y), (n, err2)
        assert len(ends) >= 3


def test_shifts_inner_solve_in_fp32():
    o, lat = setup(3, O.FUND, (4, 6, 2, 4), True)
    b = F.gaussian_spinor(4, lat.nsites(G.EVEN), o.nf)
    fb = lat.field(G.EVEN, host=b)
    for n, err2 in ((2, 1e-12), (3, 1e-20), (4, 1e-24)):
        shifts = [-0.02, -0.3, -3.0, -40.0][:n]
        outs = [lat.field(G.EVEN) for _ in shifts]
        it, ok = lat.cg_mshift(G.OP_G5CPHI_EOPRE_SQ, M, shifts, err2, fb, outs, flt=True)
        assert ok
        for s, x in zip(shifts, outs):
            xh = x.download()
            r = b - (o.g5Cphi_eopre_sq(M, xh) - s * xh)
            assert np.linalg.norm(r) ** 2 < 1.01 * err2 * np.linalg.norm(b) ** 2
