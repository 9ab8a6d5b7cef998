"""Multi-shift CG, whose shifted systems take several iterations at once: solves that end
at every place among those, with shifts that converge in different iterations, in FP64
and with the FP32 inner solve, against the oracle's solutions and iteration counts."""
import numpy as np
import pytest
import torch

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
        ends, other = set(), 0
        for e in range(4, 16):
            err2 = 10.0 ** -e
            outs = [lat.field(par) for _ in range(n)]
            if n == 1:
                lat.la("zero", outs[0])
            it, ok = lat.cg_mshift(op, M, shifts[:n], err2, fb, outs)
            xo, it_o = o.cg_mshift(op, shifts[:n], err2, b)
            # a stopping test within rounding of its limit may fall either way
            assert ok and abs(it - it_o) <= 1, (n, err2, it, it_o)
            other += it != it_o
            if it == it_o:
                ends.add((it - n) % 4)
                # the same recursion in FP64: rounding of some tens of iterations times the
                # condition number (below 1e3), far below one iteration's change (err2 >= 1e-15)
                for x, y in zip(outs, xo):
                    assert np.linalg.norm(x.download() - y) < 1e-11 * np.linalg.norm(y), (n, err2)
        assert len(ends) >= 3 and other <= 1


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


@pytest.mark.parametrize("flt", [False, True])
@pytest.mark.parametrize("ng,rep", [(3, O.FUND), (4, O.ASYM)])
def test_padding_stays_zero(ng, rep, flt):
    """The parities of these lattices are no multiple of the 32 sites that a field's components
    are padded to.  The library's workspaces are made of memory that the solve before has left
    full of numbers (another lattice, then another size of field); none of them may get into the
    padding of a solution, which the norms run over."""
    for dims in ((8, 8, 8, 8), (6, 4, 2, 10), (4, 6, 6, 14), (4, 2, 6, 2)):
        lat = G.Lattice(*dims, ng, rep)
        lat.set_gauge(F.smooth_gauge(5, lat.V, ng, 0.3))
        lat.represent_gauge_field(True)
        pad = (-lat.VH) % 32
        for op, par, n in ((G.OP_G5DPHI_SQ, G.FULL, 1), (G.OP_G5DPHI_EOPRE_SQ, G.EVEN, 10),
                           (G.OP_G5DPHI_SQ, G.FULL, 3), (G.OP_G5DPHI_EOPRE_SQ, G.EVEN, 1)):
            b = lat.field(par, host=F.gaussian_spinor(3, lat.nsites(par), lat.nf))
            outs = [lat.field(par) for _ in range(n)]
            it, ok = lat.cg_mshift(op, M, [0.0, *(-float(10.0 ** (k - 6)) for k in range(9))][:n], 1e-20, b, outs, flt=flt)
            assert ok
            for x in outs:
                v = x.buf.view(torch.float64).view(2 if par == G.FULL else 1, 4 * lat.nf, -1, 2)
                assert v.shape[2] == lat.VH + pad
                assert not v[:, :, lat.VH:].any(), (dims, op, n)
