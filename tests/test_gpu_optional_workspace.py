"""The paths that run when the workspaces of the faster ones are not taken
(hrgpu_set_optional_workspace(0), or too little free memory): the multi-shift CG updating
its shifted systems in every iteration, and the clover force in the fermion representation."""
import numpy as np
import pytest
import torch

import oracle as O
from hirep_b200 import fields as F
from hirep_b200 import hrgpu as G

pytestmark = pytest.mark.gpu


@pytest.fixture
def optional():
    lib = G.lib()
    yield lambda on: G._check(lib.hrgpu_set_optional_workspace(on), "set_optional_workspace")
    lib.hrgpu_set_optional_workspace(1)


def setup(ng, rep, dims, csw):
    lat = G.Lattice(*dims, ng, rep)
    lat.set_gauge(F.smooth_gauge(5, lat.V, ng, 0.3))
    lat.represent_gauge_field(True)
    if csw:
        lat.clover_init(csw)
    return lat


@pytest.mark.parametrize("op,par,csw", [(G.OP_G5DPHI_EOPRE_SQ, G.EVEN, 0.0), (G.OP_G5CPHI_EOPRE_SQ, G.EVEN, 1.0),
                                        (G.OP_G5DPHI_SQ, G.FULL, 0.0)])
@pytest.mark.parametrize("ng,rep", [(3, O.FUND), (4, O.ASYM)])
def test_shifts_updated_in_every_iteration(ng, rep, op, par, csw, optional):
    """The same iterations and the same solutions, bit for bit, at every place a solve can end."""
    lat = setup(ng, rep, (4, 6, 2, 6), csw)
    b = lat.field(par, host=F.gaussian_spinor(3, lat.nsites(par), lat.nf))

    def solve(shifts, err2, flt):
        outs = [lat.field(par) for _ in shifts]
        it, ok = lat.cg_mshift(op, 0.2, shifts, err2, b, outs, flt=flt)
        assert ok
        return it, [x.download() for x in outs]

    forms = [(s, e, f) for s in ([-0.3], [-0.02, -3.0], [0.0, -0.02, -3.0, -40.0, -300.0])
             for e in (1e-5, 1e-6, 1e-8, 1e-9, 1e-11, 1e-20) for f in (False, True)]
    for s, e, f in forms[:2]:  # tunes the hopping kernels in both precisions
        solve(s, e, f)
    kept = [solve(*f) for f in forms]
    optional(0)
    for f, (it, xs) in zip(forms, kept):
        it0, xs0 = solve(*f)
        assert it0 == it, f
        assert all(np.array_equal(x, y) for x, y in zip(xs, xs0)), f


@pytest.mark.parametrize("ng,rep", [(3, O.FUND), (2, O.ADJ), (3, O.SYM), (4, O.ASYM)])
def test_clover_force_without_its_workspace(ng, rep, optional):
    """The workspace is given back, and the force without it is the same up to rounding."""
    lat = setup(ng, rep, (8, 8, 8, 8), 1.3)
    x, y = (lat.field(G.FULL, host=F.gaussian_spinor(3 + k, lat.V, lat.nf)) for k in range(2))
    size = 8 * lat.V * (42 * ng**2 + 24 * (ng**2 - 1))

    def force():
        lat.momenta_set(np.zeros((lat.V, 4, lat.dimg)))
        lat.fermion_force_begin()
        lat.force_fermion_core(x, y, 1, 0.7, 1.0)
        lat.force_clover_logdet(0.2, 2.0)
        lat.fermion_force_end_momenta(0.7)
        return lat.momenta_get()

    lat.set_dirac_mass(0.2)
    with_it = force()
    lat.sync()
    before = torch.cuda.mem_get_info()[0]
    optional(0)
    assert torch.cuda.mem_get_info()[0] - before >= 0.9 * size
    without = force()
    # sums of a few hundred products of entries of order one, relative to the largest entry
    assert np.abs(with_it - without).max() < 2e-13 * np.abs(with_it).max()
    assert torch.cuda.mem_get_info()[0] - before >= 0.9 * size
    optional(1)
    assert np.array_equal(force(), with_it)


def test_other_values_are_refused(optional):
    lib = G.lib()
    for v in (-1, 2):
        assert lib.hrgpu_set_optional_workspace(v) == 2
        assert b"set_optional_workspace" in lib.hrgpu_last_error()
