"""The molecular-dynamics kernels that hold their matrices in registers (NG <= 4)
and the ones beside them for larger NG, against the oracle at the sizes where an
index could go wrong: extents of 2 (both neighbours the same site), a volume that
is no multiple of a block, and momenta large enough that the exponential scales
and squares."""
import numpy as np
import pytest

import oracle as O
from hirep_b200 import fields as F
from hirep_b200 import hrgpu as G

pytestmark = pytest.mark.gpu

DIMS = [(2, 2, 2, 2), (4, 2, 6, 2), (6, 4, 2, 10)]


def setup(ng, dims, rep=O.FUND, seed=4, eps=0.4, scale=1.0):
    o = O.Oracle(*dims, ng, rep)
    u = F.smooth_gauge(seed, o.V, ng, eps)
    o.set_gauge(o.represent_gauge_field(u, True))
    lat = G.Lattice(*dims, ng, rep, ipt=o.geometry()[0])
    lat.set_gauge(u)
    lat.represent_gauge_field(True)
    mom = scale * np.random.default_rng(seed + 1).standard_normal((o.V, 4, ng * ng - 1))
    lat.momenta_set(mom)
    return o, lat, u, mom


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("ng", [2, 3, 4, 5])
def test_force0(ng, dims):
    o, lat, u, mom = setup(ng, dims)
    lat.force0(0.1, 2.25)
    # six staples of three unitary factors: entries of order one, a few roundings each
    assert np.abs(lat.momenta_get() - o.force0(0.1, 2.25, u, mom)).max() < 1e-13


@pytest.mark.parametrize("scale", [0.0, 0.1, 1.0, 40.0])
@pytest.mark.parametrize("ng", [2, 3, 4, 5])
def test_update_gauge_field(ng, scale):
    o, lat, u, mom = setup(ng, (4, 2, 6, 2), scale=scale)
    dt = 0.2
    lat.update_gauge_field(dt)
    ref = o.update_gauge_field(dt, u, mom)
    # one rounding of a unitary matrix per product, doubled by each squaring (up to 2^6 at scale 40)
    assert np.abs(lat.gauge_get() - ref).max() < 1e-14 * max(4.0, 4 * scale)


GROUPS = [(2, O.FUND), (3, O.FUND), (4, O.FUND), (2, O.ADJ), (2, O.SYM), (3, O.SYM), (3, O.ASYM), (4, O.ASYM)]


def clover_force_pair(o, lat, exp):
    """The clover force (with the log-det force of the standard term) of the library and of the oracle."""
    m, dt = 0.2, 0.7
    x, y = (F.gaussian_spinor(3 + k, lat.V, lat.nf) for k in range(2))
    for q in (o, lat):
        (q.expclover_init if exp else q.clover_init)(1.3)
        (o.set_mass if q is o else lat.set_dirac_mass)(m)
        if q is o:
            o.compute_clover_term()
        q.fermion_force_begin()
        if q is lat:
            lat.force_fermion_core(lat.field(G.FULL, host=x), lat.field(G.FULL, host=y), 1, dt, 1.0)
        else:
            o.force_fermion_core(x, y, 1, dt, 1.0)
        if not exp:
            q.force_clover_logdet(m, 2.0)
    zero = np.zeros((lat.V, 4, lat.dimg))
    lat.momenta_set(zero)
    lat.fermion_force_end_momenta(dt)
    return lat.momenta_get(), o.fermion_force_end(dt, zero)


@pytest.mark.parametrize("exp", [False, True])
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (6, 4, 2, 10)])
@pytest.mark.parametrize("ng,rep", GROUPS)
def test_clover_force(ng, rep, dims, exp):
    o, lat, u, _ = setup(ng, dims, rep)
    got, ref = clover_force_pair(o, lat, exp)
    # sums of a few hundred products of entries of order one, relative to the largest entry
    assert np.abs(got - ref).max() < 2e-13 * np.abs(ref).max()


@pytest.mark.parametrize("off", [0.0, 1e-14, 4e-13])
@pytest.mark.parametrize("ng,rep", [(3, O.FUND), (3, O.SYM), (4, O.ASYM)])
def test_clover_force_on_links_that_are_nearly_unitary(ng, rep, off):
    """A scale factor 1 + off in every link: the force is the reference's for the links as they are."""
    o, lat, u, _ = setup(ng, (4, 2, 2, 4), rep)
    u = u * (1.0 + off)
    o.set_gauge(o.represent_gauge_field(u, True))
    lat.set_gauge(u)
    lat.represent_gauge_field(True)
    got, ref = clover_force_pair(o, lat, False)
    assert np.abs(got - ref).max() < 2e-13 * np.abs(ref).max()


@pytest.mark.parametrize("uploaded", [False, True])
def test_clover_force_in_the_representation(uploaded):
    """Links that are not unitary, and represented links uploaded by themselves."""
    o, lat, u, _ = setup(3, (4, 2, 2, 4), O.SYM)
    if uploaded:
        lat.set_gauge_f(o.represent_gauge_field(u, True))
    else:
        u = u * 1.01
        o.set_gauge(o.represent_gauge_field(u, True))
        lat.set_gauge(u)
        lat.represent_gauge_field(True)
    got, ref = clover_force_pair(o, lat, False)
    assert np.abs(got - ref).max() < 2e-13 * np.abs(ref).max()


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (6, 4, 2, 10)])
@pytest.mark.parametrize("ng,rep", GROUPS + [(5, O.FUND), (4, O.SYM), (3, O.ADJ)])
def test_links_clover_term_and_inverse(ng, rep, dims):
    """represent_gauge_field (FP64 and FP32 links), the clover term, D and D^-1 on both parities."""
    o, lat, u, _ = setup(ng, dims, rep)
    uf = o.represent_gauge_field(u, True)
    assert np.abs(lat.gauge_f() - uf).max() < 1e-15 * max(1, o.nf)  # products of two entries of order one
    o.clover_init(1.3)
    o.compute_clover_term()
    lat.clover_init(1.3)
    # 24 loops of four links
    assert np.abs(lat.clover_term() - o.clover_term()).max() < 5e-15 * max(1, o.nf)
    m = 0.2
    e = F.gaussian_spinor(5, o.V, o.nf)
    f, out = lat.field(G.FULL, host=e), lat.field(G.FULL)
    for name in ("Cphi_diag", "Cphi_diag_inv"):
        getattr(lat, name)(m, out, f)
        ref = np.concatenate([getattr(o, name)(m, e[p * o.VH:(p + 1) * o.VH], p) for p in range(2)])
        # the blocks' condition number is below 10
        assert np.abs(out.download() - ref).max() < 1e-14 * np.abs(ref).max(), name
    # the FP32 links were made with the FP64 ones
    lat.Dphi_flt_(lat.field(G.FULL, G.FLOAT), lat.field(G.FULL, G.FLOAT, host=e))
    o.set_gauge(uf)
    of = lat.field(G.FULL, G.FLOAT)
    lat.Dphi_flt_(of, lat.field(G.FULL, G.FLOAT, host=e))
    ref = o.Dphi_(e, O.FULL, O.FULL)
    assert np.abs(of.download() - ref).max() < 3e-6 * np.abs(ref).max()
