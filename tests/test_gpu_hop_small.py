"""The hopping kernels for small lattices, with one warp per direction (variant 1, NF <= 6) and
with two threads per site (variant 3), at the sizes where an index could go wrong: extents of 2, parities that are no multiple of its 32 sites,
both parities of a full field in one launch, FP32 and BF16 links; and the inverters,
whose last hop adds to the residual (variants 0 to 3) or leaves it to a kernel of its
own (variant 4), against the oracle."""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
from hirep_b200 import fields as F
from hirep_b200 import hrgpu as G

pytestmark = pytest.mark.gpu

DIMS = [(2, 2, 2, 2), (4, 2, 6, 2), (6, 4, 2, 10)]
GROUPS = [(2, O.FUND), (3, O.FUND), (4, O.FUND), (2, O.ADJ), (3, O.SYM), (4, O.ASYM)]
M = -0.1


def setup(ng, rep, dims, clover=False, represent=True):
    o = O.Oracle(*dims, ng, rep)
    u = F.smooth_gauge(5, o.V, ng, 0.3)
    uf = o.represent_gauge_field(u, True)
    o.set_gauge(uf)
    lat = G.Lattice(*dims, ng, rep, ipt=o.geometry()[0])
    if represent:
        lat.set_gauge(u)
        lat.represent_gauge_field(True)
    else:
        lat.set_gauge_f(uf)
    if clover:
        o.clover_init(1.0)
        o.compute_clover_term()
        lat.clover_init(1.0)
    return o, lat


@pytest.fixture
def pin():
    lib = G.lib()
    yield lambda v: G._check(lib.hrgpu_set_hop_variant(v), "set_hop_variant")
    lib.hrgpu_set_hop_variant(-1)
    lib.hrgpu_set_flt_link_storage(G.LINKS_F32)


@pytest.mark.parametrize("variant,represent", [(1, True), (1, False), (3, True)])
@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("ng,rep", GROUPS)
def test_operators(ng, rep, dims, variant, represent, pin):
    o, lat = setup(ng, rep, dims, True, represent)
    pin(variant)
    e, f = F.gaussian_spinor(1, o.VH, o.nf), F.gaussian_spinor(2, o.V, o.nf)
    for name, src, par in (("Dphi_eopre", e, G.EVEN), ("g5Dphi_eopre_sq", e, G.EVEN), ("Dphi", f, G.FULL),
                           ("g5Dphi_sq", f, G.FULL), ("Cphi_eopre", e, G.EVEN), ("g5Cphi", f, G.FULL)):
        fin, out = lat.field(par, host=src), lat.field(par)
        getattr(lat, name)(M, out, fin)
        ref = getattr(o, name)(M, src)
        # a sum of 8 products of NF terms, twice or four times over: a few roundings of the largest entry
        assert np.abs(out.download() - ref).max() < 2e-15 * o.nf * np.abs(ref).max(), name
    for links, tol in ((G.LINKS_F32, 2e-6), (G.LINKS_BF16, 3e-2)):
        G._check(lat.L.hrgpu_set_flt_link_storage(links), "links")
        fin, out = lat.field(G.EVEN, G.FLOAT, host=e.astype(np.complex64)), lat.field(G.EVEN, G.FLOAT)
        lat.g5Cphi_eopre_flt(M, out, fin)
        ref = o.g5Cphi_eopre(M, e)
        assert np.abs(out.download() - ref).max() < tol * np.abs(ref).max()


@pytest.mark.parametrize("variant", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("clover", [False, True])
@pytest.mark.parametrize("ng,rep", [(3, O.FUND), (2, O.ADJ)])
def test_cg_forms(ng, rep, clover, variant, pin):
    o, lat = setup(ng, rep, (4, 6, 2, 4), clover)
    m = 0.2
    o.set_mass(m)
    pin(variant)
    op = G.OP_G5CPHI_EOPRE_SQ if clover else G.OP_G5DPHI_EOPRE_SQ
    apply = o.g5Cphi_eopre_sq if clover else o.g5Dphi_eopre_sq
    b = F.gaussian_spinor(3, o.VH, o.nf)
    fb = lat.field(G.EVEN, host=b)
    for shifts, flt in (([0.0], False), ([-0.1], False), ([-0.01, -0.1, -1.0], False), ([0.0], True), ([-0.01, -1.0], True)):
        outs = [lat.field(G.EVEN) for _ in shifts]
        for _ in range(2):  # the second solve replays the captured iterations
            if len(shifts) == 1:
                lat.la("zero", outs[0])
            it, ok = lat.cg_mshift(op, m, shifts, 1e-24, fb, outs, flt=flt)
            assert ok and it > 5
        for s, x in zip(shifts, outs):
            xh = x.download()
            r = b - (apply(m, xh) - s * xh)
            assert np.linalg.norm(r) < 1.1e-12 * np.linalg.norm(b), (shifts, flt)


@pytest.mark.parametrize("variant", [0, 1, 3, 4])
@pytest.mark.parametrize("op,par", [(G.OP_DPHI_EOPRE, G.EVEN), (G.OP_CPHI_EOPRE, G.EVEN), (G.OP_DPHI, G.FULL)])
def test_g5qmr_forms(op, par, variant, pin):
    o, lat = setup(3, O.FUND, (4, 6, 2, 4), op == G.OP_CPHI_EOPRE)
    m = 0.2
    pin(variant)
    b = F.gaussian_spinor(4, lat.nsites(par), o.nf)
    fb = lat.field(par, host=b)
    apply = {G.OP_DPHI_EOPRE: o.Dphi_eopre, G.OP_CPHI_EOPRE: o.Cphi_eopre, G.OP_DPHI: o.Dphi}[op]
    for shifts in ([0.0], [0.05], [0.0, -0.1]):
        outs = [lat.field(par) for _ in shifts]
        for _ in range(2):
            if len(shifts) == 1:
                lat.la("zero", outs[0])
            it, ok = lat.g5QMR_mshift(op, m, shifts, 1e-20, fb, outs)
            assert ok and it > 3
        for s, x in zip(shifts, outs):
            xh = x.download()
            assert np.linalg.norm(b - (apply(m, xh) - s * xh)) < 1.1e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("variant", [0, 1, 3, 4])
@pytest.mark.parametrize("ng,rep", GROUPS)
def test_g5qmr_without_a_diagonal_term(ng, rep, variant, pin):
    """m = -4: the operator has no diagonal term, but the inverter's product with its input stays."""
    o, lat = setup(ng, rep, (4, 6, 2, 4))
    if variant == 4 and o.nf > 4:
        pytest.skip("variant 4 is built for NF <= 4")
    m = -4.0
    o.set_mass(m)
    pin(variant)
    b = F.gaussian_spinor(4, o.VH, o.nf)
    fb = lat.field(G.EVEN, host=b)
    # the hops have norm at most 4 each: the shifted systems have condition numbers of at most 3
    for shifts in ([40.0], [32.0, 40.0, -33.0]):
        outs = [lat.field(G.EVEN) for _ in shifts]
        if len(shifts) == 1:
            lat.la("zero", outs[0])
        it, ok = lat.g5QMR_mshift(G.OP_DPHI_EOPRE, m, shifts, 1e-20, fb, outs)
        xo, it_o = o.g5QMR_mshift(G.OP_DPHI_EOPRE, shifts, 1e-20, b)
        # the same recursion (a stopping test within rounding of its limit may fall either way)
        assert ok and abs(it - it_o) <= 1, (it, it_o)
        for s, x, y in zip(shifts, outs, xo):
            xh = x.download()
            assert np.linalg.norm(b - (o.Dphi_eopre(m, xh) - s * xh)) < 1.1e-10 * np.linalg.norm(b)
            assert np.linalg.norm(xh - y) < 1e-9 * np.linalg.norm(y)


@pytest.mark.parametrize("ng,rep", [(3, O.FUND), (2, O.ADJ)])
def test_reads_the_stored_links(ng, rep, pin):
    """In FP64 row 2 of a 3 x 3 link is not rebuilt (the other variants do where it saves traffic,
    at a few roundings): the result is that of the stored links, bit for bit."""
    o, lat = setup(ng, rep, (6, 4, 2, 10), True)
    assert lat.link_recon() in (1, 2)
    pin(1)
    e = F.gaussian_spinor(1, o.VH, o.nf)
    fin, out, full = lat.field(G.EVEN, host=e), lat.field(G.EVEN), lat.field(G.EVEN)
    try:
        for name in ("Dphi_eopre", "Cphi_eopre"):
            getattr(lat, name)(M, out, fin)
            G._check(lat.L.hrgpu_set_link_recon(0), "set_link_recon")
            getattr(lat, name)(M, full, fin)
            G._check(lat.L.hrgpu_set_link_recon(1), "set_link_recon")
            assert np.array_equal(out.download(), full.download()), name
    finally:
        lat.L.hrgpu_set_link_recon(1)


@pytest.mark.parametrize("ng,rep", [(3, O.FUND), (2, O.ADJ), (4, O.ASYM), (4, O.SYM)])
def test_choice_of_variants(ng, rep, pin):
    """The first calls on a lattice choose the variants (a call that is captured cannot, and runs
    without): captured first, choosing and chosen, each call gives the operator's result and
    counts its hops as any other does."""
    o, lat = setup(ng, rep, (4, 6, 2, 10), True)
    e, f = F.gaussian_spinor(1, o.VH, o.nf), F.gaussian_spinor(2, o.V, o.nf)
    calls = []
    for name, src, par, prec, mvm in (("Dphi_eopre", e, G.EVEN, G.DOUBLE, 1), ("g5Cphi_eopre_sq", e, G.EVEN, G.DOUBLE, 2),
                                      ("g5Dphi_sq", f, G.FULL, G.DOUBLE, 2), ("Cphi", f, G.FULL, G.DOUBLE, 1),
                                      ("Dphi_eopre_flt", e, G.EVEN, G.FLOAT, 1), ("g5Cphi_eopre_flt", e, G.EVEN, G.FLOAT, 1),
                                      ("g5Dphi_flt", f, G.FULL, G.FLOAT, 1)):
        host = src if prec == G.DOUBLE else src.astype(np.complex64)
        ref = getattr(o, name[:-4] if prec == G.FLOAT else name)(M, src)
        calls.append((name, lat.field(par, prec, host=host), lat.field(par, prec), ref, mvm))
    pin(0)
    for name, fin, out, _, _ in calls:  # the temporaries
        getattr(lat, name)(M, out, fin)
    pin(-1)
    lat.sync()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()

    def check():
        for name, fin, out, ref, _ in calls:
            # a few roundings of the largest entry per product, as in test_operators
            tol = 4e-15 * o.nf if out.prec == G.DOUBLE else 4e-6
            assert np.abs(out.download() - ref).max() < tol * np.abs(ref).max(), name
            out.buf.zero_()

    lat.L.hrgpu_set_stream(ctypes.c_void_p(stream.cuda_stream))
    try:
        with torch.cuda.graph(graph, stream=stream):
            for name, fin, out, _, _ in calls:
                getattr(lat, name)(M, out, fin)
    finally:
        lat.L.hrgpu_set_stream(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    for name, fin, out, _, _ in calls:
        out.buf.zero_()
    graph.replay()
    torch.cuda.synchronize()
    check()
    for _ in range(2):  # choosing, chosen
        for name, fin, out, _, mvm in calls:
            lat.getMVM()
            getattr(lat, name)(M, out, fin)
            assert lat.getMVM() == mvm, name
        lat.sync()
        check()
    graph.replay()
    torch.cuda.synchronize()
    check()
