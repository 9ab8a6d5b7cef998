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
