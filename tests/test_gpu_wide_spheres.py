"""The device sphere pack where a bounding box is done in several parts:
radii on both sides of what one part holds, boxes of 1 to 27 parts, clipped
to the domain in some of the axes.  The host's bytes."""
import numpy as np
import pytest

import porelb_gb300 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,rmin,rmax,phi", [
    ((120, 110, 130), 44.0, 47.5, 0.25),     # one part and two
    ((97, 96, 95), 50.0, 60.0, 0.15),        # the whole domain, a part and a cell wide
    ((193, 40, 192), 90.0, 97.0, 0.30),      # three parts, one, two
    ((250, 211, 230), 100.0, 120.0, 0.30),   # up to 27 parts
    ((400, 3, 5), 150.0, 260.0, 0.10)])
def test_pack_equals_host(dims, rmin, rmax, phi):
    for seed in (1, 2):
        a, na, pa = P.sphere_pack(seed, *dims, rmin, rmax, phi)
        b, nb, pb = P.sphere_pack_device(seed, *dims, rmin, rmax, phi)
        assert na == nb and pa == pb
        assert np.array_equal(a, b)
