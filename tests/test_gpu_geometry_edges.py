"""Device geometry at the ends of its kernels' ranges: sphere boxes wider
than the tables of the cover kernel, boxes clipped to a small domain, radii
below a cell, cell counts that are no multiple of four or 32; tables in both
node orders with slabs and half-way walls.  Bit for bit the host's."""
import numpy as np
import pytest

import porelb_gb300 as P

from helpers import noise_flag

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(4, (131, 125, 123), 45.0, 60.0, 0.30),
                                  (5, (3, 5, 7), 1.0, 4.0, 0.20),
                                  (6, (97, 3, 101), 2.0, 30.0, 0.25),
                                  (7, (33, 31, 35), 0.3, 0.9, 0.80),
                                  (8, (1, 1, 9), 0.6, 0.7, 0.5),
                                  (9, (64, 64, 2), 47.0, 47.9, 0.05)])
def test_pack_equals_host(case):
    seed, dims, rmin, rmax, phi = case
    a, na, pa = P.sphere_pack(seed, *dims, rmin, rmax, phi)
    b, nb, pb = P.sphere_pack_device(seed, *dims, rmin, rmax, phi)
    assert na == nb and pa == pb
    assert np.array_equal(a, b)


@pytest.mark.parametrize("ordering", ["morton", "reference"])
@pytest.mark.parametrize("boundary", ["reference", "halfway"])
@pytest.mark.parametrize("dims,num_p", [((41, 3, 20), 4), ((1, 37, 6), 2), ((67, 33, 5), 5),
                                        ((5, 1, 1), 1)])
def test_tables_equal_records(ordering, boundary, dims, num_p):
    flag = noise_flag(dims, 0.4, 31)
    V, vs = P.build_table(flag, *dims, num_p)
    kw = dict(tau=0.7, force=1e-3, ordering=ordering, boundary=boundary)
    with P.Simulation(V, *dims, vs, **kw) as a, \
            P.Simulation.from_flag(flag, *dims, num_p=num_p, **kw) as b:
        assert a.N == b.N
        for s in (a, b):
            s.init_dist_macro()
            s.step(4)
        assert np.array_equal(a.get_f_streamed(), b.get_f_streamed())
        assert np.array_equal(a.macros(), b.macros())


def test_bad_flag_values_are_refused():
    for at in (0, 33, 62):       # whole words and the last, short one
        flag = np.ones(63, np.uint8)
        flag[at] = 2
        with pytest.raises(P.PorelbError) as e:
            P.Simulation.from_flag(flag, 7, 9, 1)
        assert e.value.status == -1
