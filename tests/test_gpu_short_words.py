"""Short neighbour words: FP32 domains and pools that outgrow the L2 keep the
words of most 256-node blocks as 16-bit distances in row order and as whole
words in Morton order.  A node's arithmetic does not depend on the order, so
the two agree to the last bit."""
import numpy as np
import pytest

import porelb_gb300 as P
from porelb_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def noise(dims, solid, seed):
    """Random cells; `solid` is the solid fraction of each z-plane."""
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    s = np.resize(np.asarray(solid), nz)
    return (rng.random((nz, nx * ny)) >= s[:, None]).astype(np.uint8).ravel()


# odd planes; long thin rows; planes whose counts vary so much that some of
# the distances need more than 16 bits; two fluid planes, each the other's
# neighbour on both sides; one block short of a whole one
CASES = [((97, 89, 83), [0.3]), ((701, 3, 301), [0.25]),
         ((401, 399, 9), [0.1, 0.15, 0.2, 0.1, 0.2, 0.8, 0.7, 0.75, 0.1]),
         ((600, 601, 2), [0.3]), ((79, 80, 80), [0.0])]


@pytest.mark.parametrize("boundary", ["reference", "halfway"])
@pytest.mark.parametrize("dims,solid", CASES)
def test_row_and_morton_order_agree(dims, solid, boundary):
    flag = noise(dims, solid, 5)
    got = []
    for ordering in ("reference", "morton"):
        with P.Simulation.from_flag(flag, *dims, tau=0.7, force=1e-4, precision="fp32",
                                    ordering=ordering, boundary=boundary) as s:
            assert s.N > 400000
            s.init_dist_macro()
            s.step(7)
            got.append((s.get_f(), s.get_f_streamed(), s.macros(), s.permeability()))
    for a, b in zip(got[0][:3], got[1][:3]):
        assert np.array_equal(a, b)
    assert np.allclose(got[0][3], got[1][3], rtol=1e-12, atol=0)


def test_large_domains_keep_row_order():
    """FP32 row order is for planes up to 1.75 times the L2 (short words),
    measured up to 1024^3 at porosity 0.35."""
    assert P.auto_ordering(214748328, 1024, "fp32") == "reference"
    assert P.auto_ordering(375808416, 1024, "fp32") == "reference"
    assert P.auto_ordering(900000000, 1024, "fp32") == "morton"


def test_records_of_many_ranks():
    """Tables built from node records of several ranks, against Morton order."""
    dims = (120, 90, 80)
    flag = noise(dims, [0.3, 0.4], 6)
    V, vs = P.build_table(flag, *dims, 4)
    got = []
    for ordering in ("reference", "morton"):
        with P.Simulation(V, *dims, vs, tau=0.7, force=1e-4, precision="fp32",
                          ordering=ordering) as s:
            s.init_dist_macro()
            s.step(5)
            got.append((s.get_f_streamed(), s.macros()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("ordering", ["reference", "morton"])
@pytest.mark.parametrize("cta,prefetch", [(128, False), (256, False), (256, True)])
def test_pools_agree(ordering, cta, prefetch):
    """Samples together in a pool with short words, and each in a pool too
    small for them."""
    dims = [(61, 59, 57), (64, 64, 64), (40, 3, 70), (5, 4, 3)]
    kw = dict(check_every=10, ordering=ordering, cta_threads=cta, l2_prefetch=prefetch,
              keep_macros=True)
    flags = [noise(d, [0.3], 7 + k) for k, d in enumerate(dims)]
    with Batch(600000, 8, "fp32", **kw) as b:
        ids = [b.add_flag(f, *d, 0.7, 1e-4, tol=0.0) for f, d in zip(flags, dims)]
        b.run(2)
        for f, d, i in zip(flags, dims, ids):
            with Batch(200000, 1, "fp32", **kw) as c:
                j = c.add_flag(f, *d, 0.7, 1e-4, tol=0.0)
                c.run(2)
                assert np.array_equal(b.get_f(i), c.get_f(j))
                assert np.array_equal(b.macros(i), c.macros(j))


@pytest.mark.parametrize("sizes", [(600000, 60000), (60000, 600000), (600000, 600000)])
@pytest.mark.parametrize("precision", ["fp16dev", "fp32"])
def test_transfer_translates_the_words(precision, sizes):
    """A sample moved between pools that keep its words differently steps on
    as it does in a pool of the same kind."""
    dims = (40, 41, 33)
    flag = noise(dims, [0.3], 9)
    got = []
    for ns, nd in (sizes, (60000, 60000)):
        with Batch(ns, 4, precision, check_every=10, ordering="reference") as h, \
                Batch(nd, 4, "fp32", check_every=10, ordering="reference") as t:
            sid = h.add_flag(flag, *dims, 0.8, 1e-4, tol=1e-12, handoff_tol=0.5)
            h.run(3)
            new = h.transfer(sid, t)
            t.run(3)
            got.append((t.result(new)["steps"], t.get_f(new)))
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
