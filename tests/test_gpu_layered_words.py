"""16-bit neighbour words where the z-planes' node counts vary: each block of
256 nodes counts its distances from its own neighbours in the planes above and
below, so layers, gradients and domains of two planes keep them.  Which blocks
have them is checked, and that a step is the same, to the last bit, as in
Morton order with whole words."""
import numpy as np
import pytest

import porelb_gb300 as P
from porelb_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def layers(dims, solid, seed=5):
    """Random cells; `solid` is the solid fraction of each z-plane."""
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    s = np.resize(np.asarray(solid), nz)
    return (rng.random((nz, nx * ny)) >= s[:, None]).astype(np.uint8).ravel()


# (dims, solid fraction of each plane).  Nearly all blocks fit; whole words
# stay with a block that reaches over the end of the first or last plane and
# with rows at the wrap in y of planes of more than 32k nodes
CASES = [((300, 280, 12), [0.1] * 6 + [0.7] * 6),    # two layers
         ((401, 399, 9), [0.1, 0.15, 0.2, 0.1, 0.2, 0.8, 0.7, 0.75, 0.1]),
         ((600, 601, 2), [0.3]),                     # each plane is both neighbours
         ((512, 512, 5), list(np.linspace(0.05, 0.9, 5))),
         ((160, 150, 40), [0.05, 0.95]),             # every second plane nearly solid
         ((700, 700, 1), [0.1]),                     # its own neighbour
         ((97, 89, 83), [0.3])]


@pytest.mark.parametrize("boundary", ["reference", "halfway"])
@pytest.mark.parametrize("dims,solid", CASES)
def test_layers_keep_short_words(dims, solid, boundary):
    flag = layers(dims, solid)
    got = []
    for ordering in ("reference", "morton"):
        with P.Simulation.from_flag(flag, *dims, tau=0.7, force=1e-4, precision="fp32",
                                    ordering=ordering, boundary=boundary) as s:
            w = s.words()
            assert w["blocks"] == -(-s.N // 256)
            if ordering == "reference":
                assert w["ordering"] == "reference"
                assert 0.98 * w["blocks"] <= w["short_blocks"] < w["blocks"]
            else:
                assert w["ordering"] == "morton"
            s.init_dist_macro()
            s.step(7)
            got.append((s.get_f(), s.get_f_streamed(), s.macros()))
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def test_layers_take_row_order():
    dims, solid = CASES[0]
    with P.Simulation.from_flag(layers(dims, solid), *dims, precision="fp32") as s:
        w = s.words()
        assert w["ordering"] == "reference" and w["short_blocks"] > 0.98 * w["blocks"]


@pytest.mark.parametrize("records", [False, True])
def test_row_order_gives_way_where_words_do_not_fit(records):
    """Planes of three rows of 65535 cells: the rows above and below a node
    are out of 16 bits' reach and whole words do better in Morton order."""
    dims = (65535, 3, 6)
    flag = layers(dims, [0.1])
    got = []
    for ordering in ("auto", "reference"):
        kw = dict(tau=0.7, force=1e-4, precision="fp32", ordering=ordering)
        if records:
            V, vs = P.build_table(flag, *dims, 1)
            s = P.Simulation(V, *dims, vs, **kw)
        else:
            s = P.Simulation.from_flag(flag, *dims, **kw)
        with s:
            assert P.auto_ordering(s.N, dims[2], "fp32") == "reference"
            assert s.words()["ordering"] == ("morton" if ordering == "auto" else "reference")
            assert s.words()["short_blocks"] == 0
            s.init_dist_macro()
            s.step(4)
            got.append((s.get_f_streamed(), s.macros()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("ordering", ["reference", "morton"])
def test_pool_samples_of_varying_planes(ordering):
    """Uneven samples in a pool with short words and each in a pool too small
    for them."""
    cases = [((120, 110, 20), [0.1] * 10 + [0.8] * 10), ((301, 299, 2), [0.2]),
             ((64, 65, 31), list(np.linspace(0.0, 0.9, 31))), ((5, 4, 3), [0.3])]
    kw = dict(check_every=10, ordering=ordering, keep_macros=True)
    flags = [layers(d, s, 7 + k) for k, (d, s) in enumerate(cases)]
    with Batch(800000, 8, "fp32", **kw) as b:
        ids = [b.add_flag(f, *d, 0.7, 1e-4, tol=0.0) for f, (d, _) in zip(flags, cases)]
        if ordering == "reference":
            for i in ids:
                w = b.sample_words(i)
                assert w["blocks"] == -(-b.num_nodes(i) // 256)
                assert 0.9 * w["blocks"] <= w["short_blocks"] <= w["blocks"]
            w = b.sample_words(ids[1])      # planes of 72k nodes: wrap rows stay whole
            assert w["short_blocks"] < w["blocks"]
        b.run(2)
        for f, (d, _), i in zip(flags, cases, ids):
            with Batch(250000, 1, "fp32", **kw) as c:
                j = c.add_flag(f, *d, 0.7, 1e-4, tol=0.0)
                assert c.sample_words(j)["short_blocks"] == 0
                c.run(2)
                assert np.array_equal(b.get_f(i), c.get_f(j))
                assert np.array_equal(b.macros(i), c.macros(j))
