"""Steps of one call overlap each other on the device (a step's CTAs start
while the step before drains).  One call of many steps and the same steps
one call at a time, each waited for, have to give the same bits: at the
sizes where the default CTA changes, where the grid is spread over the SMs
(less than one wave), and on both sides of the number of waves up to which
the neighbour words are loaded before the wait."""
import numpy as np
import pytest

import porelb_gb300 as P
from porelb_gb300.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,dims", [
    ("fp64_exact", (9, 8, 7)), ("fp64_exact", (24, 31, 33)), ("fp64_exact", (37, 36, 41)),
    ("fp64_exact", (161, 160, 162)), ("fp64_exact", (166, 165, 167)),
    ("fp64", (30, 31, 31)), ("fp64", (108, 110, 111)), ("fp64", (112, 113, 114)),
    ("fp64_fma", (31, 30, 30)), ("fp64_exact", (60, 61, 59)), ("fp64", (36, 38, 37)),
    ("fp64_fma", (44, 43, 45)), ("fp32", (72, 71, 72)), ("fp16dev", (36, 36, 35)), ("fp32", (29, 31, 30)), ("fp32", (222, 221, 222)),
    ("fp32", (226, 225, 226)), ("fp16dev", (40, 41, 39)), ("bf16dev", (228, 226, 227))])
def test_one_call_equals_waited_steps(precision, dims):
    steps = 7
    out = []
    for chunks in ([steps], [1] * steps):
        with P.Simulation.packed(5, *dims, 0.3 + min(dims) / 40, 1.0 + min(dims) / 20, 0.35,
                                 tau=0.7, force=1e-5, precision=precision) as sim:
            sim.init_dist_macro()
            for c in chunks:
                sim.step(c)
            out.append((sim.N, sim.macros().copy(), sim.permeability()))
    assert out[0][0] == out[1][0] > 0
    assert np.array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2]


@pytest.mark.parametrize("precision,edge", [("fp16dev", 226), ("bf16dev", 226), ("fp32", 64),
                                            ("fp64", 110)])
def test_sample_alone_equals_sample_in_a_long_launch(precision, edge):
    """Pool launches of few and of many waves take different kernels in the
    16-bit forms: a small sample's bits are the same in both."""
    out = []
    for mates in (0, 1):
        with Batch(int(mates * edge ** 3 * 0.36) + 40000, 2, precision, check_every=20) as pool:
            sid = pool.add_packed(3, 33, 31, 32, 3.0, 5.0, 0.4, 0.9, 1e-6, tol=0.0,
                                  max_steps=1000)
            for _ in range(mates):
                pool.add_packed(4, edge, edge, edge, 5.0, 10.0, 0.35, 0.8, 1e-6, tol=0.0,
                                max_steps=1000)
            pool.run(2)
            out.append((pool.get_f(sid), pool.result(sid)))
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1]
