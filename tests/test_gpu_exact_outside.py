"""The bit-exact form on nodes that its integer collision hands over, at every
kind of relaxation time: velocities past its range, single populations past
their ranges, and states that trip the density guard.  Distributions, macros
and the guard's report equal the oracle's."""
import numpy as np
import pytest

import oracle_py as O
import porelb_gb300 as P
from porelb_gb300._lib import Q
from porelb_gb300.batch import Batch

from helpers import W, noise_flag

pytestmark = pytest.mark.gpu

DIMS = (11, 9, 13)
EX = np.array((0, 1, -1, 0, 0, 0, 0, 0, 0, 0, 0, -1, 1, -1, 1, -1, 1, -1, 1))
EY = np.array((0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, -1, 1))
EZ = np.array((0, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, -1, 1, 1, -1, 0, 0, 0, 0))
TAUS = [0.505, 0.8, 0.97, 0.9999, 1.0, 1.03, 2.6, 20.0, 40.0, 300.0]


def equilibrium(rho, u):
    eu = u @ np.stack([EX, EY, EZ])
    return W * rho[:, None] * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * (u * u).sum(1)[:, None])


def state(kind, V, seed):
    """Distributions of the nodes of V: `fast` (a flow that turns with z and
    is faster than 0.11 in one direction over most of the domain), `single`
    (two opposite populations of one node in twelve at 2.4 or 0.1 of their
    weight, the rest population making up the density)."""
    rng = np.random.default_rng(seed)
    n = len(V)
    rho = 1 + 0.02 * (rng.random(n) - 0.5)
    if kind == "fast":
        turn = 2 * np.pi * V["z"] / DIMS[2]
        u = 0.14 * np.stack([np.cos(turn), np.sin(turn), 0.3 * np.cos(2 * turn)], 1)
        return equilibrium(rho, u + 1e-3 * (rng.random((n, 3)) - 0.5))
    f = equilibrium(rho, 0.016 * (rng.random((n, 3)) - 0.5))
    for i in np.flatnonzero(rng.random(n) < 0.08):
        j = 1 + 2 * rng.integers(0, 9)
        to = W[j] * rng.choice([2.4, 0.1])
        f[i, 0] += f[i, j] + f[i, j + 1] - 2 * to
        f[i, j] = f[i, j + 1] = to
    return f


def oracle(V, vs, tau, force, f0, steps):
    s = O.OracleSim(V, *DIMS, vs, tau, force)
    s.init()
    np.ctypeslib.as_array(s.lib.orc_f0(s.h), (f0.size,))[:] = f0
    return s, s.run(steps)


@pytest.mark.parametrize("kind", ["fast", "single"])
@pytest.mark.parametrize("tau", TAUS)
def test_bits_equal_oracle(tau, kind):
    flag = noise_flag(DIMS, 0.03, 21)
    V, vs = P.build_table(flag, *DIMS, 1)
    f0 = state(kind, V, 3).reshape(-1)
    s, rc = oracle(V, vs, tau, 1e-6, f0, 1)
    assert kind == "single" or np.mean(np.abs(s.macros()[1:]).max(0) >= 0.11) > 0.3
    s, rc = oracle(V, vs, tau, 1e-6, f0, 3)
    assert rc[0] == 0
    with P.Simulation(V, *DIMS, vs, tau=tau, force=1e-6) as sim:
        sim.init_dist_macro()
        sim.set_f(f0)
        sim.step(3)
        assert np.array_equal(sim.get_f(), s.f0())
        assert np.array_equal(sim.macros(), s.macros())


@pytest.mark.parametrize("tau", TAUS)
def test_guard_reports_the_oracles_node(tau):
    flag = noise_flag(DIMS, 0.03, 21)
    V, vs = P.build_table(flag, *DIMS, 1)
    f0 = state("fast", V, 4)
    f0[(V["z"] >= 5) & (V["z"] < 9)] *= 1.21
    f0 = f0.reshape(-1)
    _, rc = oracle(V, vs, tau, 1e-6, f0, 3)
    assert rc[0] != 0
    with P.Simulation(V, *DIMS, vs, tau=tau, force=1e-6) as sim:
        sim.init_dist_macro()
        sim.set_f(f0)
        with pytest.raises(P.PorelbError) as e:
            sim.step(3)
        assert e.value.status == -6
        err = sim.last_error()
        assert (err["it"], err["node"]) == (rc[1], rc[2])


@pytest.mark.parametrize("tau", [0.8, 1.02, 50.0])
def test_pool_equals_plain_on_fast_flow(tau):
    """A strong force drives a pool sample past the velocity range."""
    dims = (17, 16, 18)
    flag = noise_flag(dims, 0.004, 5)
    with Batch(4096 * 2, 2, "fp64_exact", check_every=30) as pool, \
            P.Simulation.from_flag(flag, *dims, tau=tau, force=5e-3) as sim:
        sid = pool.add_flag(flag, *dims, tau, 5e-3, tol=0.0, max_steps=1000)
        pool.run(1)
        sim.init_dist_macro()
        sim.step(30)
        assert np.mean(np.abs(sim.macros()[1:]).max(0) > 0.11) > 0.1
        assert np.array_equal(pool.get_f(sid), sim.get_f())
        assert pool.get_f(sid).size == sim.N * Q
