"""The bit-exact form where its integer collision hands a node over: every
relaxation time it treats apart (1 - omega zero, small, near -1, tau > 2.5,
beyond its constants), forces that take nodes past its velocity range, and
states past its ranges of f and rho.  f and macros equal the oracle's bits."""
import numpy as np
import pytest

import oracle_py as O
import porelb_gb300 as P
from porelb_gb300.batch import Batch

from helpers import W, noise_flag

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau", [0.505, 0.8, 0.97, 0.9999, 1.0, 1.03, 2.6, 20.0, 60.0])
@pytest.mark.parametrize("force,spread", [(0.0, 0.05), (1e-5, 1e-4), (4e-3, 0.1), (1e-5, 0.8)])
def test_bits_equal_oracle(tau, force, spread):
    dims = (11, 9, 13)
    flag = noise_flag(dims, 0.35, 21)
    V, vs = P.build_table(flag, *dims, 1)
    rng = np.random.default_rng(7)
    f0 = (W[None, :] * (1.0 + spread * (rng.random((len(V), 19)) - 0.5))).reshape(-1)
    s = O.OracleSim(V, *dims, vs, tau, force)
    s.init()
    np.ctypeslib.as_array(s.lib.orc_f0(s.h), (f0.size,))[:] = f0
    rc = s.run(6)[0]
    with P.Simulation(V, *dims, vs, tau=tau, force=force) as sim:
        sim.init_dist_macro()
        sim.set_f(f0)
        try:
            sim.step(6)
        except P.PorelbError as e:
            assert e.status == -6 and rc != 0
            return
        assert rc == 0
        assert np.array_equal(sim.get_f(), s.f0())
        assert np.array_equal(sim.macros(), s.macros())


@pytest.mark.parametrize("tau,force", [(1.02, 1e-5), (0.7, 2e-2), (50.0, 1e-4)])
def test_pool_hands_over_too(tau, force):
    dims = (17, 16, 18)
    flag = noise_flag(dims, 0.3, 5)
    with Batch(4096 * 2, 2, "fp64_exact", check_every=20) as pool, \
            P.Simulation.from_flag(flag, *dims, tau=tau, force=force) as sim:
        sid = pool.add_flag(flag, *dims, tau, force, tol=0.0, max_steps=1000)
        pool.add_flag(flag, *dims, 0.8, 1e-6, tol=0.0, max_steps=1000)
        pool.run(1)
        sim.init_dist_macro()
        sim.step(20)
        assert np.array_equal(pool.get_f(sid), sim.get_f())
