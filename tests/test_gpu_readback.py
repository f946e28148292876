"""Read-backs make the pages of a fresh host buffer present before the device
writes them, from four threads above 16 MB.  The values equal a read into
pinned memory, whatever the buffer's place, and what lies next to it in its
pages is left alone."""
import ctypes

import numpy as np
import pytest
import torch

import porelb_gb300 as P

pytestmark = pytest.mark.gpu
GUARD = 7


@pytest.mark.parametrize("edge", [12, 40, 90, 128])
@pytest.mark.parametrize("rows", ["together", "apart", "some"])
def test_fresh_buffers(edge, rows):
    with P.Simulation.packed(2, edge, edge, edge, 0.1 * edge, 0.2 * edge, 0.35, tau=0.8,
                             force=1e-5, precision="fp32") as sim:
        sim.init_dist_macro()
        sim.step(3)
        n = sim.N
        want = torch.empty((4, n), dtype=torch.float64, pin_memory=True).numpy()
        sim.macros(out=want)
        gap = 0 if rows == "together" else 1001
        buf = np.full(4 * (n + gap) + 2 * GUARD, -5.0)
        fresh = np.empty(buf.size)          # pages that nothing has touched
        at = [GUARD + c * (n + gap) for c in range(4)]
        use = [c != 2 or rows != "some" for c in range(4)]
        for a in (buf, fresh):
            ptr = [ctypes.c_void_p(a.ctypes.data + 8 * at[c]) if use[c] else None
                   for c in range(4)]
            assert sim._lib.plb_get_macros(sim._h, *ptr) == 0
            for c in range(4):
                if use[c]:
                    assert np.array_equal(a[at[c]:at[c] + n], want[c])
        left = np.ones(buf.size, bool)
        for c in range(4):
            if use[c]:
                left[at[c]:at[c] + n] = False
        assert (buf[left] == -5.0).all()
        f = sim.get_f()
        twice = sim.get_f()
        assert np.array_equal(f, twice)
