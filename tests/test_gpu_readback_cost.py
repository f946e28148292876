"""What a read-back of a small handle costs: its staging memory is a few
microseconds to make and free whatever the size (the handle's arrays leave
room for it in a page of the device), so macros of 13k nodes take about as
long as those of 3k."""
import time

import pytest
import torch

import porelb_gb300 as P

from helpers import pack_flag

pytestmark = pytest.mark.gpu


def macros_time(dims, porosity, radius):
    flag = pack_flag(dims, 3, radius, radius + 2.0, porosity)
    with P.Simulation.from_flag(flag, *dims, tau=0.8, force=1e-6) as s:
        s.init_dist_macro()
        s.step(2)
        out = torch.empty(4, s.N, dtype=torch.float64, pin_memory=True).numpy()
        best = float("inf")
        for _ in range(50):
            t0 = time.perf_counter()
            s.macros(out=out)
            best = min(best, time.perf_counter() - t0)
        return best


def test_small_handles_stage_cheaply():
    # 27 and 30 us measured; with no room beside the handle's arrays 130
    assert macros_time((32, 32, 32), 0.40, 3.0) < 2.5 * macros_time((20, 20, 20), 0.45, 2.0)
