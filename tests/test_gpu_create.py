"""What it costs to create and release a domain."""
import time

import pytest

import pbpic_b200
from pbpic_b200 import configs

pytestmark = pytest.mark.gpu


def test_creating_a_domain_costs_the_same_at_any_size(gpu_lib):
    """A domain's arrays are one allocation: a million particles (75 MB) take at most twice the time of a
    few hundred. (With an allocation an array, each of a megabyte or more mapped by
    itself, they took 4.4 times as long to create.)"""
    best = {}
    for side, ppc in ((16, 1), (128, 32)):
        cfg, _ = configs.uniform_c1(mx=side, my=side, ppc=ppc)
        for _ in range(12):
            t = time.perf_counter()
            s = pbpic_b200.Simulation.from_config(cfg, precision="fp32", capacity=2 * side * side * ppc)
            t = time.perf_counter() - t
            s.close()
            best[side] = min(t, best.get(side, t))
    assert best[128] <= 2.0 * best[16], best
