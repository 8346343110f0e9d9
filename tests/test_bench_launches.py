"""bench.py's launch count and flux kernel name follow what the grid runs,
by the library's rules as well as by a knob."""
import importlib.util
import os

import pytest

from test_fx_launch_choice import by_rule, choice, counts  # noqa: F401  (by_rule: autouse fixture)

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def bench():
    spec = importlib.util.spec_from_file_location("bench_module", os.path.join(REPO, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


@pytest.mark.parametrize("n,launches,kernel", [(128, 11, "k_fx_flux_tile"), (8, 9, "k_fx_flux")])
def test_by_rule_and_by_knob(n, launches, kernel):
    from bhgpu import fixed as fx

    class Grid:
        def launch_choice(self, knob):
            return choice(knob, "mixed", counts(n))
    b, g = bench(), Grid()
    assert (b.step_launches(g), b.flux_kernel(g)) == (launches, kernel)
    fx.tune_set("mixed", "split", 0)
    fx.tune_set("mixed", "stage", 1)
    assert (b.step_launches(g), b.flux_kernel(g)) == (9, "k_fx_flux_tile")
