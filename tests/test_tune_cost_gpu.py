"""What the tuner costs: shapes far from the fastest are given up after four launches, so that at 16^4 x 8 it takes
fewer than the 2296 launches that it took before the t-sweep and the general form 3 were among its shapes."""
import pytest

from fresh_process import run_fresh

pytestmark = pytest.mark.gpu


def test_tuner_launches(gpu):
    run_fresh("""
import gridbench_gb300 as gb
lat = gb.Lattice.periodic((16, 16, 16, 16), 8)
g = gb.Gauge(lat, None, gb.F32, seed=3)
x, y = gb.Field(lat, gb.F32).gaussian(1), gb.Field(lat, gb.F32)
gb.dhop(g, y, x)
before = gb.launch_count()
gb.tune_dhop(g, y, x)
n = gb.launch_count() - before
assert n < BOUND, n
""".replace("BOUND", "2296"))
