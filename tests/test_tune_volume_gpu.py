"""A t-sweep chosen by the tuner on one lattice does not decide for lattices of another volume with the same
slices: there the rules by size hold.  A pinned shape holds everywhere."""
import pytest

from fresh_process import run_fresh

pytestmark = pytest.mark.gpu

SETUP = """
import gridbench_gb300 as gb
def case(dims):
    lat = gb.Lattice.periodic(dims, 8)
    g = gb.Gauge(lat, None, gb.F32, seed=3)
    return lat, g, gb.Field(lat, gb.F32).gaussian(1), gb.Field(lat, gb.F32)
lat, g, x, y = case((16, 16, 16, 16))
l8, g8, x8, y8 = case((8, 8, 8, 8))
untuned = gb.tune_query(g8, x8), gb.tune_query_m(g8, x8)
"""


def test_tuned_sweep_stays_with_its_volume(gpu, tmp_path):
    path = str(tmp_path / "tune.json")
    run_fresh(SETUP + f"""
gb.tune_dhop(g, y, x)
assert gb.tune_query(g, x)[2] == 4 and gb.tune_query_m(g, x)[2] == 4
assert (gb.tune_query(g8, x8), gb.tune_query_m(g8, x8)) == untuned
gb.tune_save({path!r})
""")
    run_fresh(SETUP + f"""
gb.tune_load({path!r})
assert gb.tune_query(g, x)[2] == 4 and gb.tune_query_m(g, x)[2] == 4
assert (gb.tune_query(g8, x8), gb.tune_query_m(g8, x8)) == untuned
gb.tune_set(g, x, 64, 2, 4, 4)
assert gb.tune_query(g8, x8)[2] == 4
""")
