"""Pinning a tile split or a t-brick on a field that nothing was tuned for: it is taken (or refused) by
the same rules on every lattice size, whichever form the untuned field runs."""
import pytest

from fresh_process import run_fresh

pytestmark = pytest.mark.gpu

PINS = """
import numpy as np, pytest
import gridbench_gb300 as gb
dims, Ls, form, split, brick, no_brick = {}
lat = gb.Lattice.periodic(dims, Ls)
g = gb.Gauge(lat, None, gb.F32, seed=3)
x, y, z = gb.Field(lat, gb.F32).gaussian(1), gb.Field(lat, gb.F32), gb.Field(lat, gb.F32)
assert gb.tune_query(g, x)[2] == form
gb.dhop(g, y, x)
with pytest.raises(gb.GbdwError):
    gb.tune_set_brick(g, x, no_brick)      # does not divide Lt
with pytest.raises(gb.GbdwError):
    gb.tune_set_split(g, x, 64)            # no whole slice groups
assert gb.tune_query(g, x)[2] == form      # a refusal pins nothing
{}
assert gb.tune_query(g, x)[2] in (0, 3)
gb.dhop(g, z, x)
z.axpby(-1.0, y, 1.0)
assert z.norm2() < 1e-12 * y.norm2()
"""


@pytest.mark.parametrize("dims,Ls,form,split,brick,no_brick", [
    ((16, 16, 16, 16), 16, 4, 2, 2, 3),    # the t-sweep
    ((16, 16, 16, 12), 30, 2, 3, 2, 5),    # the warp rings
    ((4, 4, 4, 6), 9, 3, 3, 3, 4)])        # form 3, an odd extent
def test_split_and_brick_on_untuned_fields(gpu, dims, Ls, form, split, brick, no_brick):
    case = repr((dims, Ls, form, split, brick, no_brick))
    run_fresh(PINS.format(case, "gb.tune_set_split(g, x, split)\nassert gb.tune_split(g, x) == split"))
    run_fresh(PINS.format(case, "gb.tune_set_brick(g, x, brick)\nassert gb.tune_brick(g, x) == brick"))
