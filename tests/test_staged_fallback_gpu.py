"""A warp-ring shape pinned with one slice per thread, whose rings no longer fit once the Mobius adjoint asks
for two: the pass runs in form 0, with form 0's count of CTAs for the sum."""
import pytest

from fresh_process import run_fresh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ls", [4, 8])
def test_mobius_adjoint_where_the_rings_do_not_fit(gpu, Ls):
    run_fresh(f"""
import numpy as np
import gridbench_gb300 as gb
from conftest import make_case, rel_err
from oracle import mobius as mob
dims, Ls = (4, 4, 4, 6), {Ls}
c = make_case(dims, Ls)
lat = gb.Lattice.periodic(dims, Ls)
g = gb.Gauge(lat, c["U"], gb.F32)
x, y, t = gb.Field(lat, gb.F32).load(c["phi"]), gb.Field(lat, gb.F32), gb.Field(lat, gb.F32)
gb.tune_set(g, x, 256, 1, 2, 4)
n2 = gb.mobius_m(g, y, t, x, 1.5, 0.5, 1.8, 0.05, 1, want_norm=True)
out = y.numpy()
assert rel_err(out, mob.mobius_m(c["U"], c["phi"], c["nbr"], c["prm"], c["nsite"], Ls, 1.5, 0.5, 1.8, 0.05, 1)) < 1e-6
assert abs(n2 - float(np.sum(out ** 2))) < 1e-6 * n2
""")
