"""The t-sweep as an untuned field takes it, in a process where nothing was tuned or pinned: the form and
the slices of t per CTA that the rules choose, with a shorter last piece, against the oracle."""
import pytest

from fresh_process import run_fresh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,Ls,m", [((8, 8, 8, 11), 24, False), ((8, 8, 6, 11), 40, False),
                                       ((14, 12, 10, 11), 8, True), ((10, 8, 8, 17), 12, True)])
def test_untuned_sweep(gpu, dims, Ls, m):
    run_fresh(f"""
import numpy as np, oracle
import gridbench_gb300 as gb
from conftest import make_case, rel_err
dims, Ls, m = {dims}, {Ls}, {m}
c = make_case(dims, Ls)
lat = gb.Lattice.periodic(dims, Ls)
g = gb.Gauge(lat, c["U"], gb.F32)
x, y = gb.Field(lat, gb.F32).load(c["phi"]), gb.Field(lat, gb.F32)
assert gb.tune_query(g, x)[2] == 4 and dims[3] % gb.tune_brick(g, x) != 0, gb.tune_brick(g, x)
assert (gb.tune_query_m(g, x)[2] == 4) == m
for dag in (0, 1):
    gb.dhop(g, y, x, dag)
    assert rel_err(y.numpy(), oracle.dslash(c["U"], c["phi"], c["nbr"], c["prm"], c["nsite"], Ls, dag)) < 1e-6
    n2 = gb.dwf_m(g, y, x, 1.8, 0.01, dag, want_norm=True)
    out = y.numpy()
    assert rel_err(out, oracle.dwf_m(c["U"], c["phi"], c["nbr"], c["nsite"], Ls, 1.8, 0.01, dag)) < 1e-6
    assert abs(n2 - float(np.sum(out ** 2))) / n2 < 1e-7
""")
