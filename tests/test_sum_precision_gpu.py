"""What the operators' sums keep: |M x|^2 is FP64 above a thread's 48 squares, whatever its walk along t."""
import pytest

import gridbench_gb300 as gb
from conftest import make_case
from test_sweep_gpu import pin  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,Ls", [((2, 2, 4, 32), 8), ((4, 2, 2, 16), 12), ((2, 4, 2, 16), 16)])
def test_norm_does_not_depend_on_the_slices_of_a_cta(gpu, pin, dims, Ls):  # noqa: F811
    """Every site's squares are the same FP32 number however the CTAs cut t; only FP64 adds differ, of
    fewer than 2^12 terms each off by 2^-53."""
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    g = gb.Gauge(lat, c["U"], gb.F32)
    x, y = gb.Field(lat, gb.F32).load(c["phi"]), gb.Field(lat, gb.F32)
    for dag in (0, 1):
        n = []
        for nt in (2, 5, 16):
            pin(Ls, nt)
            assert gb.tune_query(g, x)[2] == 4
            n.append(gb.dwf_m(g, y, x, 1.8, 0.05, dag, want_norm=True))
        assert max(n) - min(n) < 2.0 ** -41 * n[0], n
