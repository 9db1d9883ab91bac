"""What the operators' sums keep: |M x|^2 is FP64 above a thread's 48 squares, whatever its walk along t,
and the FP32 residual's |r|^2 is at least FP64 above one row."""
import ctypes as C

import numpy as np
import pytest

import gridbench_gb300 as gb
from conftest import make_case
from gridbench_gb300 import _native
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


def test_residual_sum_of_fp32_rows(gpu):
    """With zero links, M5 = 5 and mf = 0, M only shifts slices and M^dag M drops the components that leave
    at a wall, so a solve's first step leaves a residual of chosen FP32 numbers there: rows of 1, 2^-26 and
    four of 2^-50 in their squares, which FP64 adds without rounding and 48 bits do not."""
    dims, Ls = (4, 4, 4, 4), 8
    V = 256
    lat = gb.Lattice.periodic(dims, Ls)
    U = np.zeros(V * 8 * 18)
    g64, g32 = gb.Gauge(lat, U, gb.F64), gb.Gauge(lat, U, gb.F32)
    b = np.zeros((V, Ls, 12, 2))
    b[:, Ls - 1, :6, 0] = [1.0, 2.0 ** -13] + 4 * [2.0 ** -25]  # spins 0 and 1 at the last slice
    b[7, 3, 2, 1] = 2.0 ** 24                                   # what the step removes: alpha = 1 + 2^-40
    want = V * (1.0 + 2.0 ** -26 + 2.0 ** -48)
    bb = want + 2.0 ** 48
    x, rhs = gb.Field(lat, gb.F64), gb.Field(lat, gb.F64).load(b)
    x.zero()
    prm = _native.CGParams(1e-12, 1, 1e-10, gb.F32, gb.F32, 0)
    st = _native.CGStats()
    lib = gb.load()
    status = lib.gbdw_cg_solve(g64.h, None, g32.h, x.h, rhs.h, 5.0, 0.0, gb.CG_MIXED, C.byref(prm),
                               C.byref(st))
    assert status == 5 and st.iterations == 1 and st.reliable_updates == 0  # the iteration limit
    assert abs(st.final_rr * bb - want) <= 2.0 ** -51 * want, (st.final_rr * bb - want) / want
