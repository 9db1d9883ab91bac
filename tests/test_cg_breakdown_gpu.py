"""A guess that holds an infinity has a residual that is NaN.  The step's scalars then say so, whatever an
earlier solve left in their place, and the solver stops at once instead of running to its iteration limit."""
import numpy as np
import pytest

import gridbench_gb300 as gb
from conftest import make_case

pytestmark = pytest.mark.gpu

DIVERGED = 6
M5, MF = 1.8, 0.1


@pytest.mark.parametrize("mode,low,sloppy_residual", [(gb.CG_DOUBLE, gb.F32, 0), (gb.CG_PLAIN, gb.F32, 0),
                                                      (gb.CG_MIXED, gb.F32, 0), (gb.CG_MIXED, gb.F16, 0),
                                                      (gb.CG_MIXED, gb.F16, 1)])
@pytest.mark.parametrize("eo", [False, True])
def test_infinite_guess_diverges(gpu, mode, low, sloppy_residual, eo):
    dims, Ls = (4, 4, 4, 4), 8
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    g64, gl = gb.Gauge(lat, c["U"], gb.F64), gb.Gauge(lat, c["U"], low)
    if eo:
        halves = lat.checkerboard()
        g64, gl = (tuple(g.checkerboard(h) for h in halves) for g in (g64, gl))
    b, x = gb.Field(lat, gb.F64).load(c["phi"]), gb.Field(lat, gb.F64)
    solve = gb.cg_solve_eo if eo else gb.cg_solve
    how = dict(mode=mode, tol=1e-6, max_iter=400, delta=0.1)
    if mode != gb.CG_DOUBLE:
        how.update({"g32": gl} if mode == gb.CG_PLAIN else
                   {"gsloppy": gl, "sloppy_prec": low, "sloppy_residual": sloppy_residual})
    x.zero()
    solve(g64, x, b, M5, MF, **how)  # converges, and leaves its own scalars behind
    bad = c["phi"].copy()
    bad.reshape(c["nsite"], -1)[129, 0] = np.inf  # x = 1, t = 2: an odd site
    x.load(bad)
    with pytest.raises(gb.GbdwError) as e:
        solve(g64, x, b, M5, MF, **how)
    assert e.value.status == DIVERGED
