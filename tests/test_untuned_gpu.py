"""Shapes that run when nothing was tuned, against the oracle: odd extents in slice pairs, the
small-lattice hopping kernel at its edges, the generic form 3, and the Mobius adjoint in one pass for
even Ls that are no power of two.  Extents are ones no other test tunes."""
import numpy as np
import pytest

import gridbench_gb300 as gb
import oracle
from conftest import make_case, rel_err
from oracle import mobius as mob
from test_eo_gpu import halves, masked

pytestmark = pytest.mark.gpu

M5, MF = 1.8, 0.01
TOL = {gb.F64: 1e-12, gb.F32: 1e-6, gb.F16: 5e-3}


@pytest.mark.parametrize("prec", [gb.F32, gb.F64, gb.F16])
@pytest.mark.parametrize("dims,Ls", [((3, 2, 5, 2), 1), ((2, 3, 2, 3), 7), ((5, 4, 3, 2), 9), ((8, 6, 5, 7), 11),
                                     ((4, 4, 4, 4), 22), ((2, 1, 1, 1), 18), ((6, 7, 5, 9), 14)])
def test_untuned_dhop_and_m(gpu, prec, dims, Ls):
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    g = gb.Gauge(lat, c["U"], prec)
    x, y = gb.Field(lat, prec).load(c["phi"]), gb.Field(lat, prec)
    for dag in (0, 1):
        gb.dhop(g, y, x, dag)
        assert rel_err(y.numpy(), oracle.dslash(c["U"], c["phi"], c["nbr"], c["prm"], c["nsite"], Ls, dag)) < TOL[prec]
        n2 = gb.dwf_m(g, y, x, M5, MF, dag, want_norm=True)
        out = y.numpy()
        assert rel_err(out, oracle.dwf_m(c["U"], c["phi"], c["nbr"], c["nsite"], Ls, M5, MF, dag)) < TOL[prec]
        assert abs(n2 - float(np.sum(out ** 2))) / n2 < 1e-5


@pytest.mark.parametrize("Ls", [3, 9])
@pytest.mark.parametrize("form,threads", [(0, 128), (3, 64)])
def test_odd_extents_in_pairs(gpu, Ls, form, threads):
    """Pinned pairs of an odd extent, chained: the padding stays out of the result and of sums."""
    dims = (4, 3, 2, 5)
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    g = gb.Gauge(lat, c["U"], gb.F32)
    x, y, z = gb.Field(lat, gb.F32).load(c["phi"]), gb.Field(lat, gb.F32), gb.Field(lat, gb.F32)
    gb.tune_set(g, x, threads, 2, form, 4)
    gb.dhop(g, y, x, 0)
    gb.dhop(g, z, y, 1)
    one = oracle.dslash(c["U"], c["phi"], c["nbr"], c["prm"], c["nsite"], Ls, 0)
    two = oracle.dslash(c["U"], one, c["nbr"], c["prm"], c["nsite"], Ls, 1)
    assert rel_err(z.numpy(), two) < TOL[gb.F32]
    assert abs(z.norm2() - float(np.sum(two ** 2))) / z.norm2() < 1e-5
    z.axpby(0.5, x, 2.0)
    assert rel_err(z.numpy(), 0.5 * c["phi"] + 2.0 * two) < TOL[gb.F32]
    lt = gb.Lattice.from_table(c["nbr"], c["prm"], c["nsite"], Ls)
    gt = gb.Gauge(lt, c["U"], gb.F32)
    xt, yt = gb.Field(lt, gb.F32, 3), gb.Field(lt, gb.F32, 3)
    for r in range(3):
        xt.load(c["phi"] * (r + 1), r)
    gb.dhop(gt, yt, xt, 0)  # an odd number of slices over three right-hand sides
    for r in range(3):
        assert rel_err(yt.numpy(r), one * (r + 1)) < TOL[gb.F32], r


@pytest.mark.parametrize("dims,Ls", [((2, 2, 2, 2), 6), ((4, 2, 2, 4), 10), ((4, 4, 2, 2), 20), ((2, 2, 4, 2), 34),
                                     ((4, 2, 2, 2), 62)])
def test_mobius_adjoint_for_other_even_ls(gpu, dims, Ls):
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    g = gb.Gauge(lat, c["U"], gb.F32)
    x, y, t = gb.Field(lat, gb.F32).load(c["phi"]), gb.Field(lat, gb.F32), gb.Field(lat, gb.F32)
    for dag in (0, 1):
        n2 = gb.mobius_m(g, y, t, x, 1.5, 0.5, M5, MF, dag, want_norm=True)
        ref = mob.mobius_m(c["U"], c["phi"], c["nbr"], c["prm"], c["nsite"], Ls, 1.5, 0.5, M5, MF, dag)
        out = y.numpy()
        assert rel_err(out, ref) < TOL[gb.F32], dag
        assert abs(n2 - float(np.sum(out ** 2))) / n2 < 1e-5
    if all(d % 2 == 0 for d in dims):
        le, lo = lat.checkerboard()
        ge = g.checkerboard(le)
        xo, ye, te = gb.Field(lo, gb.F32).pick(x), gb.Field(le, gb.F32), gb.Field(le, gb.F32)
        gb.mobius_meooe(ge, ye, te, xo, 1.5, 0.5, MF, 1)
        src = masked(c["phi"], dims, Ls, 1)
        full = mob.mobius_m(c["U"], src, c["nbr"], c["prm"], c["nsite"], Ls, 1.5, 0.5, M5, MF, 1)
        assert rel_err(ye.numpy(), halves(full, dims, Ls)[0]) < TOL[gb.F32]


@pytest.mark.parametrize("dims,Ls", [((8, 8, 8, 11), 24), ((8, 8, 6, 10), 40), ((14, 12, 10, 11), 8)])
def test_untuned_sweep_slices(gpu, dims, Ls):
    """Above 120 thousand 5D sites the t-sweep, with slices per CTA that leave a shorter last piece."""
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    g = gb.Gauge(lat, c["U"], gb.F32)
    x, y = gb.Field(lat, gb.F32).load(c["phi"]), gb.Field(lat, gb.F32)
    for dag in (0, 1):
        gb.dhop(g, y, x, dag)
        assert rel_err(y.numpy(), oracle.dslash(c["U"], c["phi"], c["nbr"], c["prm"], c["nsite"], Ls, dag)) < TOL[gb.F32]
        n2 = gb.dwf_m(g, y, x, M5, MF, dag, want_norm=True)
        out = y.numpy()
        assert rel_err(out, oracle.dwf_m(c["U"], c["phi"], c["nbr"], c["nsite"], Ls, M5, MF, dag)) < TOL[gb.F32]
        assert abs(n2 - float(np.sum(out ** 2))) / n2 < 1e-5
