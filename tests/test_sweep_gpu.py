"""The t-sweep form of the FP32 hopping kernel (2x2x2 columns walked along t) against the oracle:
every epilogue, whole rows and slice tiles, full and half lattices, chunks of t that do and do not
divide Lt, the smallest extents it takes, and the shapes it leaves to the other forms."""
import json

import numpy as np
import pytest

import gridbench_gb300 as gb
import oracle
from conftest import make_case, rel_err
from oracle import mobius as mob
from test_eo_gpu import halves, masked

pytestmark = pytest.mark.gpu

M5, MF = 1.8, 0.01
TOL = 1e-6  # FP32 against the FP64 oracle, as for every other form


@pytest.fixture
def pin(gpu, tmp_path):
    """Pins the sweep form (nt slices of t per CTA) for rows of LsE slices through a tune-cache file;
    afterwards those keys hold the untuned default again."""
    pinned = set()

    def write(LsE, shape):
        f = tmp_path / "pin.json"
        f.write_text(json.dumps({f"g1_s1_L{LsE}_e{e}": shape for e in (0, 1, 16, 17, 32, 33)}))
        gb.tune_load(str(f))

    def do(LsE, nt):
        pinned.add(LsE)
        write(LsE, [64, 2, 4, 4, 1, nt])

    yield do
    for LsE in pinned:
        write(LsE, [128, 2, 0, 4, 1, 1])


@pytest.mark.parametrize("dims,Ls,nt", [((2, 2, 2, 1), 8, 8), ((2, 2, 2, 3), 16, 2), ((4, 2, 6, 5), 12, 4),
                                        ((6, 4, 2, 8), 16, 8), ((4, 4, 4, 9), 8, 4), ((4, 2, 2, 4), 16, 16)])
def test_sweep_dhop_m_and_mobius(gpu, pin, dims, Ls, nt):
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    g = gb.Gauge(lat, c["U"], gb.F32)
    x, y, t = gb.Field(lat, gb.F32).load(c["phi"]), gb.Field(lat, gb.F32), gb.Field(lat, gb.F32)
    pin(Ls, nt)
    assert gb.tune_query(g, x)[2] == 4
    for dag in (0, 1):
        y.zero()
        gb.dhop(g, y, x, dag)
        assert rel_err(y.numpy(), oracle.dslash(c["U"], c["phi"], c["nbr"], c["prm"], c["nsite"], Ls, dag)) < TOL
        n2 = gb.dwf_m(g, y, x, M5, MF, dag, want_norm=True)
        out = y.numpy()
        assert rel_err(out, oracle.dwf_m(c["U"], c["phi"], c["nbr"], c["nsite"], Ls, M5, MF, dag)) < TOL
        assert abs(n2 - float(np.sum(out ** 2))) / n2 < 1e-5
        gb.mobius_m(g, y, t, x, 1.5, 0.5, M5, MF, dag)  # fused where Ls is a power of two
        ref = mob.mobius_m(c["U"], c["phi"], c["nbr"], c["prm"], c["nsite"], Ls, 1.5, 0.5, M5, MF, dag)
        assert rel_err(y.numpy(), ref) < TOL, dag


@pytest.mark.parametrize("dims,Ls,nrhs", [((2, 4, 2, 5), 8, 2), ((4, 2, 2, 4), 12, 12), ((2, 2, 4, 3), 16, 3),
                                          ((2, 2, 2, 4), 24, 1), ((4, 2, 2, 2), 5, 8)])
def test_sweep_slice_tiles(gpu, pin, dims, Ls, nrhs):
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    g = gb.Gauge(lat, c["U"], gb.F32)
    X, Y = gb.Field(lat, gb.F32, nrhs), gb.Field(lat, gb.F32, nrhs)
    srcs = [gb.generate_fermion(dims, Ls, 1, (5 + r, 6, 7, 8)) for r in range(nrhs)]
    for r in range(nrhs):
        X.load(srcs[r], r)
    pin(Ls * nrhs, 4)
    for dag in (0, 1):
        gb.dhop(g, Y, X, dag)
        for r in range(nrhs):
            ref = oracle.dslash(c["U"], srcs[r], c["nbr"], c["prm"], c["nsite"], Ls, dag)
            assert rel_err(Y.numpy(r), ref) < TOL, (dag, r)


@pytest.mark.parametrize("dims,Ls,nt", [((4, 2, 2, 4), 8, 4), ((8, 4, 2, 6), 12, 4), ((4, 4, 6, 4), 16, 8)])
def test_sweep_half_lattices(gpu, pin, dims, Ls, nt):
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    g = gb.Gauge(lat, c["U"], gb.F32)
    le, lo = lat.checkerboard()
    G = (g.checkerboard(le), g.checkerboard(lo))
    L = (le, lo)
    x = gb.Field(lat, gb.F32).load(c["phi"])
    X = [gb.Field(L[k], gb.F32).pick(x) for k in (0, 1)]
    pin(Ls, nt)
    for par in (0, 1):
        src = masked(c["phi"], dims, Ls, 1 - par)
        out = gb.Field(L[par], gb.F32)
        for dag in (0, 1):
            full = oracle.dslash(c["U"], src, c["nbr"], c["prm"], c["nsite"], Ls, dag)
            gb.dhop_eo(G[par], out, X[1 - par], dag)
            assert rel_err(out.numpy(), halves(full, dims, Ls)[par]) < TOL, (par, dag)
            # M's rows of this parity
            gb.dwf_meo(G[par], out, X[1 - par], X[par], M5, MF, dag)
            ref = oracle.dwf_m(c["U"], c["phi"], c["nbr"], c["nsite"], Ls, M5, MF, dag)
            assert rel_err(out.numpy(), halves(ref, dims, Ls)[par]) < TOL, (par, dag)


def test_sweep_in_the_solvers(gpu, pin):
    """The residual epilogues (FP64 and FP32 r) in whole solves: the returned true residual, which the
    FP64 operator computes, reaches the tolerance."""
    dims, Ls = (4, 4, 4, 4), 8
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    g64, g32 = gb.Gauge(lat, c["U"], gb.F64), gb.Gauge(lat, c["U"], gb.F32)
    b = gb.Field(lat, gb.F64).load(c["phi"])
    pin(Ls, 4)
    for kw in (dict(mode=gb.CG_PLAIN, g32=g32), dict(mode=gb.CG_MIXED, gsloppy=g32, sloppy_prec=gb.F32)):
        x = gb.Field(lat, gb.F64)
        x.zero()
        st = gb.cg_solve(g64, x, b, M5, 0.1, tol=1e-10, **kw)
        t, r = gb.Field(lat, gb.F64), gb.Field(lat, gb.F64)
        gb.dwf_mdagm(g64, r, t, x, M5, 0.1)
        assert st["true_residual"] <= 1e-10
        assert rel_err(r.numpy(), c["phi"]) < 2e-10


def test_sweep_falls_back_where_it_does_not_apply(gpu, pin):
    """Odd extents, table lattices and FP16 fields run another form under the same pin."""
    for dims in ((3, 2, 2, 4), (2, 5, 2, 4), (4, 2, 3, 2)):
        c = make_case(dims, 8)
        pin(8, 4)
        for lat in (gb.Lattice.periodic(dims, 8), gb.Lattice.from_table(c["nbr"], c["prm"], c["nsite"], 8)):
            g = gb.Gauge(lat, c["U"], gb.F32)
            x, y = gb.Field(lat, gb.F32).load(c["phi"]), gb.Field(lat, gb.F32)
            gb.dhop(g, y, x)
            assert rel_err(y.numpy(), oracle.dslash(c["U"], c["phi"], c["nbr"], c["prm"], c["nsite"], 8)) < TOL
