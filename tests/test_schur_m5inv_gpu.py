"""D5^-1 in the hopping kernel's epilogue: Mpc and its adjoint against their three factors applied one by
one (hopping term, D5^-1, Schur step), at every window count of the lane recursion: one to 32 slice pairs
on form 3, and 4, 6 and 8 on the t-sweep.  Both orders round each FP32 step once, so they differ by a few
1e-7; FP16 storage in between differs by its own rounding, 2^-11 of a slice's largest component."""
import numpy as np
import pytest

import gridbench_gb300 as gb
from conftest import make_case, rel_err

pytestmark = pytest.mark.gpu

M5 = 1.8


def tuned(tmp_path, shape, prec, Ls):
    p = tmp_path / "tune.json"
    p.write_text("{\n" + ",\n".join(f'  "g{prec}_s{prec}_L{Ls}_e{e}": {shape}' for e in (32, 33)) + "\n}\n")
    gb.tune_load(str(p))


@pytest.mark.parametrize("dag", [0, 1])
@pytest.mark.parametrize("mf", [0.05, 1.0])
@pytest.mark.parametrize("prec,form,Ls,dims", [
    (gb.F32, 3, 2, (4, 2, 2, 4)), (gb.F32, 3, 4, (2, 2, 4, 2)), (gb.F32, 3, 8, (4, 4, 2, 2)),
    (gb.F32, 3, 16, (2, 4, 2, 6)), (gb.F32, 3, 32, (4, 2, 2, 2)), (gb.F32, 3, 64, (2, 2, 2, 2)),
    (gb.F32, 4, 8, (4, 2, 4, 6)), (gb.F32, 4, 12, (8, 2, 2, 4)), (gb.F32, 4, 16, (4, 4, 2, 2)),
    (gb.F16, 3, 16, (4, 2, 2, 6))])
def test_fused_equals_factors(gpu, tmp_path, prec, form, Ls, dims, mf, dag):
    tuned(tmp_path, [64, 2, form, 4, 1, 4 if form == 4 else 1], prec, Ls)
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    even, odd = lat.checkerboard()
    g = gb.Gauge(lat, c["U"], prec)
    ge, go = g.checkerboard(even), g.checkerboard(odd)
    x = gb.Field(odd, prec).pick(gb.Field(lat, prec).load(c["phi"]))
    out, t1, t2 = gb.Field(odd, prec), gb.Field(even, prec), gb.Field(even, prec)
    before = gb.launch_count()
    gb.dwf_mpc(go, ge, out, t1, t2, x, M5, mf, dag)
    assert gb.launch_count() - before == 2
    want, u1, u2 = gb.Field(odd, prec), gb.Field(even, prec), gb.Field(even, prec)
    gb.dhop_eo(ge, u1, x, dag)
    gb.dwf_m5inv(u2, u1, M5, mf, dag)
    gb.dwf_meo(go, want, u2, x, M5, mf, dag, khop=0.25)
    tol = 1e-6 if prec == gb.F32 else 2e-3
    assert rel_err(t2.numpy(), u2.numpy()) < tol
    assert rel_err(out.numpy(), want.numpy()) < tol
