"""Launches that come up while the one before them drains: a long chain of dependent kernels, in which
every kernel reads what the one before wrote and buffers are reused at once, gives bit for bit what the
same chain gives with a wait after every call."""
import numpy as np
import pytest

import gridbench_gb300 as gb
from conftest import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [gb.F32, gb.F64, gb.F16])
@pytest.mark.parametrize("dims,Ls", [((4, 4, 4, 4), 8), ((3, 2, 5, 2), 7), ((8, 8, 8, 16), 16)])
def test_chain_equals_waited_chain(gpu, prec, dims, Ls):
    c = make_case(dims, Ls)
    lat = gb.Lattice.periodic(dims, Ls)
    g = gb.Gauge(lat, c["U"], prec)

    def chain(wait):
        x, y, z = gb.Field(lat, prec).load(c["phi"]), gb.Field(lat, prec), gb.Field(lat, prec)
        sums, outs = [], []
        for k in range(24):
            for call in (lambda: gb.dhop(g, y, x, k & 1), lambda: z.copy_from(y), lambda: z.axpby(0.25, x, 0.125),
                         lambda: gb.dwf_m(g, x, z, 1.8, 0.05, k & 1), lambda: x.axpby(0.0, z, 0.0625)):
                call()
                if wait:
                    gb.synchronize()
            sums.append(x.norm2())
            if k % 8 == 7:
                outs.append(x.numpy())
        return sums, outs

    sums, outs = chain(False)
    sums_w, outs_w = chain(True)
    assert sums == sums_w and all(np.isfinite(sums))
    assert all(np.array_equal(a, b) for a, b in zip(outs, outs_w))
