"""The drop-in call's own memory: lattice, links and fields out of one kept buffer, host arrays read in place.
Calls of changing size reuse that buffer, arrays off a 16-byte boundary are copied, and a table whose s
neighbours do not follow the 4D ones takes the general path; every result equals the one of objects
made one by one, which neither shares memory nor reads host arrays in place."""
import numpy as np
import pytest

import gridbench_gb300 as gb
from conftest import make_case

pytestmark = pytest.mark.gpu


def shifted(a, by):
    raw = np.zeros(a.nbytes + 64, dtype=np.uint8)
    off = (-raw.ctypes.data) % 64 + by
    out = raw[off:off + a.nbytes].view(a.dtype).reshape(a.shape)
    out[...] = a
    return out


def objects(c, Ls, nsimd, dt, dag):
    lat = gb.Lattice.from_table(c["nbr"], c["prm"], c["nsite"], Ls, nsimd)
    prec = gb.F64 if dt == np.float64 else gb.F32
    x, y = gb.Field(lat, prec).load(c["phi"].astype(dt)), gb.Field(lat, prec)
    gb.dhop(gb.Gauge(lat, c["U"].astype(dt), prec), y, x, dag)
    out = np.empty_like(c["phi"], dtype=dt)
    y.export_into(out)
    return out


@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("by", [0, 8])
def test_seam_equals_objects(gpu, dt, by):
    for dims, Ls, nsimd in (((4, 4, 4, 4), 3, 1), ((2, 3, 5, 2), 1, 1), ((8, 4, 4, 8), 8, 4), ((2, 2, 2, 2), 9, 1)):
        c = make_case(dims, Ls, nsimd)
        for dag in (0, 1):
            want = objects(c, Ls, nsimd, dt, dag)
            out = shifted(np.zeros_like(c["phi"], dtype=dt), by)
            gb.dslash_kernel(2, shifted(c["U"].astype(dt), by), out, shifted(c["phi"].astype(dt), by),
                             shifted(c["nbr"], by), c["nsite"], Ls, c["prm"], nsimd, dag)
            assert np.array_equal(out, want)


def test_seam_general_table_and_refusal(gpu):
    dims, Ls = (4, 2, 2, 4), 4
    c = make_case(dims, Ls)
    nbr = c["nbr"].reshape(c["nsite"], Ls, 8).copy()
    nbr[:, :, 2] = nbr[:, ::-1, 2].copy()  # s neighbours out of order: not a product of a 4D table
    c["nbr"] = nbr.reshape(c["nbr"].shape)
    want = objects(c, Ls, 1, np.float64, 0)
    out = np.zeros_like(c["phi"])
    gb.dslash_kernel(1, c["U"], out, c["phi"], c["nbr"], c["nsite"], Ls, c["prm"])
    assert np.array_equal(out, want)
    bad = c["nbr"].copy()
    bad.reshape(-1)[5] = c["nsite"] * Ls
    with pytest.raises(gb.GbdwError):
        gb.dslash_kernel(1, c["U"], out, c["phi"], bad, c["nsite"], Ls, c["prm"])
    gb.dslash_kernel(1, c["U"], out, c["phi"], c["nbr"], c["nsite"], Ls, c["prm"])
    assert np.array_equal(out, want)
