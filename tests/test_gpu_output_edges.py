"""Output variables where their kernels can go wrong: columns shorter than,
equal to and one beyond a group of eight levels, planes that are no multiple
of a block, more classes than a kernel parameter holds, states with zeros,
subnormal and large values.  Bit for bit the oracle's restatement on the same
state (binary64 in the reference's order of operations)."""
import numpy as np
import pytest

import fall3d_gb300 as F
import oracle_lib as O
from fall3d_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [F.PREC_FP64, F.PREC_FP32])
@pytest.mark.parametrize("nx,ny,nz,nc", [(3, 3, 3, 1), (31, 3, 7, 2), (32, 4, 8, 9), (11, 7, 9, 8), (9, 8, 17, 17),
                                         (8, 9, 16, 130)])
def test_outputs_at_edges(prec, nx, ny, nz, nc):
    s = synth.make_scenario("small", seed=3, nx=nx, ny=ny, nz=nz, nc=nc, phimin=3.0, phimax=9.0, run_h=0.6)
    r = np.random.default_rng(nx * nz)
    c = np.zeros((nc, nz + 2, ny + 2, nx + 2))
    shape = c[:, 1:-1, 1:-1, 1:-1].shape
    c[:, 1:-1, 1:-1, 1:-1] = r.random(shape) * r.choice([0.0, 0.0, 1.0, 1e-12, 1e-42, 1e20], shape)
    if nc > 1:
        c[-1, 1:-1, 1:-1, 1] = 0.0
    g = F.Context(s, prec)
    g.meteo(0)
    dep = r.random((nc + 1, ny, nx)) * r.choice([0.0, 1.0, 1e-9], (nc + 1, ny, nx))
    g.upload_state(c, dep, 0.5 * dep)
    f = g.fields()
    var = [(F.OUT_COL_MASS, 0), (F.OUT_PM_COL, 20), (F.OUT_C_GRND, 0), (F.OUT_PM_GRND, 20), (F.OUT_AOT05, 0),
           (F.OUT_CON, 0), (F.OUT_CON, nc)]
    for v, index in var:
        for asl in ((False, True) if v == F.OUT_CON else (False,)):
            got, want = g.output(v, index, asl=asl), O.output(s.grid, f, v, index, asl=asl)
            assert np.array_equal(got, want), (v, index, asl)
            g32 = g.output(v, index, asl=asl, binary32=True)
            with np.errstate(over="ignore"):
                assert np.array_equal(g32, got.astype(np.float32)), (v, index, asl)
    assert np.max(g.output(F.OUT_COL_MASS, 0)) > 0.0
    g.close()
