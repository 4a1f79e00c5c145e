"""Concentrations at heights above sea level (ter2asl) where successive heights
share a pair of model levels, skip some, or repeat one: stretched, uniform and
decreasing levels over terrain from the sea to above the model top.  Bit for
bit the oracle's restatement."""
import numpy as np
import pytest

import fall3d_gb300 as F
import oracle_lib as O
from fall3d_gb300 import synth

pytestmark = pytest.mark.gpu

Z = {"stretched": lambda n: np.round(50.0 * 1.25 ** np.arange(n) - 50.0), "uniform": lambda n: 400.0 * np.arange(n),
     "shrinking steps": lambda n: np.round(9000.0 * (1.0 - 0.8 ** np.arange(n))),
     "a step down": lambda n: np.where(np.arange(n) == n // 2, 300.0, 400.0 * np.arange(n))}


@pytest.mark.parametrize("prec", [F.PREC_FP64, F.PREC_FP32])
@pytest.mark.parametrize("levels", sorted(Z))
@pytest.mark.parametrize("nc", [1, 9])
def test_heights_above_sea_level(prec, levels, nc):
    nx, ny, nz = 13, 11, 15
    s = synth.make_scenario("small", seed=2, nx=nx, ny=ny, nz=nz, nc=nc, run_h=0.5)
    s.grid["zlayer"] = Z[levels](nz)
    r = np.random.default_rng(nc)
    s.grid["topg"] = r.choice([-50.0, 0.0, 120.0, 800.0, 3333.3, 20000.0], (ny, nx))
    c = np.zeros((nc, nz + 2, ny + 2, nx + 2))
    c[:, 1:-1, 1:-1, 1:-1] = r.random((nc, nz, ny, nx)) * r.choice([0.0, 1.0, 1e-9], (nc, nz, ny, nx))
    g = F.Context(s, prec)
    g.upload_state(c)
    f = g.fields()
    for index in (0, nc):
        got, want = g.output(F.OUT_CON, index, asl=True), O.output(s.grid, f, F.OUT_CON, index, asl=True)
        assert np.array_equal(got, want)
        assert np.max(want) > 0.0
    g.close()
