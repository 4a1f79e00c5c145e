"""The settling chain cut into segments of whole columns (the iterating drag
models) and of any length: columns shorter than, as long as and longer than
the shortest segment, last segments of a single column, all four models.  The
oracle's iteration counts, velocities and chain value to 1e-12, and the same
bits from an update made ahead of its time (which takes its segments from a
counter)."""
import numpy as np
import pytest

import fall3d_gb300 as F
import oracle_lib as O
from fall3d_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modv", [1, 2, 3, 4])
@pytest.mark.parametrize("nx,ny,nz,nc", [(5, 4, 63, 2), (5, 4, 64, 3), (3, 5, 65, 2), (7, 3, 130, 1), (31, 17, 6, 3),
                                         (61, 40, 21, 4)])
def test_against_the_oracle(nx, ny, nz, nc, modv):
    s = synth.make_scenario("tiny", seed=1, nx=nx, ny=ny, nz=nz, nc=nc, modv=modv, run_h=0.5)
    o = O.OracleCtx(s)
    o.meteo(0)
    ref = o.fields()["vset"]
    g = F.Context(s, F.PREC_FP64)
    g.meteo(0)
    vset = g.fields()["vset"]
    assert np.max(np.abs(vset / ref - 1.0)) <= 1e-12
    assert np.array_equal(g.iters(), o.iters())
    assert abs(g.state()["cd"] / o.state()["cd"] - 1.0) <= 1e-12
    g.close()


@pytest.mark.parametrize("modv", [1, 2, 3, 4])
def test_made_ahead(modv):
    s = synth.make_scenario("small", seed=8, nx=61, ny=40, nz=21, nc=4, modv=modv, run_h=0.6, met_dt_h=0.25)
    out = []
    for pref in (0, 1):
        g = F.Context(s, F.PREC_FP64)
        g.set_option(F.OPT_PREFETCH, pref)
        g.run()
        out.append((g.fields()["vset"], g.iters(), g.state()["cd"]))
        g.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
