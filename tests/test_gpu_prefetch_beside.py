"""The step kernel's build for a look-ahead update in flight (64x32 tiles, fewer
registers): runs that take it, because the tile shape was set or because the
grid has more 64x16 tiles than the device has SMs, give the bits of runs
that make every update when it is due.  Both sweep orders, wet deposition,
eight updates; that the build was launched is read from the profile."""
import numpy as np
import pytest

import fall3d_gb300 as F
from fall3d_gb300 import synth
from helpers import assert_same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modv", [2, 4])
@pytest.mark.parametrize("nx,ny,nz,nc,tile", [(32, 28, 14, 4, 3), (59, 27, 21, 2, 3), (120, 121, 12, 6, None)])
def test_steps_beside_an_update(nx, ny, nz, nc, tile, modv):
    s = synth.make_scenario("small", seed=21, nx=nx, ny=ny, nz=nz, nc=nc, run_h=2.0, met_dt_h=0.25, wetdep=True,
                            modv=modv)
    s.met["prate"][:] = np.float32(2.0 / 3600.0)
    runs = []
    for pref in (0, 1):
        g = F.Context(s, F.PREC_FP32)
        if tile is not None:
            g.set_option(F.OPT_TILE, tile)
        g.set_option(F.OPT_PREFETCH, pref)
        g.profile(True)
        log = g.run()
        steps = g.profile_read()
        runs.append((g.fields(), log, g.state(), g.iters(), {k: v[0] for k, v in steps.items()}))
        g.close()
    (fa, la, sa, ia, pa), (fb, lb, sb, ib, pb) = runs
    assert pa.get("step_beside", 0) == 0
    assert pb.get("step_beside", 0) >= 8 and pb.get("step_beside", 0) + pb.get("step_fused", 0) == pa["step_fused"]
    for k in ("c", "cdry", "cwet", "vset", "vdep"):
        assert_same_bits(fa[k], fb[k], k)
    for k in la:
        assert_same_bits(np.asarray(la[k], float), np.asarray(lb[k], float), "log " + k)
    assert sa == sb and np.array_equal(ia, ib)
    assert np.max(fa["c"]) > 0.0
