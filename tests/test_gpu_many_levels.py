"""Columns around the longest that the step kernel's shared memory holds, alone
and in a batch: every length steps (longer ones with a kernel per routine), and
a batch refuses at once what its kernel cannot hold."""
import numpy as np
import pytest

import fall3d_gb300 as F
from fall3d_gb300 import synth

pytestmark = pytest.mark.gpu


def _scenario(nz):
    s = synth.make_scenario("tiny", seed=1, nx=4, ny=3, nz=nz, nc=1, run_h=0.2, H=3000.0)
    return s, np.random.default_rng(nz).random((1, nz + 2, 5, 6)).astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("tile", [None, 3])
@pytest.mark.parametrize("nz", [500, 984, 985, 1023, 1024, 1025, 1027, 1028, 1100])
def test_alone(nz, tile):
    """The cells within binary32 rounding of the plain form's, as in the tests of
    smaller grids (a step rounds each value a few tens of times).  The ghosts
    along the domain's vertical edges are in no stencil; what an upload puts
    there only the in-place forms keep."""
    s, c = _scenario(nz)
    out = []
    for prec in (F.PREC_FP32, F.PREC_FP64):
        g = F.Context(s, prec)
        if tile is not None and prec == F.PREC_FP32:
            g.set_option(F.OPT_TILE, tile)
        g.meteo(0)
        g.source(0)
        g.upload_state(c)
        g.step(3)
        g.sync()
        out.append(g.fields()["c"][:, 1:-1, 1:-1, 1:-1])
        g.close()
    assert np.max(np.abs(out[0] - out[1])) <= 30 * 3 * 2.0 ** -24 * np.max(np.abs(out[1]))


@pytest.mark.parametrize("tile", [0, 3])
def test_in_a_batch(tile):
    longest = None
    b = F.Batch(2)
    b.set_option(F.OPT_TILE, tile)
    for nz in range(1024, 980, -1):
        s, _ = _scenario(nz)
        g = F.Context(s, F.PREC_FP32)
        try:
            slot = b.add(g, max_steps=2)
        except F.F3DError:
            g.close()
            continue
        longest = nz
        b.run()
        b.release(slot)
        g.sync()
        alone = F.Context(s, F.PREC_FP32)
        alone.run(max_steps=2)
        assert np.array_equal(g.fields()["c"], alone.fields()["c"])
        g.close()
        break
    assert longest == 984  # 227 KB less the staging, planes and the batch's tables
    b.close()
