"""Batches on the paths that a small one does not take: so many members that no
column is cut (a launch of a member's own cuts it), and members whose sweep
orders differ (one joins a step after the other), for both tile shapes and
through the graph or not.  Every member has the bits of running alone."""
import pytest

import fall3d_gb300 as F
from fall3d_gb300 import synth
from helpers import assert_same_bits

pytestmark = pytest.mark.gpu


def _scenario(k):
    return synth.make_scenario("small", seed=k, nx=59 + k % 3, ny=27 + k % 2, nz=20 + k % 4, nc=2, wetdep=bool(k % 2),
                               run_h=1.0, H=5000.0)


def _same(ctx, s, steps):
    alone = F.Context(s, F.PREC_FP32)
    alone.run(max_steps=steps)
    a, b = alone.fields(), ctx.fields()
    for k in ("c", "cdry", "cwet"):
        assert_same_bits(b[k], a[k], k)
    alone.close()


@pytest.mark.parametrize("tile", [0, 3])
def test_uncut_columns(tile):
    scen = [_scenario(k) for k in range(8)]
    b = F.Batch(48)
    b.set_option(F.OPT_TILE, tile)
    ctx = [F.Context(scen[q % 8], F.PREC_FP32) for q in range(48)]
    slots = [b.add(c, max_steps=6) for c in ctx]
    b.run()
    for q in slots:
        b.release(q)
    for q in (0, 1, 2, 3, 20, 45, 46, 47):
        _same(ctx[q], scen[q % 8], 6)
    for c in ctx:
        c.close()
    b.close()


@pytest.mark.parametrize("tile,graph", [(0, 1), (3, 1), (3, 0)])
def test_mixed_sweep_orders(tile, graph):
    scen = [_scenario(k) for k in range(5)]
    b = F.Batch(8)
    b.set_option(F.OPT_TILE, tile)
    b.set_option(F.OPT_GRAPH, graph)
    ctx = [F.Context(s, F.PREC_FP32) for s in scen]
    slots = []
    for c in ctx:  # each a step after the one before
        slots.append(b.add(c, max_steps=9))
        b.step()
    b.run()
    for q in slots:
        b.release(q)
    for c, s in zip(ctx, scen):
        _same(c, s, 9)
        c.close()
    b.close()
