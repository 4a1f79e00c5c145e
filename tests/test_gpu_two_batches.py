"""Two batches alive at the same time, stepped in turn and from two threads,
with members of different sizes and counts: each member has the bits of
running alone.  (The step kernel's arguments of one batch must not be those of
the other.)"""
import threading

import pytest

import fall3d_gb300 as F
from fall3d_gb300 import synth
from helpers import assert_same_bits

pytestmark = pytest.mark.gpu
STEPS = 12


def _members(first, sizes):
    return [synth.make_scenario("small", seed=first + k, nx=nx, ny=ny, nz=nz, nc=nc, run_h=1.0, H=5000.0,
                                wetdep=bool(k % 2)) for k, (nx, ny, nz, nc) in enumerate(sizes)]


SETS = [_members(1, [(64, 33, 24, 3), (30, 28, 14, 2), (59, 61, 17, 2)]), _members(9, [(21, 12, 40, 1), (90, 20, 12, 4)])]


def _alone(s):
    g = F.Context(s, F.PREC_FP32)
    g.run(max_steps=STEPS)
    f = g.fields()
    g.close()
    return f


def _start(scen, tile):
    b = F.Batch(4)
    b.set_option(F.OPT_TILE, tile)
    ctx = [F.Context(s, F.PREC_FP32) for s in scen]
    return b, ctx, [b.add(c, max_steps=STEPS) for c in ctx]


def _check(b, ctx, slots, scen):
    b.sync()
    for q in slots:
        b.release(q)
    for c, s in zip(ctx, scen):
        a, f = _alone(s), c.fields()
        for k in ("c", "cdry", "cwet"):
            assert_same_bits(f[k], a[k], k)
        c.close()
    b.close()


@pytest.mark.parametrize("tiles", [(3, 3), (0, 3)])
def test_in_turn(tiles):
    runs = [_start(scen, tile) for scen, tile in zip(SETS, tiles)]
    for _ in range(STEPS):
        for b, _, _ in runs:
            b.step()
    for (b, ctx, slots), scen in zip(runs, SETS):
        _check(b, ctx, slots, scen)


def test_from_two_threads():
    runs = [_start(scen, 3) for scen in SETS]
    errors = []

    def go(b):
        try:
            b.run()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=go, args=(b,)) for b, _, _ in runs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for (b, ctx, slots), scen in zip(runs, SETS):
        _check(b, ctx, slots, scen)
