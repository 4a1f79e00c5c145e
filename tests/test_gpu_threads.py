"""Contexts of different column and line lengths stepped from several threads
at once: every one has the bits of being stepped alone, and no launch fails.
(The kernels' shared-memory limits must not depend on who launched last.)"""
import threading

import numpy as np
import pytest

import fall3d_gb300 as F
from fall3d_gb300 import synth

pytestmark = pytest.mark.gpu
STEPS = 3000


def _scenarios(prec):
    sizes = [(5, 4, 8, 1), (5, 4, 300, 1), (6, 5, 900, 1), (40, 30, 10, 2)] if prec == F.PREC_FP32 else \
            [(1500, 3, 3, 1), (3, 1400, 3, 1), (3000, 3, 3, 1), (3, 3900, 3, 1)]
    return [synth.make_scenario("tiny", seed=k, nx=nx, ny=ny, nz=nz, nc=nc, spacing=0.002, run_h=0.3, H=2500.0)
            for k, (nx, ny, nz, nc) in enumerate(sizes)]


def _steps(s, prec, out, k):
    try:
        g = F.Context(s, prec)
        if prec == F.PREC_FP32:
            g.set_option(F.OPT_TILE, 3)
        g.meteo(0)
        g.source(0)
        g.step(STEPS)
        g.sync()
        out[k] = g.fields()["c"]
        g.close()
    except Exception as e:  # noqa: BLE001
        out[k] = e


@pytest.mark.parametrize("prec", [F.PREC_FP32, F.PREC_FP64])
def test_side_by_side(prec):
    scen = _scenarios(prec)
    alone, beside = [None] * len(scen), [None] * len(scen)
    for k, s in enumerate(scen):
        _steps(s, prec, alone, k)
    threads = [threading.Thread(target=_steps, args=(s, prec, beside, k)) for k, s in enumerate(scen)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, beside):
        assert isinstance(a, np.ndarray) and isinstance(b, np.ndarray), (a, b)
        assert np.array_equal(a, b)
