"""Checkpoints taken when an update is due and not yet made (the run stopped at
the first step past the interval's end): the restored run enters the update
from the settling chain's value that the uninterrupted run enters it from, and
with aggregation calls agrpar as often.  Bit for bit, at every step around both
ends, with the look-ahead update on and off."""
import numpy as np
import pytest

import fall3d_gb300 as F
from fall3d_gb300 import synth
from helpers import assert_same_bits

pytestmark = pytest.mark.gpu


def _compare(make, tmp_path, steps, more):
    ref = make()
    ref.run(max_steps=steps)
    path = tmp_path / "at.ckpt"
    ref.save(path)
    st = ref.state()
    ref.run(max_steps=more)
    new = make()
    new.restore(path)
    new.run(max_steps=more)
    a, b = ref.fields(), new.fields()
    for k in ("c", "cdry", "cwet"):
        assert_same_bits(b[k], a[k], (steps, k))
    # values: a gas class's zero changes its sign with every update, of which a restored run makes fewer
    assert np.array_equal(b["vset"], a["vset"])
    assert ref.state() == new.state()
    ref.close()
    new.close()
    return st["time"], st["dt"]


def _around_the_update(make, tmp_path):
    """Checkpoints a step before, at and after the first step past 900 s."""
    probe = make()
    n = 0
    while probe.state()["time"] < 900.0:
        probe.run(max_steps=1)
        n += 1
    probe.close()
    due = 0
    for steps in range(n - 1, n + 2):
        time, dt = _compare(make, tmp_path, steps, 3)
        due += 900.0 <= time < 900.0 + dt
    assert due == 1  # one of them stopped with the update due


@pytest.mark.parametrize("prec,pref", [(F.PREC_FP32, 0), (F.PREC_FP32, 1), (F.PREC_FP64, 0), (F.PREC_FP64, 1)])
def test_meteo_update_due(tmp_path, prec, pref):
    s = synth.make_scenario("small", seed=178, nx=31, ny=7, nz=21, nc=2, coord=synth.COORD_UTM, spacing=4187.0, modv=2,
                            u10=1.0, spectral=True, hill=0.0, ztop=18800.0, run_h=1.0, met_dt_h=0.25, H=4000.0)

    def make():
        g = F.Context(s, prec)
        g.set_option(F.OPT_PREFETCH, pref)
        return g

    _around_the_update(make, tmp_path)


@pytest.mark.parametrize("prec", [F.PREC_FP32, F.PREC_FP64])
@pytest.mark.parametrize("met_dt_h", [0.25, 1.0])  # with the source update at 900 s, and the source update alone
def test_aggregation_and_source_update_due(tmp_path, prec, met_dt_h):
    s = synth.make_scenario("small", seed=9, nx=16, ny=14, nz=12, nc=7, phimin=3.0, phimax=8.0,
                            aggregate=[0.2, 1000.0, 0.2], M0=1e7, run_h=1.0, met_dt_h=met_dt_h, erupt_h=0.25)
    synth.add_gas_class(s)
    agg = synth.aggregation_inputs(s)

    def make():
        g = F.Context(s, prec)
        g.set_aggregation(agg)
        return g

    _around_the_update(make, tmp_path)
