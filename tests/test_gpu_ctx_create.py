"""Creating a context computes nothing of a meteorological update: the drag
model's class constants are made with the first one and kept for the others."""
import numpy as np
import pytest

import fall3d_gb300 as F
from fall3d_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modv", [1, 2, 3, 4])
def test_class_constants_come_with_the_first_update(modv):
    s = synth.make_scenario("small", seed=3, modv=modv, run_h=0.5)
    n = F.kernel_launches()
    g = F.Context(s, F.PREC_FP64)
    assert F.kernel_launches() == n
    counts, vset = [], []
    for _ in range(3):
        n = F.kernel_launches()
        g.meteo(0)
        g.upload_state(cd=1.0)  # the chain starts again
        counts.append(F.kernel_launches() - n)
        vset.append(g.fields()["vset"])
    assert counts[0] == counts[1] + 1 == counts[2] + 1
    assert np.array_equal(vset[0], vset[1]) and np.array_equal(vset[0], vset[2])
    g.close()
