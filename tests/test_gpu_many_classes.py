"""Output variables of contexts with very many classes: more than the doubles of
a block's default shared memory, and class numbers beyond 16 bits.  Bit for bit
the oracle's restatement."""
import numpy as np
import pytest

import fall3d_gb300 as F
import oracle_lib as O
from fall3d_gb300 import synth

pytestmark = pytest.mark.gpu


def _context(nc):
    s = synth.make_scenario("tiny", seed=1, nx=3, ny=3, nz=3, nc=nc, run_h=0.2)
    return s, F.Context(s, F.PREC_FP64)


@pytest.mark.parametrize("nc", [127, 128, 129, 6144, 6145, 6400])
def test_thickness(nc):
    s, g = _context(nc)
    r = np.random.default_rng(nc)
    dry, wet = r.random((nc + 1, 3, 3)), r.random((nc + 1, 3, 3))
    g.upload_state(cdry=dry, cwet=wet)
    f = dict(c=np.zeros((nc, 5, 5, 5)), cdry=dry, cwet=wet)
    for v in (F.OUT_LOAD, F.OUT_THICK):
        assert np.array_equal(g.output(v), O.output(s.grid, f, v))
    g.close()


def test_class_numbers_beyond_16_bits():
    nc = 65600
    s, g = _context(nc)
    c = np.zeros((nc, 5, 5, 5))
    c[:, 1:-1, 1:-1, 1:-1] = np.arange(1, nc + 1)[:, None, None, None]
    g.upload_state(c)
    hm = np.asarray(s.grid["Hm1"])
    for index in (1, 65535, 65536, 65537, nc):  # class `index`
        assert np.array_equal(g.output(F.OUT_CON, index), 1e3 * (np.full((3, 3, 3), float(index)) / hm)), index
    g.close()
