"""kappa3 on grids whose threads take one level of a column, several, and the
most, with a short last group, and with both diffusivities constant: the
oracle's values, bit for bit in the vertical (square roots at most), to a few
ulp in the horizontal (RAMS takes a power from the C library)."""
import numpy as np
import pytest

import fall3d_gb300 as F
import oracle_lib as O
from fall3d_gb300 import synth
from helpers import assert_close, assert_same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modkv,modkh", [(1, 1), (2, 2), (1, 0), (0, 1), (0, 0)])
@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 3), (33, 29, 14), (90, 80, 13), (80, 80, 25), (128, 121, 23),
                                      (300, 121, 19)])
def test_kappa3(nx, ny, nz, modkv, modkh):
    s = synth.make_scenario("small", seed=4, nx=nx, ny=ny, nz=nz, nc=1, rmol=-1.0 / 300.0, rkh0=321.0, rkv0=12.5,
                            run_h=0.5)
    g, m = s.grid, s.met
    f3 = [np.ascontiguousarray(m[k][0]) for k in ("u", "v", "tp")]
    f2 = [np.ascontiguousarray(m[k][0]) for k in ("ust", "pblh", "rmol")]
    f2[2] = np.ascontiguousarray(f2[2] * np.linspace(-1.0, 1.0, nx)[None, :])  # both stabilities
    num = (nx, ny, nz, modkv, modkh, 0, g["rkv0"], g["rkh0"], g["Csh"], g["dX1"], g["dX2"], g["dx"], g["dy"])
    kva, kha, kvb, khb = (np.full((nz, ny, nx), 7.0) for _ in range(4))
    arr = [g["dz"], g["zlayer"], g["Hm1"], *f3, *f2]
    O.load().orc_kappa3(*num, *(O.p(a) for a in arr), O.p(kva), O.p(kha))
    F.kappa3(*num, *arr, kvb, khb)
    assert_same_bits(kvb, kva, "rkver")
    assert_close(khb, kha, 1e-13, 0.0, "rkhor")
