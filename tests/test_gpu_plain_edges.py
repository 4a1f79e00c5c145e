"""The plain form's sweeps where their kernels can go wrong: the smallest
lines, sides around a warp and a block, columns cut into pieces, lines too long for the staged products
(advcty), tails that fall off through the subnormals to zero, signed zeros and
non-finite values in the diffusion's end faces.  Against the oracle, bit for
bit (NaN payloads aside)."""
import numpy as np
import pytest

import fall3d_gb300 as F
import oracle_lib as O
from helpers import assert_close, assert_same_bits, oracle_state

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (4, 5, 3), (31, 4, 4), (32, 65, 5), (127, 3, 9), (129, 7, 4), (257, 33, 3), (5, 290, 4),
         (3, 1451, 3), (3, 4200, 3), (9, 8, 33), (33, 5, 41), (6, 5, 63)]


def _state(nx, ny, nz, special):
    r = np.random.default_rng(nx + 10 * ny + 100 * nz)
    shape = (nz + 2, ny + 2, nx + 2)
    c = r.random(shape) * 10.0 ** r.uniform(-3, 3, shape)
    c *= 10.0 ** np.minimum(0.0, np.linspace(20.0, -330.0, nx + 2))[None, None, :] if nx > 40 else 1.0
    c[r.random(shape) < 0.1] = 0.0
    if special:
        pool = np.array([0.0, -0.0, 5e-324, -3e-310, 1e308, -1e308, np.inf, -np.inf, np.nan])
        m = r.random(shape) < 0.2
        c[m] = r.choice(pool, m.sum())
    met = {k: np.ascontiguousarray(r.uniform(lo, hi, (nz, ny, nx)))
           for k, lo, hi in (("v", -20.0, 20.0), ("k", 0.0, 900.0), ("rho", 0.4, 1.3), ("vs", -2.0, 0.0))}
    met["v"][r.random((nz, ny, nx)) < 0.05] = 0.0
    return np.ascontiguousarray(c), met, r.uniform(100.0, 700.0, nz + 1)


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_sweeps(nx, ny, nz, special):
    c, m, dz = _state(nx, ny, nz, special)
    lib, dt, dx = O.load(), 3.1, 1234.5
    full, part = (nx, ny, nz, nz, 1), (nx, ny, nz, nz - 1, 2)
    calls = []
    for a in (full, part):
        calls += [("advctx", (*a, m["v"], dx, dt)), ("advcty", (*a, m["v"], dx, dt)),
                  ("advctzc", (*a, m["v"], m["vs"], dz, dt)), ("diffx", (*a, dx, dt, m["k"], m["rho"])),
                  ("diffy", (*a, dx, dt, m["k"], m["rho"])), ("diffz", (*a, dz, dt, m["k"], m["rho"]))]
    with np.errstate(all="ignore"):
        for name, args in calls:
            a, b = c.copy(), c.copy()
            getattr(lib, "orc_" + name)(O.p(a), *[O.p(v) if isinstance(v, np.ndarray) else v for v in args])
            getattr(F, name)(b, *args)
            assert_same_bits(b, a, f"{name} {args[:5]}")


@pytest.mark.parametrize("nx,ny,nz,nc", [(20, 18, 9, 3), (70, 9, 19, 5), (9, 75, 33, 2)])
def test_steps_of_split_classes_and_pieces(nx, ny, nz, nc):
    """The plain form's steps where lines and columns do not fill the chip
    (classes spread over blocks, narrow tiles, pieces of columns): the oracle's
    state to the tolerance of whole runs (its settling velocities differ by a
    few ulp, the sweeps by nothing)."""
    s, o = oracle_state("small", seed=11, steps=6, nx=nx, ny=ny, nz=nz, nc=nc, run_h=1.0)
    g = F.Context(s, F.PREC_FP64)
    g.meteo(0)
    g.source(0)
    g.step(6)
    g.sync()
    fo, fg = o.fields(), g.fields()
    for k in ("c", "cdry", "cwet"):
        assert_close(fg[k], fo[k], 1e-12, 1e-9, k)
    assert np.max(fg["c"]) > 0.0
