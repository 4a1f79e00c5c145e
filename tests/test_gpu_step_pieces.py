"""The step kernel where its dispatch can go wrong: columns cut into pieces
(few tiles, many levels), a mixing height that forces a tall first piece, the
smallest grid, sides around the tile's 58 columns and 10 or 26 rows, and even
and odd row lengths (padded rows).  Every shape agrees bit for bit, a batch
agrees with the context alone, and the state stays within binary32 rounding
of the plain form: a step rounds each value a few tens of times, so N steps
differ by at most about 30*N*2^-24 of the largest concentration."""
import numpy as np
import pytest

import fall3d_gb300 as F
from fall3d_gb300 import synth
from helpers import assert_same_bits

pytestmark = pytest.mark.gpu
STEPS = 8


@pytest.mark.parametrize("nx,ny,nz,nc,pblh", [
    (3, 3, 3, 1, 1000.0), (4, 3, 40, 1, 1000.0), (5, 12, 17, 2, 3000.0), (12, 10, 60, 2, 9000.0),
    (57, 25, 33, 3, 1000.0), (58, 26, 33, 2, 1000.0), (59, 27, 21, 2, 20000.0), (61, 11, 13, 2, 1000.0),
    (116, 53, 25, 2, 2500.0), (117, 20, 24, 3, 1000.0)])
def test_pieces_and_edges(nx, ny, nz, nc, pblh):
    s = synth.make_scenario("small", seed=5, nx=nx, ny=ny, nz=nz, nc=nc, wetdep=True, run_h=1.0, H=6000.0, pblh=pblh)
    s.met["prate"][:] = np.float32(3.0 / 3600.0)
    r = np.random.default_rng(nx * ny)
    c0 = np.zeros((nc, nz + 2, ny + 2, nx + 2))
    c0[:, 1:-1, 1:-1, 1:-1] = r.random((nc, nz, ny, nx)).astype(np.float32)

    def run(prec, tile=3):
        g = F.Context(s, prec)
        if prec == F.PREC_FP32:
            g.set_option(F.OPT_TILE, tile)
        g.meteo(0)
        g.source(0)
        g.upload_state(c0)
        g.step(STEPS)
        g.sync()
        return g.fields(), g.state()["outmass"]

    a, out_a = run(F.PREC_FP32, 3)
    b, out_b = run(F.PREC_FP32, 0)
    for k in ("c", "cdry", "cwet"):
        assert_same_bits(b[k], a[k], k)
    assert out_a == out_b
    d, out_d = run(F.PREC_FP64)
    tol = 30 * STEPS * 2.0 ** -24
    for k in ("c", "cdry", "cwet"):
        assert np.max(np.abs(a[k] - d[k])) <= tol * max(np.max(np.abs(d[k])), 1e-300), k
    assert abs(out_a - out_d) <= tol * abs(out_d)
    if np.any(np.asarray(s.grid["diam"]) <= 1e-4):  # wet deposition acts on particles of at most 100 um
        assert np.max(a["cwet"]) > 0.0


@pytest.mark.parametrize("nx,ny,nz,nc", [(30, 20, 9, 3), (58, 10, 9, 152), (58, 10, 9, 153), (117, 41, 8, 8)])
def test_default_shape_equals_the_set_ones(nx, ny, nz, nc):
    """Where no tile shape was set the step picks one by the number of tiles
    (both sides of one tile per SM): the same bits as with either."""
    s = synth.make_scenario("small", seed=7, nx=nx, ny=ny, nz=nz, nc=nc, run_h=1.0, H=5000.0)
    out = []
    for tile in (None, 0, 3):
        g = F.Context(s, F.PREC_FP32)
        assert g.get_option(F.OPT_TILE) == 3
        if tile is not None:
            g.set_option(F.OPT_TILE, tile)
        g.meteo(0)
        g.source(0)
        g.step(STEPS)
        g.sync()
        out.append((g.fields(), g.state()["outmass"]))
    for f, om in out[1:]:
        for k in ("c", "cdry"):
            assert_same_bits(f[k], out[0][0][k], k)
        assert om == out[0][1]


def test_batch_of_pieces_equals_alone():
    """Members of different sizes in one batch: the batched launch cuts the
    columns as a launch of its own does, and the results are the same bits."""
    scen = [synth.make_scenario("small", seed=k, nx=nx, ny=ny, nz=nz, nc=2, wetdep=bool(k % 2), run_h=1.0, H=5000.0)
            for k, (nx, ny, nz) in enumerate([(12, 10, 40), (59, 27, 17), (64, 33, 24)])]
    alone = []
    for s in scen:
        g = F.Context(s, F.PREC_FP32)
        g.run(max_steps=STEPS)
        alone.append(g.fields())
    b = F.Batch(4)
    b.set_option(F.OPT_TILE, 3)
    ctx = [F.Context(s, F.PREC_FP32) for s in scen]
    slots = [b.add(g, max_steps=STEPS) for g in ctx]
    b.run()
    for slot in slots:
        b.release(slot)
    for g, ref in zip(ctx, alone):
        f = g.fields()
        for k in ("c", "cdry", "cwet"):
            assert_same_bits(f[k], ref[k], k)


@pytest.mark.parametrize("nx,ny,nz,nc", [(3, 3, 3, 1), (7, 5, 13, 3), (40, 30, 20, 12), (33, 31, 29, 5)])
@pytest.mark.parametrize("modv", [1, 2, 3, 4])
def test_setvset_segments(nx, ny, nz, nc, modv):
    """The settling chain through the fine-grained entry point on sizes whose
    chain has one, an odd and an even number of segments, with a short last
    one (what the call keeps behind the segments' arrays must stay aligned),
    against the oracle: the velocities to 1e-12, the chain's exit value too."""
    import oracle_lib as O

    r = np.random.default_rng(nx + nz)
    T = r.uniform(215.0, 300.0, (nz, ny, nx)).astype(np.float32).astype(float)
    rho = r.uniform(0.05, 1.25, (nz, ny, nx)).astype(np.float32).astype(float)
    diam = np.round(2.0 ** -np.linspace(-2.0, 6.0, nc), 6) / 1e3
    rhop, sphe = np.linspace(2500.0, 1000.0, nc), np.full(nc, 0.9)
    psi = synth.setpsi(modv, sphe, diam)
    v = np.zeros((nc, nz, ny, nx))
    cd = F.setvset(nx, ny, nz, nc, nc, modv, diam, rhop, psi, sphe, T, rho, 0, 1.0, v, 1.0)
    s = synth.make_scenario("tiny", seed=1, nx=nx, ny=ny, nz=nz, nc=nc, modv=modv)
    s.grid.update(diam=diam, rhop=rhop, sphe=sphe, psi=psi)
    s.met["t"][0], s.met["rho"][0] = T, rho
    o = O.OracleCtx(s)
    o.meteo(0)
    ref = o.fields()["vset"]
    assert np.max(np.abs(v / ref - 1.0)) <= 1e-12
    assert abs(cd / o.state()["cd"] - 1.0) <= 1e-12
